"""The stand-alone cell grid's scatter never writes outside its buffer, also
when overlapping calls clear each other's counters. Checked on the host, on the
function the kernel calls (csrc/vlj_place.h): nothing out of range runs."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_scatter_places_stay_in_the_buffer(tmp_path):
    exe = str(tmp_path / "test_place")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror",
                    "-I" + os.path.join(ROOT, "virial-engine_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "test_place.cpp"), "-o", exe], check=True)
    done = subprocess.run([exe], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout
