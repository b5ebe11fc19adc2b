"""Host checks of the cell grid's arithmetic, on the functions that its kernels
and launches call, so that nothing out of range runs.

- The stand-alone grid's scatter (csrc/vlj_place.h) never writes outside its
  buffer, also when overlapping calls clear each other's counters.
- The scan's split into blocks (csrc/vlj_scan_shape.h) covers every cell once and
  does not read the square of a large box's cells."""

import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("name", ["test_place", "test_scan_shape"])
def test_on_the_host(tmp_path, name):
    exe = str(tmp_path / name)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror",
                    "-I" + os.path.join(ROOT, "virial-engine_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", name + ".cpp"), "-o", exe], check=True)
    done = subprocess.run([exe], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout
