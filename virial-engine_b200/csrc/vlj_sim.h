// The simulation object behind the opaque vlj_sim handle.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <vector>

#include "virial_lj.h"
#include "vlj_internal.cuh"

namespace vlj {

constexpr int kRing = 3;  // measurement read-back slots (lennard_jones.rs:320)
constexpr uint32_t kGraphChunk = 16;  // most steps per graph launch
constexpr int kChunks = 4;            // graphs of 16, 8, 4 and 2 steps
// The call with a use for it in which a graph of 8, 4 or 2 steps is captured
// (sim_enqueue_steps); until then its steps go out in smaller ones.
constexpr uint32_t kChunkUses = 32;
// Steps that a run enqueues at a time: whole graphs of 16.
constexpr uint32_t kRunSteps = 12 * kGraphChunk;

// The words the host reads back, one after the other on the device (the
// measurement sums, control words and thermostats of every box, then the
// arena's global words), so that one copy brings them all. For a single box:
struct Readback {
    long long slots[kSlots];
    Control ctrl;
    Thermo nh;
    Global glob;
};
static_assert(sizeof(Readback) == sizeof(long long) * kSlots + sizeof(Control) + sizeof(Thermo) + sizeof(Global),
              "the words lie side by side");

double scale_for(double magnitude);
vlj_status check_settings(const vlj_settings* st);
vlj_status make_box(const vlj_particle* p, size_t count, const double box_size[3], double cutoff,
                    double skin, double dt, bool shifted_force, const vlj_thermostat& t,
                    uint32_t profile_bins, Box& b, uint32_t min_cells);

}  // namespace vlj

struct vlj_sim {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    vlj_settings settings{};
    uint32_t n = 0;
    bool shifted_force = false;
    bool nose_hoover = false;  // steps on canonical velocities with the thermostat
    bool exchange = false;     // heat exchange on (constant energy, canonical velocities)
    vlj_heat_exchange exchange_settings{};
    bool canonical() const { return nose_hoover || exchange; }
    bool grid_every_step = false;  // bin, scan, scatter, sort every step; lists on the trigger
    bool tiles_on = true;  // the step kernel stages cell tiles (when the box has them)
    bool list_growth = true;   // grow the list capacity when a list overflows
    bool grow_pending = false; // a polled measurement showed an overflow
    uint32_t list_grows = 0;   // capacity grows so far
    vlj::Box box{};
    // batched: one Box per replica, in slot order (empty for a single box)
    std::vector<vlj::Box> replicas;
    vlj::Arena arena{};
    CUtensorMap list_map;  // list rows for the force kernels' TMA tiles
    std::vector<void*> allocations;
    uint64_t steps = 0;
    // measurement read-back ring
    vlj::Readback* ring = nullptr;
    cudaEvent_t ring_event[vlj::kRing] = {};
    bool ring_busy[vlj::kRing] = {};
    uint64_t ring_step[vlj::kRing] = {};
    // those words of every box, pinned (sim_read_status)
    unsigned char* status = nullptr;
    size_t status_bytes = 0;
    const long long* status_slots() const { return reinterpret_cast<const long long*>(status); }
    const vlj::Control* status_ctrl() const {
        return reinterpret_cast<const vlj::Control*>(status + sizeof(long long) * vlj::kSlots * arena.nboxes);
    }
    const vlj::Global* status_glob() const {
        return reinterpret_cast<const vlj::Global*>(status + status_bytes - sizeof(vlj::Global));
    }
    // profiles
    uint64_t profile_samples = 0;
    // heat current series
    uint32_t series_samples = 0;
    // the last requested sample is not taken yet: the next step's force pass
    // takes it (or, before anything that would change the state or read the
    // series, the sampling kernel)
    bool heat_pending = false;
    uint32_t series_capacity = 0;
    unsigned long long* series = nullptr;  // owned here (reallocated by record)
    // pinned staging for a batch's particle uploads (x, v: 3 * seg; id: seg)
    double* pin_x = nullptr;
    double* pin_v = nullptr;
    uint32_t* pin_id = nullptr;
    // captured steps: graphs of kGraphChunk >> k steps and one of a single
    // step, each step's rebuild chain under a conditional node; those of 16 and
    // of one step captured when first needed, the others in the kChunkUses-th
    // call with a use for them
    bool use_graphs = true;
    cudaStream_t capture_stream = nullptr;
    cudaGraphExec_t graph_chunk[vlj::kChunks] = {};
    uint32_t chunk_uses[vlj::kChunks] = {};  // calls with a use for each since the last drop
    cudaGraphExec_t graph_one = nullptr;
    // graph_one's template (kept for node updates) and its decide node: while
    // the last step enqueued was graph_one's, whose step kernel took this
    // step's decision and set graph_one's condition, the node is disabled
    cudaGraph_t graph_one_tmpl = nullptr;
    cudaGraphNode_t one_decide = nullptr;
    bool one_decide_on = true;
    bool one_ready = false;
    // the lists were brought up to date and nothing has changed since (lists_now)
    bool lists_current = false;
    // some of the sim's work was enqueued while the caller captured its stream:
    // from then on it may run again at any time, unseen by the host
    bool captured = false;
    cudaGraphExec_t graph_one_heat = nullptr;  // one step that also takes the pending sample
    cudaGraphExec_t graph_lists = nullptr;  // decide -> IF(rebuild){rebuild chain}
    // per-launch timing of the step kernel (direct launches while on)
    bool timing = false;
    std::vector<cudaEvent_t> ev_start, ev_end;
    size_t ev_used = 0;

    ~vlj_sim();
};

namespace vlj {
vlj_status sim_allocate(vlj_sim* s, void* stream);
vlj_status make_list_map(const Arena& a, uint32_t rows, CUtensorMap* out);
// Decide and, when due, rebuild the lists now (positions are about to be read).
vlj_status sim_lists_now(vlj_sim* s);
// Whether work was, or is being, captured into a graph of the caller's.
bool sim_note_capture(vlj_sim* s);
// Everything enqueued so far, then the status words, waited for; an error
// where a kernel recorded a fault.
vlj_status sim_read_status(vlj_sim* s);
vlj_status fault_status(uint32_t fault);
// The same, and lists that overflowed grow: what ends a run.
vlj_status sim_settle(vlj_sim* s);
vlj_status sim_enqueue_steps(vlj_sim* s, uint32_t steps);
// Takes a pending heat-current sample now, with the sampling kernel.
vlj_status sim_flush_heat(vlj_sim* s);
// With list growth on and a list overflowed since the last build: raise the
// capacity of every box that overflowed, reallocate the lists, drop the
// captured graphs and force a rebuild (waits). *grew says whether it did.
vlj_status sim_grow_lists(vlj_sim* s, bool* grew);
// List growth at creation: on, unless the environment sets VLJ_LIST_GROWTH=0
// (the reference's report-only behaviour from the first build on).
bool list_growth_default();
// Drops the captured step graphs (their shape changed).
void sim_drop_step_graphs(vlj_sim* s);
// The decision and, when due, the rebuild as one graph launch.
vlj_status sim_launch_lists_graph(vlj_sim* s);
}  // namespace vlj
