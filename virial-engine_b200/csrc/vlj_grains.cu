// Contacts of granular spheres found through the cell grid:
// vlj_grain_cells, vlj_grain_contacts.
//
// The reference's granular solver includes the same grid as the
// Lennard-Jones one (granular.rs:327-328 appends grid.wgsl to granular.wgsl):
// it bins the grains into cells of at least one diameter, sorts each cell by
// grain index, and every grain visits the 27 cells around its own (not
// periodic: cells past a wall are skipped) in the order dz, dy, dx = -1..1,
// each in its sorted order, keeping the grains whose spheres overlap its own
// (granular.wgsl:204-263). Here that search runs on the library's grid
// pipeline (vlj_binning.cuh) and writes each grain's partners in that order,
// the table the reference's contact springs are indexed by.
//
// Arithmetic as the reference's: positions as double-float (hi = f32(x), lo
// = f32(x - hi)), d = (x_i.hi - x_j.hi) + (x_i.lo - x_j.lo) per axis in f32,
// dist2 = dot(d, d), reach = r_i + r_j (f32 radii), dist = sqrt(dist2), and a
// contact when reach - dist > 0 and dist2 > 0, each operation rounded as
// written (no contraction).
#include <cuda_runtime.h>

#include <cmath>

#include "virial_lj.h"
#include "vlj_binning.cuh"
#include "vlj_common.h"

namespace vlj {
namespace {

struct GrainGrid {
    uint32_t n;        // grains
    uint32_t cells;    // cells per axis
    uint32_t capacity; // partners kept per grain
};

__device__ __forceinline__ void df_parts(const double* pos, uint32_t i, float h[3], float l[3]) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const double x = pos[3 * (size_t)i + k];
        h[k] = (float)x;
        l[k] = (float)(x - (double)h[k]);
    }
}

// kGrainLanes consecutive threads a grain. The 27 cells around its own (dz,
// dy, dx) are nine rows of up to three cells, each row one run of the sorted
// order; a lane per row reads the run's ends, which makes the rows one stream
// of candidates in the reference's order, and the lanes test kGrainLanes of
// them at a time. The hits' rank in the ballot keeps the order of the partner
// table; counts[i] is the number of contacts (also those past the capacity,
// which are not written).
// One thread a grain spent its time on chains of dependent loads, a cell and
// a candidate after the other: 67 us for 100,000 grains of a packed bed
// (49 candidates a grain), 41 us so. (A whole warp a grain: a pass of 98 us
// against 90, its last lanes idle.)
constexpr uint32_t kGrainLanes = 16;

__global__ void __launch_bounds__(128) grain_contacts_kernel(const double* __restrict__ pos,
                                      const double* __restrict__ radius, GrainGrid g,
                                      const uint32_t* __restrict__ sorted,
                                      const uint32_t* __restrict__ cell_start,
                                      const uint32_t* __restrict__ cell_of,
                                      uint32_t* __restrict__ partners,
                                      uint32_t* __restrict__ counts) {
    constexpr int kW = (int)kGrainLanes;
    const uint32_t sub = threadIdx.x % kGrainLanes;
    const uint32_t k = blockIdx.x * (128u / kGrainLanes) + threadIdx.x / kGrainLanes;
    const bool valid = k < g.n;
    const uint32_t i = valid ? k : 0u;
    const int32_t n = (int32_t)g.cells;
    const uint32_t c = cell_of[i];
    uint32_t from = 0, cnt = 0;
    if (valid && sub < 9u) {
        const int32_t x = (int32_t)(c % g.cells);
        const int32_t y = (int32_t)((c / g.cells) % g.cells) + (int32_t)(sub % 3u) - 1;
        const int32_t z = (int32_t)(c / (g.cells * g.cells)) + (int32_t)(sub / 3u) - 1;
        if (y >= 0 && z >= 0 && y < n && z < n) {
            const uint32_t row = ((uint32_t)z * g.cells + (uint32_t)y) * g.cells;
            from = cell_start[row + (uint32_t)max(x - 1, 0)];
            cnt = cell_start[row + (uint32_t)min(x + 1, n - 1) + 1u] - from;
        }
    }
    float xh[3], xl[3];
    df_parts(pos, i, xh, xl);
    const float r = (float)radius[i];
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < kW; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o, kW);
        if (sub >= (uint32_t)o) incl += t;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, kW - 1, kW);
    const uint32_t most = __reduce_max_sync(0xffffffffu, total);
    const uint32_t shift = (threadIdx.x & 31u) - sub;
    uint32_t found = 0;
    for (uint32_t t0 = 0; t0 < most; t0 += kGrainLanes) {
        const uint32_t t = t0 + sub;
        // the row of candidate t: the first whose run ends past it
        uint32_t row = 0;
#pragma unroll
        for (int o = kW / 2; o > 0; o >>= 1)
            if (__shfl_sync(0xffffffffu, incl, (int)row + o - 1, kW) <= t) row += (uint32_t)o;
        const uint32_t at = __shfl_sync(0xffffffffu, incl - cnt, (int)row, kW);
        const uint32_t start = __shfl_sync(0xffffffffu, from, (int)row, kW);
        bool hit = false;
        uint32_t j = 0;
        if (t < total) {
            j = sorted[start + (t - at)];
            float ph[3], pl[3];
            df_parts(pos, j, ph, pl);
            float d[3];
#pragma unroll
            for (int a = 0; a < 3; a++)
                d[a] = __fadd_rn(__fsub_rn(xh[a], ph[a]), __fsub_rn(xl[a], pl[a]));
            const float dist2 = __fadd_rn(__fadd_rn(__fmul_rn(d[0], d[0]), __fmul_rn(d[1], d[1])),
                                          __fmul_rn(d[2], d[2]));
            const float reach = __fadd_rn(r, (float)radius[j]);
            const float dist = __fsqrt_rn(dist2);
            hit = j != i && __fsub_rn(reach, dist) > 0.0f && dist2 > 0.0f;
        }
        const uint32_t mask = (__ballot_sync(0xffffffffu, hit) >> shift) & ((1u << kGrainLanes) - 1u);
        const uint32_t place = found + (uint32_t)__popc(mask & ((1u << sub) - 1u));
        if (hit && place < g.capacity) partners[(size_t)i * g.capacity + place] = j;
        found += (uint32_t)__popc(mask);
    }
    if (valid && sub == 0u) counts[i] = found;
}

}  // namespace
}  // namespace vlj

using vlj::fail;

extern "C" {

vlj_status vlj_grain_cells(double box_size, double max_radius, uint32_t* cells) {
    if (!cells) return fail(VLJ_INVALID_ARG, "grain_cells: null argument");
    if (!(box_size > 0.0) || !(box_size < 1e30) || !(max_radius > 0.0) || !(max_radius < 1e30))
        return fail(VLJ_INVALID_ARG, "grain_cells: box size and radius must be positive and finite");
    // granular.rs:179-181
    const double c = std::floor(box_size / (2.0 * max_radius));
    *cells = c < 1.0 ? 1u : (c > 64.0 ? 64u : (uint32_t)c);
    return VLJ_OK;
}

vlj_status vlj_grain_contacts(const double* pos, const double* radius, size_t count,
                              double box_size, uint32_t cells, uint32_t capacity,
                              uint32_t* scratch, uint32_t* sorted, uint32_t* cell_start,
                              uint32_t* cell_of, uint32_t* partners, uint32_t* counts,
                              void* stream) {
    if (!pos || !radius || !scratch || !sorted || !cell_start || !cell_of || !counts ||
        (!partners && capacity))
        return fail(VLJ_INVALID_ARG, "grain_contacts: null argument");
    if (count == 0 || count >= (1ull << 31))
        return fail(VLJ_INVALID_ARG, "grain_contacts: count must be in 1 .. 2^31 - 1");
    if (!(box_size > 0.0) || !(box_size < 1e30))
        return fail(VLJ_INVALID_ARG, "grain_contacts: box size must be positive and finite");
    if (cells == 0 || cells > 64)
        return fail(VLJ_INVALID_ARG, "grain_contacts: cells per axis must be in 1 .. 64");
    if ((uint64_t)count * capacity >= (1ull << 40))
        return fail(VLJ_INVALID_ARG, "grain_contacts: partner table too large");
    vlj::BinGrid g;
    for (int k = 0; k < 3; k++) {
        g.cells[k] = cells;
        // granular.rs:182: the cell side in f64, then f32 as the shader gets it
        g.cell_size[k] = (float)(box_size / (double)cells);
    }
    g.total = cells * cells * cells;
    g.n = (uint32_t)count;
    const cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaError_t e = vlj::enqueue_binning(pos, g, scratch, sorted, cell_start, cell_of, s);
    if (e == cudaSuccess) {
        const vlj::GrainGrid gg{g.n, cells, capacity};
        const unsigned blocks = (unsigned)(((uint64_t)g.n * vlj::kGrainLanes + 127u) / 128u);
        vlj::grain_contacts_kernel<<<blocks, 128, 0, s>>>(
            pos, radius, gg, sorted, cell_start, cell_of, partners, counts);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return fail(VLJ_CUDA_ERROR, "grain_contacts: %s", cudaGetErrorString(e));
    return VLJ_OK;
}

}  // extern "C"
