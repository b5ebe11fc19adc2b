// CUDA kernels of the pair forces, the integrator and the measurements,
// sm_100a.
//
// One thread per particle, 128 per block (small grids: several lanes per
// particle, lanes_for). Each thread reads its Verlet-list
// rows (a row is four entries of a particle, 16 B; a warp's rows are 512
// contiguous bytes) one ahead with loads that do not allocate in L1, issues
// the four neighbour gathers of a row through L1 together, then does the four
// pairs' arithmetic. The force kernels use almost no shared memory and ask for
// the largest L1 carve-out, so the L1 holds the neighbourhood the gathers
// reuse. (The alternative, VLJ_LIST_STREAM=0, stages the rows in shared memory
// as TMA tiles of kTileRows rows x 128 particles on an mbarrier ring; the
// tuner measured it 16-45 % slower on the 256k-atom box, because the tiles
// take the shared memory the L1 needs.) Reference kernels are cited at each
// kernel.
#include <cuda.h>
#include <cuda_runtime.h>

#include "vlj_device.cuh"
#include "vlj_internal.cuh"

namespace vlj {

constexpr uint32_t kTileBytes = kTileRows * kForceThreads * 16u;
// Resident blocks of 128 per SM that the step kernel's register budget is sized
// for: 64 registers at eight. Left to itself the compiler takes 66, which
// leaves seven blocks of 128 and three of 256: 324 us against 300 so on 512
// replicas at 128 particles a block and 362 against 306 at 256, 47.1 against
// 46.2 and 53.3 against 45.5 on the 256,000-atom box (no spill). The form that
// takes a heat-current sample needs more and has no such bound.
#ifndef VLJ_STEP_MIN_BLOCKS
#define VLJ_STEP_MIN_BLOCKS 8
#endif
constexpr int kStepMinBlocks = VLJ_STEP_MIN_BLOCKS;
// Lanes per particle of the force kernels, by grid size (lanes_for): at most
// this many threads per SM after the split.
#ifndef VLJ_LANE_THREADS_PER_SM
#define VLJ_LANE_THREADS_PER_SM 512
#endif
constexpr unsigned long long kWaitLimitNs = 500000000ull;  // 0.5 s per TMA tile

struct PairSums {
    float ax, ay, az;
    float pe, pe_lo;  // this particle's half of its pair energies, hi + lo
    float w, w_lo;    // and of its pair virials r . F
    uint32_t near;    // neighbours within 1.5 sigma
    // heat current: half of the pair energies, and T = sum_j d d^T |F| / r
    // (xx yy zz xy xz yz)
    float e_half, t[6];
    // The force is summed in parts of two list rows (eight entries): each
    // part's sum starts from zero (px, py, pz) and joins the total (ax, ay,
    // az) in list order (end_part). One thread walking all rows and several
    // lanes taking a part each then give the same bits.
    float px, py, pz;
    // likewise the part's energies and virials
    float ppe, ppe_lo, pw, pw_lo;
};

__device__ __forceinline__ void end_part(PairSums& s) {
    s.ax = __fadd_rn(s.ax, s.px);
    s.ay = __fadd_rn(s.ay, s.py);
    s.az = __fadd_rn(s.az, s.pz);
    s.px = s.py = s.pz = 0.0f;
}

// A part's energy and virial into the totals, hi and lo.
__device__ __forceinline__ void add_part_energies(PairSums& s, float pe, float pe_lo, float w,
                                                  float w_lo) {
    float t, e;
    two_sum(s.pe, pe, t, e);
    s.pe = t;
    s.pe_lo = __fadd_rn(s.pe_lo, __fadd_rn(pe_lo, e));
    two_sum(s.w, w, t, e);
    s.w = t;
    s.w_lo = __fadd_rn(s.w_lo, __fadd_rn(w_lo, e));
}

// end_part with the energies.
template <bool ENERGIES>
__device__ __forceinline__ void finish_part(PairSums& s) {
    end_part(s);
    if (ENERGIES) {
        add_part_energies(s, s.ppe, s.ppe_lo, s.pw, s.pw_lo);
        s.ppe = s.ppe_lo = s.pw = s.pw_lo = 0.0f;
    }
}

__device__ __forceinline__ void add_force(PairSums& s, float dx, float dy, float dz, float f) {
    s.px = __fmaf_rn(-dx, f, s.px);
    s.py = __fmaf_rn(-dy, f, s.py);
    s.pz = __fmaf_rn(-dz, f, s.pz);
}

// Shared memory of a force-kernel block: the tile ring and its barriers
// (none when the rows stream straight from global memory).
#if VLJ_LIST_STREAM
struct Stage {
    unsigned long long unused;
};
#else
struct Stage {
    uint4 rows[kTileSlots][kTileRows][kForceThreads];
    unsigned long long bar[kTileSlots];
};
#endif

// A list row (four entries of one slot, 16 B) read once: no L1 allocation,
// so the L1 keeps the neighbour positions the gathers reuse.
__device__ __forceinline__ uint4 load_row_streaming(const uint4* p) {
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}

// ---- TMA and mbarrier primitives (PTX, sm_90+) ----
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void bar_init(unsigned long long* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ void init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// One tile: rows [y, y + kTileRows) of the block's particles (x = first
// particle * 2 u64 elements). Rows and particles past the list's end arrive
// as zeros. No multicast.
__device__ __forceinline__ void tile_load(const CUtensorMap* map, void* dst, unsigned long long* bar,
                                          int x, int y) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                 ::"r"(smem_addr(bar)), "r"(kTileBytes) : "memory");
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_addr(dst)), "l"((unsigned long long)map), "r"(x), "r"(y), "r"(smem_addr(bar))
        : "memory");
}

__device__ __forceinline__ bool bar_try_wait(unsigned long long* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done) : "r"(smem_addr(bar)), "r"(parity) : "memory");
    return done != 0;
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Waits for a tile with a time limit; false when it did not arrive.
__device__ __forceinline__ bool bar_wait(unsigned long long* bar, uint32_t parity) {
    if (bar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    while (!bar_try_wait(bar, parity))
        if (global_ns() - t0 > kWaitLimitNs) return false;
    return true;
}

// ---- forces from the list (lennard_jones.wgsl:503-545) ----
// One list entry's terms into the particle's sums: the separation from the
// 32-bit box fractions (the wrapped integer difference is the nearest
// image), the force factor (the same expression in every pass, so the step,
// the first forces and the measurement agree to the bit), and with ENERGIES
// the halves of the pair energy and virial as unevaluated f32 pairs (as the
// reference sums them in double-float, lennard_jones.wgsl:518-519). A zero
// separation (the padding of a list's last row) adds nothing.
template <bool SHIFTED_FORCE, bool ENERGIES, bool HEAT, bool NEAR = false>
__device__ __forceinline__ void pair_terms(PairSums& s, const uint4 own, const uint4 pj,
                                           const Box& bx, float dec0, float dec1, float dec2,
                                           uint32_t rc2_bits_m1, float fshift) {
    const float dx = decode_diff(pj.x, own.x, dec0);
    const float dy = decode_diff(pj.y, own.y, dec1);
    const float dz = decode_diff(pj.z, own.z, dec2);
    const float r2 = sep_r2(dx, dy, dz);
    const bool in = __float_as_uint(r2) - 1u < rc2_bits_m1;
    // branch-free: most list entries are inside the cutoff; the select
    // drops whatever the pair math gives for entries that are not
    const float f = in ? lj_force_over_r2<SHIFTED_FORCE>(r2, fshift) : 0.0f;
    add_force(s, dx, dy, dz, f);
    if (HEAT) {
        s.e_half += in ? 0.5f * lj_energy_fast<SHIFTED_FORCE>(r2, bx) : 0.0f;
        const float fx = dx * f, fy = dy * f, fz = dz * f;
        s.t[0] += dx * fx;
        s.t[1] += dy * fy;
        s.t[2] += dz * fz;
        s.t[3] += dx * fy;
        s.t[4] += dx * fz;
        s.t[5] += dy * fz;
    }
    if (ENERGIES && in) {
        // The sums take r^2 rounded once from the exact separation (the
        // integer differences times the box step are exact in f64): on a
        // lattice, where every pair at one distance rounds alike, the f32
        // components' three roundings would bias the virial coherently.
        const double ex = (double)(int32_t)(pj.x - own.x) * (double)dec0;
        const double ey = (double)(int32_t)(pj.y - own.y) * (double)dec1;
        const double ez = (double)(int32_t)(pj.z - own.z) * (double)dec2;
        float rf, u, t, e;
        lj_pair<SHIFTED_FORCE>((float)__fma_rn(ez, ez, __fma_rn(ey, ey, __dmul_rn(ex, ex))), bx, rf, u);
        two_sum(s.ppe, 0.5f * u, t, e);
        s.ppe = t;
        s.ppe_lo += e;
        two_sum(s.pw, 0.5f * rf, t, e);
        s.pw = t;
        s.pw_lo += e;
    }
    if (ENERGIES || NEAR) s.near += in && r2 < 2.25f ? 1u : 0u;
}

// pair_terms on positions given as f32 offsets from a common origin near
// both (the cell tiles' f32 form): the separation is their plain difference.
template <bool SHIFTED_FORCE, bool HEAT>
__device__ __forceinline__ void pair_terms_rel(PairSums& s, const float4 own, const float4 pj,
                                               const Box& bx, uint32_t rc2_bits_m1, float fshift) {
    const float dx = __fsub_rn(pj.x, own.x);
    const float dy = __fsub_rn(pj.y, own.y);
    const float dz = __fsub_rn(pj.z, own.z);
    const float r2 = sep_r2(dx, dy, dz);
    const bool in = __float_as_uint(r2) - 1u < rc2_bits_m1;
    const float f = in ? lj_force_over_r2<SHIFTED_FORCE>(r2, fshift) : 0.0f;
    add_force(s, dx, dy, dz, f);
    if (HEAT) {
        s.e_half += in ? 0.5f * lj_energy_fast<SHIFTED_FORCE>(r2, bx) : 0.0f;
        const float fx = dx * f, fy = dy * f, fz = dz * f;
        s.t[0] += dx * fx;
        s.t[1] += dy * fy;
        s.t[2] += dz * fz;
        s.t[3] += dx * fy;
        s.t[4] += dx * fz;
        s.t[5] += dy * fz;
    }
}

// The particle's pair sums over its list. Every thread of the block must
// call this: it synchronises the block between tiles.
template <bool SHIFTED_FORCE, bool ENERGIES, bool HEAT = false, bool NEAR = false>
__device__ __forceinline__ PairSums block_pair_sums(Stage& st, const CUtensorMap* map,
                                                    const Arena& a, const Box& bx, uint32_t i,
                                                    bool valid, const uint4* __restrict__ cur,
                                                    uint32_t block0 = 0) {
    PairSums s = {};
#if !VLJ_LIST_STREAM
    const uint32_t first = (block0 + blockIdx.x) * kForceThreads;
    const uint32_t rows = a.block_rows[block0 + blockIdx.x];
    const uint32_t tiles = (rows + kTileRows - 1u) / kTileRows;
    if (threadIdx.x == 0) {
        for (int k = 0; k < kTileSlots; k++) bar_init(&st.bar[k]);
        init_fence();
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (uint32_t t = 0; t < tiles && t < (uint32_t)kTileSlots; t++)
            tile_load(map, &st.rows[t][0][0], &st.bar[t], (int)(first * 2u), (int)(t * kTileRows));
#else
    (void)st;
    (void)map;
    (void)block0;  // the grid's first block of kForceThreads slots (the TMA tiles' unit)
#endif

    uint4 own = make_uint4(0u, 0u, 0u, 0u);
    uint32_t cnt = 0;
    if (valid) {
        own = __ldg(cur + i);
        cnt = __ldg(a.list_count + i);
    }
    const uint32_t my_rows = (cnt + 3u) / 4u;
    const float dec0 = bx.dec[0], dec1 = bx.dec[1], dec2 = bx.dec[2], rc2 = bx.rc2;
    const float fshift = bx.force_shift;
    // 0 < r2 < rc2 as one unsigned comparison of the bit patterns (r2 >= +0)
    const uint32_t rc2_bits_m1 = __float_as_uint(rc2) - 1u;
    // The list's last row is padded with the particle itself, whose zero
    // separation drops out with the entries beyond the cutoff.
    auto add = [&](const uint4 pj) {
        pair_terms<SHIFTED_FORCE, ENERGIES, HEAT, NEAR>(s, own, pj, bx, dec0, dec1, dec2,
                                                        rc2_bits_m1, fshift);
    };
    // the four entries of list row `row`; a part ends with its odd row
    auto row_terms = [&](uint32_t row, const uint4 p0, const uint4 p1, const uint4 p2,
                         const uint4 p3) {
        add(p0);
        add(p1);
        add(p2);
        add(p3);
        if (row & 1u) finish_part<ENERGIES>(s);
    };

#if VLJ_LIST_STREAM
    const uint4* rowp = reinterpret_cast<const uint4*>(a.list) + i;
#if VLJ_GATHER_AHEAD
    // gathers one row ahead: row r + 1's neighbours are in flight while row
    // r's pairs are computed (its list row two ahead)
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    uint4 e_next = my_rows > 1u ? load_row_streaming(rowp + a.seg) : zero;
    uint4 q0 = own, q1 = own, q2 = own, q3 = own;
    if (my_rows) {
        const uint4 e = load_row_streaming(rowp);
        q0 = __ldg(cur + e.x);
        q1 = __ldg(cur + e.y);
        q2 = __ldg(cur + e.z);
        q3 = __ldg(cur + e.w);
    }
    for (uint32_t row = 0; row < my_rows; row++) {
        const uint4 p0 = q0, p1 = q1, p2 = q2, p3 = q3;
        if (row + 1u < my_rows) {
            const uint4 e = e_next;
            if (row + 2u < my_rows) e_next = load_row_streaming(rowp + (size_t)(row + 2u) * a.seg);
            q0 = __ldg(cur + e.x);
            q1 = __ldg(cur + e.y);
            q2 = __ldg(cur + e.z);
            q3 = __ldg(cur + e.w);
        }
        row_terms(row, p0, p1, p2, p3);
    }
#else
    // each thread its own rows, the next one in flight while it works on
    // this; two rows an iteration: a part of the force sum
    uint4 next = my_rows ? load_row_streaming(rowp) : make_uint4(0u, 0u, 0u, 0u);
    for (uint32_t row = 0; row < my_rows; row += 2u) {
        {
            const uint4 e = next;
            if (row + 1u < my_rows) next = load_row_streaming(rowp + (size_t)(row + 1u) * a.seg);
            const uint4 p0 = __ldg(cur + e.x);
            const uint4 p1 = __ldg(cur + e.y);
            const uint4 p2 = __ldg(cur + e.z);
            const uint4 p3 = __ldg(cur + e.w);
            add(p0);
            add(p1);
            add(p2);
            add(p3);
        }
        if (row + 1u < my_rows) {
            const uint4 e = next;
            if (row + 2u < my_rows) next = load_row_streaming(rowp + (size_t)(row + 2u) * a.seg);
            const uint4 p0 = __ldg(cur + e.x);
            const uint4 p1 = __ldg(cur + e.y);
            const uint4 p2 = __ldg(cur + e.z);
            const uint4 p3 = __ldg(cur + e.w);
            add(p0);
            add(p1);
            add(p2);
            add(p3);
            finish_part<ENERGIES>(s);
        }
    }
#endif
    finish_part<ENERGIES>(s);
    return s;
#else
    bool lost = false;
    for (uint32_t t = 0; t < tiles; t++) {
        const uint32_t slot = t % kTileSlots;
        const bool ok = bar_wait(&st.bar[slot], (t / kTileSlots) & 1u);
        if (__syncthreads_or(!ok)) {
            lost = true;
            break;
        }
#pragma unroll
        for (int r = 0; r < kTileRows; r++) {
            const uint32_t row = t * kTileRows + (uint32_t)r;
            if (row < my_rows) {
                // one row: four entries, the last ones live only up to cnt
                const uint4 e = st.rows[slot][r][threadIdx.x];
                const uint4 p0 = __ldg(cur + e.x);
                const uint4 p1 = __ldg(cur + e.y);
                const uint4 p2 = __ldg(cur + e.z);
                const uint4 p3 = __ldg(cur + e.w);
                row_terms(row, p0, p1, p2, p3);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0 && t + kTileSlots < tiles) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            tile_load(map, &st.rows[slot][0][0], &st.bar[slot], (int)(first * 2u),
                      (int)((t + kTileSlots) * kTileRows));
        }
    }
    if (lost) {
        // record the fault, then let the tiles still in flight land before
        // the block's shared memory goes away
        if (threadIdx.x == 0) {
            atomicCAS(&a.glob->fault, 0u, kFaultTmaTimeout);
            for (uint32_t t = 0; t < tiles && t < (uint32_t)kTileSlots; t++)
                bar_wait(&st.bar[t], 0u);
        }
        __syncthreads();
    }
    finish_part<ENERGIES>(s);
    return s;
#endif
}

// The pair sums of particle i (in every lane) with LANES consecutive threads
// sharing its list: in each round lane `sub` sums part round * LANES + sub
// (two rows, eight gathers in flight), and the round's parts join the totals
// in list order, so the bits are block_pair_sums's. The next round's rows load
// behind this one's pairs. A row past the list's end reads as the particle
// itself, whose zero separation adds nothing. Every lane of the warp must call
// this.
template <bool SHIFTED_FORCE, int LANES, bool ENERGIES = false, bool NEAR = false>
__device__ __forceinline__ PairSums lane_pair_sums(const Arena& a, const Box& bx, uint32_t i,
                                                   bool valid, uint32_t sub,
                                                   const uint4* __restrict__ cur) {
    const uint32_t at = valid ? i : 0u;
    const uint4 own = __ldg(cur + at);
    const uint32_t rows = valid ? (__ldg(a.list_count + at) + 3u) / 4u : 0u;
    const uint32_t rounds =
        __reduce_max_sync(0xffffffffu, (rows + 2u * LANES - 1u) / (2u * LANES));
    const float dec0 = bx.dec[0], dec1 = bx.dec[1], dec2 = bx.dec[2];
    const float fshift = bx.force_shift;
    const uint32_t rc2_bits_m1 = __float_as_uint(bx.rc2) - 1u;
    const uint4* rowp = reinterpret_cast<const uint4*>(a.list) + at;
    const uint4 self = make_uint4(at, at, at, at);
    uint32_t row = 2u * sub;
    uint4 e0 = row < rows ? load_row_streaming(rowp + (size_t)row * a.seg) : self;
    uint4 e1 = row + 1u < rows ? load_row_streaming(rowp + (size_t)(row + 1u) * a.seg) : self;
    PairSums s = {};
    for (uint32_t r = 0; r < rounds; r++) {
        const uint4 p[8] = {__ldg(cur + e0.x), __ldg(cur + e0.y), __ldg(cur + e0.z), __ldg(cur + e0.w),
                            __ldg(cur + e1.x), __ldg(cur + e1.y), __ldg(cur + e1.z), __ldg(cur + e1.w)};
        row += 2u * LANES;
        e0 = row < rows ? load_row_streaming(rowp + (size_t)row * a.seg) : self;
        e1 = row + 1u < rows ? load_row_streaming(rowp + (size_t)(row + 1u) * a.seg) : self;
        s.px = s.py = s.pz = 0.0f;
        s.ppe = s.ppe_lo = s.pw = s.pw_lo = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; k++)
            pair_terms<SHIFTED_FORCE, ENERGIES, false, NEAR>(s, own, p[k], bx, dec0, dec1, dec2,
                                                             rc2_bits_m1, fshift);
#pragma unroll
        for (int k = 0; k < LANES; k++) {
            s.ax = __fadd_rn(s.ax, __shfl_sync(0xffffffffu, s.px, k, LANES));
            s.ay = __fadd_rn(s.ay, __shfl_sync(0xffffffffu, s.py, k, LANES));
            s.az = __fadd_rn(s.az, __shfl_sync(0xffffffffu, s.pz, k, LANES));
            if (ENERGIES)
                add_part_energies(s, __shfl_sync(0xffffffffu, s.ppe, k, LANES),
                                  __shfl_sync(0xffffffffu, s.ppe_lo, k, LANES),
                                  __shfl_sync(0xffffffffu, s.pw, k, LANES),
                                  __shfl_sync(0xffffffffu, s.pw_lo, k, LANES));
        }
    }
    if (ENERGIES || NEAR) {
#pragma unroll
        for (int o = 1; o < LANES; o <<= 1) s.near += __shfl_xor_sync(0xffffffffu, s.near, o);
    }
    return s;
}

// Sum of one heat-current sample's three components over the block into
// series slot 1 + 3 * sample: one atomic each (integer sums, any order).
__device__ __forceinline__ void block_sum_series(const Arena& a, const long long (&raw)[3],
                                                 uint32_t sample) {
    __shared__ long long s_sum[kBlock / 32][3];  // blocks of up to kBlock threads
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        long long x = raw[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) s_sum[warp][c] = x;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        long long x = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) x += s_sum[w][threadIdx.x];
        if (x) atomicAdd(&a.series[1 + 3 * (size_t)sample + threadIdx.x], (unsigned long long)x);
    }
}

// Langevin noise of a particle at a step: Philox-4x32-10 (Salmon et al.,
// SC'11) with counter (id, step lo, step hi, 0) and key (seed, "LJV1");
// uniforms in (0, 1] from 24 bits as the reference's uniform01
// (lennard_jones.wgsl:175-178); Box-Muller in f32: x and y from the first
// pair of uniforms (cosine and sine), z from the second (cosine).
__device__ __forceinline__ void langevin_noise(uint32_t id, unsigned long long step,
                                               uint32_t seed, float xi[3]) {
    const uint4 r = philox(id, step, seed);
    // (q + 1) / 2^24 for a 24-bit q: the sum is exact and so is scaling by a
    // power of two, so the product is the IEEE quotient
    const float scale = 5.9604644775390625e-08f;  // 2^-24
    const float u0 = ((float)(r.x >> 8) + 1.0f) * scale;
    const float u1 = ((float)(r.y >> 8) + 1.0f) * scale;
    const float u2 = ((float)(r.z >> 8) + 1.0f) * scale;
    const float u3 = ((float)(r.w >> 8) + 1.0f) * scale;
    const float ra = sqrtf(-2.0f * logf(u0));
    const float aa = 6.283185307179586f * u1;
    const float rb = sqrtf(-2.0f * logf(u2));
    const float ab = 6.283185307179586f * u3;
    xi[0] = ra * cosf(aa);
    xi[1] = ra * sinf(aa);
    xi[2] = rb * cosf(ab);
}

// The heat current of slot i in the state a step starts from, as the
// sampling kernel takes it: J_i = e_i v_i + T_i v_i / 2 with the canonical
// velocity v_i = v + a dt / 2 (one box, velocities half a kick behind), each
// component to 32.32 fixed point, added into raw.
__device__ __forceinline__ void heat_terms(const Arena& a, const Box& bx, uint32_t i,
                                           const PairSums& s, long long (&raw)[3]) {
    const float acc3[3] = {s.ax, s.ay, s.az};
    double v[3];
#pragma unroll
    for (int c = 0; c < 3; c++) v[c] = canonical_velocity(a, bx, 0, i, c, acc3[c]);
    const double e = 0.5 * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) + (double)s.e_half;
    const double tv[3] = {s.t[0] * v[0] + s.t[3] * v[1] + s.t[4] * v[2],
                          s.t[3] * v[0] + s.t[1] * v[1] + s.t[5] * v[2],
                          s.t[4] * v[0] + s.t[5] * v[1] + s.t[2] * v[2]};
#pragma unroll
    for (int c = 0; c < 3; c++) raw[c] += fixed_raw_f64(e * v[c] + 0.5 * tv[c]);
}

// Component c of langevin_noise alone.
__device__ __forceinline__ float langevin_noise_of(uint32_t c, uint32_t id, unsigned long long step,
                                                   uint32_t seed) {
    const uint4 r = philox(id, step, seed);
    const float scale = 5.9604644775390625e-08f;  // 2^-24
    const float u = ((float)((c < 2u ? r.x : r.z) >> 8) + 1.0f) * scale;
    const float t = ((float)((c < 2u ? r.y : r.w) >> 8) + 1.0f) * scale;
    const float radius = sqrtf(-2.0f * logf(u));
    const float angle = 6.283185307179586f * t;
    return radius * (c == 1u ? sinf(angle) : cosf(angle));
}

// One component's step: both half kicks, then the drift. Every operation
// spelled out, so each kernel gets the same bits.
__device__ __forceinline__ void advance_component(const Box& bx, double side, float acc, float xi,
                                                  double& x, double& v) {
    v = __fma_rn((double)acc, bx.dt, v);
    if (bx.thermostat == 1) {
        x = __fma_rn(v, bx.half_dt, x);
        v = __fma_rn(bx.c1, v, __dmul_rn(bx.c2, (double)xi));
        x = __fma_rn(v, bx.half_dt, x);
    } else {
        x = __fma_rn(v, bx.dt, x);
    }
    x = wrap(x, side);
}

// begin + force_kick of the reference for slot i (lennard_jones.wgsl:204-276,
// 556-574), with its forces in s: the stored velocity is half a kick behind,
// so the two half kicks go on together, then the drift: x += v dt (constant
// energy), or the Langevin A-O-A: x += v dt/2; v = c1 v + c2 xi; x += v dt/2.
// State in f64; the new position goes to the other cache copy (neighbours
// still read this step's). Returns the squared displacement since the last
// list build.
__device__ __forceinline__ float advance_slot(const Arena& a, const Box& bx, uint32_t i,
                                              uint32_t phase, const PairSums& s) {
    const float acc[3] = {s.ax, s.ay, s.az};
    float xi[3] = {0.0f, 0.0f, 0.0f};
    const bool langevin = bx.thermostat == 1;
    if (langevin) langevin_noise(a.id[i], a.glob->step, bx.seed, xi);
    const uint4 snap = a.snap[i];
    const uint32_t sw[3] = {snap.x, snap.y, snap.z};
    uint32_t enc[3];
    float disp2 = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const size_t q = (size_t)k * a.seg + i;
        double x = a.x[q], v = a.v[q];
        advance_component(bx, bx.box[k], acc[k], xi[k], x, v);
        a.x[q] = x;
        a.v[q] = v;
        enc[k] = encode(x, bx.enc[k]);
        const float d = decode_diff(enc[k], sw[k], bx.dec[k]);
        disp2 = __fmaf_rn(d, d, disp2);
    }
    a.cache[phase ^ 1u][i] = make_uint4(enc[0], enc[1], enc[2], 0u);
    return disp2;
}

// The end of a step kernel: the displacement trigger, then, with `next` (or
// a heat-current sample taken), the last block to finish takes the next
// step's rebuild decision and moves the heat-current series on. Called by
// every thread of the block. Only a displacement past the trigger is written
// (the decision asks for no more), so on most steps the block's count is the
// one global round trip, with no fence to wait for.
template <bool HEAT>
__device__ __forceinline__ void finish_step(const Arena& a, bool valid, uint32_t b, float disp2,
                                            cudaGraphConditionalHandle next) {
    const bool over = note_displacement(a, valid, b, disp2);
    if (!next && blockIdx.x == 0 && threadIdx.x == 0) {
        // the next decide finishes this step, and decides anew
        a.glob->pending = 1u;
        a.glob->decided = 0u;
    }
    if (!next && !HEAT) return;
    __shared__ int s_last;
    const int any_over = __syncthreads_or(over);
    if (threadIdx.x == 0) {
        if (any_over) __threadfence();
        s_last = atomicAdd(&a.glob->blocks_done, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (threadIdx.x == 0) {
        a.glob->blocks_done = 0u;
        if (HEAT) a.glob->heat_next += 1u;
    }
    if (next) decide_block(a, next, true, true);
}

// ---- prime (lennard_jones.wgsl:547-553): first forces; the stored velocity
// becomes half a kick behind the given one ----
template <bool SHIFTED_FORCE>
__global__ void __launch_bounds__(kForceThreads) prime_kernel(Arena a,
                                                              const __grid_constant__ CUtensorMap map) {
    count_kernel(a);
    __shared__ __align__(128) Stage st;
    const uint32_t i = blockIdx.x * kForceThreads + threadIdx.x;
    const bool valid = i < a.nslots;
    const Box& bx = a.boxes[valid ? box_of_slot(a, i) : 0u];
    const PairSums s =
        block_pair_sums<SHIFTED_FORCE, false>(st, &map, a, bx, i, valid, a.cache[a.glob->phase]);
    if (!valid) return;
    a.v[i] -= (double)s.ax * bx.half_dt;
    a.v[a.seg + i] -= (double)s.ay * bx.half_dt;
    a.v[2 * (size_t)a.seg + i] -= (double)s.az * bx.half_dt;
}

// ---- one step: begin + force_kick of the reference fused
// (lennard_jones.wgsl:204-276, 556-574) ----
// The stored velocity is half a kick behind, so this kernel's force pass
// applies the previous step's closing half kick and this step's opening half
// kick together, then drifts: x += v dt (constant energy), or the Langevin
// A-O-A: x += v dt/2; v = c1 v + c2 xi; x += v dt/2. State updates in f64.
// The new position goes to the other cache copy (neighbours still read this
// step's), and a squared displacement since the last list build that is past
// the trigger feeds the next step's rebuild decision.
// The block's run of particles when the blocks that share an SM in the
// first wave take neighbouring runs (VLJ_STEP_REMAP): the hardware hands out
// blocks g, g + sms, g + 2 sms, ... to one SM in that wave, so within each
// group of sms x per_sm blocks the order is transposed; blocks past the last
// whole group keep their own run. A bijection on [0, n).
__device__ __forceinline__ uint32_t resident_neighbours(uint32_t b, uint32_t n, uint32_t sms,
                                                       uint32_t per_sm) {
    const uint32_t w = sms * per_sm;
    if (w == 0u || b >= n / w * w) return b;
    const uint32_t t = b % w;
    return b - t + (t % sms) * per_sm + t / sms;
}

// THREADS particles per block (Arena::step_threads, tuned per replica set
// by virial_lj.tune_batch; the TMA tile ring needs kForceThreads).
template <bool SHIFTED_FORCE, bool HEAT, int THREADS>
__global__ void __launch_bounds__(THREADS, HEAT ? 1 : kStepMinBlocks * 128 / THREADS) step_kernel(Arena a,
                                                             const __grid_constant__ CUtensorMap map,
                                                             cudaGraphConditionalHandle next) {
    static_assert(VLJ_LIST_STREAM || THREADS == kForceThreads, "TMA tiles need kForceThreads");
    count_kernel(a);
    __shared__ __align__(128) Stage st;
#if VLJ_STEP_REMAP
    const uint32_t vb = resident_neighbours(blockIdx.x, gridDim.x, a.remap_sms, a.remap_per_sm);
#else
    const uint32_t vb = blockIdx.x;
#endif
    const uint32_t i = vb * THREADS + threadIdx.x;
    const bool valid = i < a.nslots;
    const uint32_t phase = a.glob->phase;
    const uint32_t b = valid ? box_of_slot(a, i) : 0u;
    const Box& bx = a.boxes[b];
    const PairSums s =
        block_pair_sums<SHIFTED_FORCE, false, HEAT>(st, &map, a, bx, i, valid, a.cache[phase]);
    if (HEAT) {
        const uint32_t sample = a.glob->heat_next;
        long long raw[3] = {0, 0, 0};
        if (valid) heat_terms(a, bx, i, s, raw);
        block_sum_series(a, raw, sample);
    }
    float disp2 = 0.0f;
    if (valid) disp2 = advance_slot(a, bx, i, phase, s);
    finish_step<HEAT>(a, valid, b, disp2, next);
}

// ---- one step with LANES lanes per particle, for grids that leave the chip
// idle at one (lanes_for): a lone warp cannot hide its latency behind others,
// so its chain of rows and gathers is what the step takes. The list's parts
// go to the lanes (lane_pair_sums); with four lanes or more, lane c < 3 then
// steps component c, its state loaded before the forces. The same step as
// step_kernel to the bit (no heat-current sample). ----
template <bool SHIFTED_FORCE, int LANES, int THREADS>
__global__ void __launch_bounds__(THREADS) step_kernel_lanes(Arena a, cudaGraphConditionalHandle next) {
    count_kernel(a);
    constexpr uint32_t kPer = THREADS / LANES;  // particles per block
    const uint32_t sub = threadIdx.x % LANES;
    const uint32_t i = blockIdx.x * kPer + threadIdx.x / LANES;
    const bool valid = i < a.nslots;
    const uint32_t phase = a.glob->phase;
    const uint32_t b = valid ? box_of_slot(a, i) : 0u;
    const Box& bx = a.boxes[b];
    if constexpr (LANES >= 4) {
        const bool mine = valid && sub < 3u;
        const size_t q = (size_t)sub * a.seg + i;
        double x = 0.0, v = 0.0;
        uint32_t sw = 0, id = 0;
        if (mine) {
            x = a.x[q];
            v = a.v[q];
            sw = reinterpret_cast<const uint32_t*>(a.snap + i)[sub];
            if (bx.thermostat == 1) id = a.id[i];
        }
        const PairSums s = lane_pair_sums<SHIFTED_FORCE, LANES>(a, bx, i, valid, sub, a.cache[phase]);
        float d = 0.0f;
        if (mine) {
            const float xi = bx.thermostat == 1 ? langevin_noise_of(sub, id, a.glob->step, bx.seed) : 0.0f;
            advance_component(bx, bx.box[sub], sub == 0u ? s.ax : (sub == 1u ? s.ay : s.az), xi, x, v);
            a.x[q] = x;
            a.v[q] = v;
            const uint32_t enc = encode(x, bx.enc[sub]);
            d = decode_diff(enc, sw, bx.dec[sub]);
            reinterpret_cast<uint32_t*>(a.cache[phase ^ 1u] + i)[sub] = enc;
        }
        float disp2 = 0.0f;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const float dk = __shfl_sync(0xffffffffu, d, k, LANES);
            disp2 = __fmaf_rn(dk, dk, disp2);
        }
        finish_step<false>(a, valid, b, disp2, next);
    } else {
        const PairSums s = lane_pair_sums<SHIFTED_FORCE, LANES>(a, bx, i, valid, sub, a.cache[phase]);
        const bool mine = valid && sub == 0u;
        finish_step<false>(a, mine, b, mine ? advance_slot(a, bx, i, phase, s) : 0.0f, next);
    }
}

// ---- one step over cell tiles: the same step as step_kernel, with the
// neighbour positions staged in shared memory ----
// A block takes one brick (a run of cells along x in one row of the box; the
// bricks tile the box) and stages its tile -- the encoded positions of every
// particle in the nine neighbour rows of those cells, each row one or two
// runs of the sorted order -- in shared memory, 16 B a particle. Its threads
// take the brick's home particles in sorted order; each walks its list as
// 16-bit tile indices (eight to a 16-byte row, streamed past L1), so every
// neighbour read is a shared-memory load instead of a scattered global
// gather. The list order and the pair arithmetic are step_kernel's, so the
// step is the same to the bit. A brick whose tile would not fit in
// a.tile_cap entries walks the slot list with global gathers instead.
template <bool SHIFTED_FORCE, bool HEAT>
__global__ void __launch_bounds__(kBlock) tile_step_kernel(Arena a, cudaGraphConditionalHandle next) {
    count_kernel(a);
    extern __shared__ __align__(16) uint4 s_tile[];
    __shared__ uint32_t s_run[9][3];  // per tile row: first run's sorted start, its length, second run's start
    __shared__ uint32_t s_base[10];   // tile index of each row's first particle; [9]: the tile's size
    __shared__ uint32_t s_home[3];    // the brick's home particles' sorted range; [2]: first one's tile index
    const uint32_t phase = a.glob->phase;
    const uint4* __restrict__ cur = a.cache[phase];
    const Box& bx = a.boxes[0];
    const Brick k = brick_at(bx, blockIdx.x - bx.brick_base);
    const uint32_t* __restrict__ cs = a.cell_start;
    if (threadIdx.x < 9u) {
        const uint32_t row = tile_row_cell(bx, k, threadIdx.x);
        const uint32_t nx = bx.cells[0], end = k.x_start + k.rx;
        const uint32_t first = cs[row + k.x_start];
        const uint32_t len1 = cs[row + min(end, nx)] - first;
        const uint32_t len2 = end > nx ? cs[row + end - nx] - cs[row] : 0u;
        s_run[threadIdx.x][0] = first;
        s_run[threadIdx.x][1] = len1;
        s_run[threadIdx.x][2] = cs[row];
        s_base[threadIdx.x + 1] = len1 + len2;
    } else if (threadIdx.x == 32u) {
        const uint32_t row = tile_row_cell(bx, k, 4u);
        s_home[0] = cs[row + k.x0];
        s_home[1] = cs[row + k.x0 + k.w];
        s_home[2] = tile_row_prefix(cs, bx, k, row, tile_col(bx, k, k.x0, 0));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        s_base[0] = 0u;
        for (int r = 0; r < 9; r++) s_base[r + 1] += s_base[r];
    }
    __syncthreads();
    const uint32_t tile_size = s_base[9];
    // until a build has written the tile lists for these bricks (tiles just
    // switched on or resized), every block takes the slot list
    const bool staged = tile_size <= a.tile_cap && a.glob->tiles_ready != 0u;
#if VLJ_TILE_F32
    // the tile as f32 offsets from the brick's centre (encoded)
    const uint32_t org[3] = {
        encode(((double)k.x0 + 0.5 * (double)k.w) * (double)bx.cell_size_f[0], bx.enc[0]),
        encode(((double)k.y + 0.5) * (double)bx.cell_size_f[1], bx.enc[1]),
        encode(((double)k.z + 0.5) * (double)bx.cell_size_f[2], bx.enc[2])};
    float4* s_tilef = reinterpret_cast<float4*>(s_tile);
#endif
    if (staged) {
        for (uint32_t t = threadIdx.x; t < tile_size; t += blockDim.x) {
            uint32_t rho = 0;
            while (t >= s_base[rho + 1]) rho++;
            const uint32_t q = t - s_base[rho];
            const uint32_t p = q < s_run[rho][1] ? s_run[rho][0] + q : s_run[rho][2] + (q - s_run[rho][1]);
#if VLJ_TILE_F32
            const uint4 w = cur[a.sorted[p]];
            s_tilef[t] = make_float4(decode_diff(w.x, org[0], bx.dec[0]), decode_diff(w.y, org[1], bx.dec[1]),
                                     decode_diff(w.z, org[2], bx.dec[2]), 0.0f);
#else
            s_tile[t] = cur[a.sorted[p]];
#endif
        }
    }
    __syncthreads();
    const uint32_t h0 = s_home[0], h1 = s_home[1];
    const uint32_t own0 = s_base[4] + s_home[2] - h0;  // tile index of home p: own0 + p
    const float dec0 = bx.dec[0], dec1 = bx.dec[1], dec2 = bx.dec[2];
    const float fshift = bx.force_shift;
    const uint32_t rc2_bits_m1 = __float_as_uint(bx.rc2) - 1u;
    float disp2 = 0.0f;
    long long raw[3] = {0, 0, 0};
    const uint32_t sample = HEAT ? a.glob->heat_next : 0u;
    for (uint32_t p = h0 + threadIdx.x; p < h1; p += blockDim.x) {
        const uint32_t i = a.sorted[p];
        const uint32_t cnt = a.list_count[i];
        PairSums s = {};
        if (staged) {
#if VLJ_TILE_F32
            const float4 own = s_tilef[own0 + p];
            // a 16-bit row is two rows of the slot list: a part of the force sum
            auto add = [&](const float4 pj) {
                pair_terms_rel<SHIFTED_FORCE, HEAT>(s, own, pj, bx, rc2_bits_m1, fshift);
            };
            auto fetch = [&](uint32_t t) { return s_tilef[t]; };
            using Pos = float4;
#else
            const uint4 own = s_tile[own0 + p];
            auto add = [&](const uint4 pj) {
                pair_terms<SHIFTED_FORCE, false, HEAT>(s, own, pj, bx, dec0, dec1, dec2,
                                                       rc2_bits_m1, fshift);
            };
            auto fetch = [&](uint32_t t) { return s_tile[t]; };
            using Pos = uint4;
#endif
            const uint4* rowp = reinterpret_cast<const uint4*>(a.list16) + p;
            const uint32_t rows = (cnt + 7u) / 8u;
            uint4 nxt = rows ? load_row_streaming(rowp) : make_uint4(0u, 0u, 0u, 0u);
#if VLJ_TILE_PIPE
            // the next row's eight neighbours are read while this row's pairs
            // are computed
            Pos q[8];
            if (rows) {
                const uint4 e = nxt;
                if (rows > 1u) nxt = load_row_streaming(rowp + a.seg);
                q[0] = fetch(e.x & 0xffffu); q[1] = fetch(e.x >> 16);
                q[2] = fetch(e.y & 0xffffu); q[3] = fetch(e.y >> 16);
                q[4] = fetch(e.z & 0xffffu); q[5] = fetch(e.z >> 16);
                q[6] = fetch(e.w & 0xffffu); q[7] = fetch(e.w >> 16);
            }
            for (uint32_t row = 0; row < rows; row++) {
                Pos c[8];
#pragma unroll
                for (int m = 0; m < 8; m++) c[m] = q[m];
                if (row + 1u < rows) {
                    const uint4 e = nxt;
                    if (row + 2u < rows) nxt = load_row_streaming(rowp + (size_t)(row + 2u) * a.seg);
                    q[0] = fetch(e.x & 0xffffu); q[1] = fetch(e.x >> 16);
                    q[2] = fetch(e.y & 0xffffu); q[3] = fetch(e.y >> 16);
                    q[4] = fetch(e.z & 0xffffu); q[5] = fetch(e.z >> 16);
                    q[6] = fetch(e.w & 0xffffu); q[7] = fetch(e.w >> 16);
                }
#pragma unroll
                for (int m = 0; m < 8; m++) add(c[m]);
                end_part(s);
            }
#else
            for (uint32_t row = 0; row < rows; row++) {
                const uint4 e = nxt;
                if (row + 1u < rows) nxt = load_row_streaming(rowp + (size_t)(row + 1u) * a.seg);
                add(fetch(e.x & 0xffffu));
                add(fetch(e.x >> 16));
                add(fetch(e.y & 0xffffu));
                add(fetch(e.y >> 16));
                add(fetch(e.z & 0xffffu));
                add(fetch(e.z >> 16));
                add(fetch(e.w & 0xffffu));
                add(fetch(e.w >> 16));
                end_part(s);
            }
#endif
        } else {
            const uint4 own = cur[i];
            const uint4* rowp = reinterpret_cast<const uint4*>(a.list) + i;
            const uint32_t rows = (cnt + 3u) / 4u;
            for (uint32_t row = 0; row < rows; row++) {
                const uint4 e = load_row_streaming(rowp + (size_t)row * a.seg);
                const uint4 p0 = __ldg(cur + e.x), p1 = __ldg(cur + e.y);
                const uint4 p2 = __ldg(cur + e.z), p3 = __ldg(cur + e.w);
                for (const uint4& pj : {p0, p1, p2, p3})
                    pair_terms<SHIFTED_FORCE, false, HEAT>(s, own, pj, bx, dec0, dec1, dec2, rc2_bits_m1, fshift);
                if (row & 1u) end_part(s);
            }
        }
        end_part(s);
        if (HEAT) heat_terms(a, bx, i, s, raw);
        disp2 = fmaxf(disp2, advance_slot(a, bx, i, phase, s));
    }
    if (HEAT) block_sum_series(a, raw, sample);
    finish_step<HEAT>(a, true, 0u, disp2, next);
}

// ---- measure (lennard_jones.wgsl:576-626) ----
// Per particle: half of each pair energy and virial, neighbours within
// 1.5 sigma, the velocity at the step (stored velocity plus the closing half
// kick), kinetic energy and momentum in f64. Each value goes to 32.32 fixed
// point scaled like the reference and is summed exactly.
// Several lanes per particle on small grids, as in the step (lanes_for).
template <bool SHIFTED_FORCE, int LANES>
__global__ void __launch_bounds__(kForceThreads) measure_kernel(Arena a,
                                                                const __grid_constant__ CUtensorMap map) {
    count_kernel(a);
    __shared__ __align__(128) Stage st;
    constexpr uint32_t kPer = kForceThreads / LANES;
    const uint32_t i = blockIdx.x * kPer + threadIdx.x / LANES;
    const uint32_t b = i < a.nslots ? box_of_slot(a, i) : 0u;
    const Box& bx = a.boxes[b];
    const bool valid = i < a.nslots && threadIdx.x % LANES == 0u;  // lane 0 keeps the particle
    PairSums s;
    if constexpr (LANES > 1)
        s = lane_pair_sums<SHIFTED_FORCE, LANES, true>(a, bx, i, i < a.nslots, threadIdx.x % LANES,
                                                       a.cache[a.glob->phase]);
    else
        s = block_pair_sums<SHIFTED_FORCE, true>(st, &map, a, bx, i, valid, a.cache[a.glob->phase]);
    long long v[kSlots] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (valid) {
        const float acc[3] = {s.ax, s.ay, s.az};
        double vel[3], ke = 0.0;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            vel[k] = canonical_velocity(a, bx, b, i, k, acc[k]);
            ke += vel[k] * vel[k];
        }
        ke *= 0.5;
        const double es = (double)bx.energy_scale, ms = (double)bx.momentum_scale;
        v[0] = fixed_raw_f64(ke * es);
        v[1] = fixed_raw_f32(s.pe * bx.energy_scale) + fixed_raw_f32(s.pe_lo * bx.energy_scale);
        v[2] = fixed_raw_f32(s.w * bx.energy_scale) + fixed_raw_f32(s.w_lo * bx.energy_scale);
#pragma unroll
        for (int k = 0; k < 3; k++) v[3 + k] = fixed_raw_f64(vel[k] * ms);
        v[6] = s.near >= bx.near_count ? (1ll << 32) : 0ll;
        a.pe_half[2 * i] = s.pe;
        a.pe_half[2 * i + 1] = s.pe_lo;
        a.w_half[2 * i] = s.w;
        a.w_half[2 * i + 1] = s.w_lo;
        a.vel4[i] = make_float4((float)vel[0], (float)vel[1], (float)vel[2], (float)s.near);
    }
    block_sum_slots(a, valid, b, blockIdx.x * kPer, v);
}

// ---- particles out (lennard_jones.rs:1354-1374; input order) ----
// Slots first .. first + count - 1 (one box, or a replica's): the forces for
// the canonical velocity and the neighbours within 1.5 sigma, with no
// energies, then positions and velocities straight into the particles as the
// API passes them, at out[id]. A measurement in its place computed every
// pair's energy in f64 for nothing (95 us at 256,000 atoms, 42 us so).
template <bool SHIFTED_FORCE, int LANES>
__global__ void __launch_bounds__(kForceThreads) read_kernel(Arena a, const __grid_constant__ CUtensorMap map,
                                                             uint32_t first, uint32_t count,
                                                             double* __restrict__ out) {
    count_kernel(a);
    __shared__ __align__(128) Stage st;
    const uint32_t sub = threadIdx.x % LANES;
    // the grid starts at the slot of its first whole block
    const uint32_t block0 = LANES == 1 ? first / kForceThreads : 0u;
    const uint32_t from = LANES == 1 ? block0 * kForceThreads : first;
    const uint32_t i = from + blockIdx.x * (kForceThreads / LANES) + threadIdx.x / LANES;
    const bool valid = i >= first && i - first < count;
    const uint32_t b = valid ? box_of_slot(a, i) : 0u;
    const Box& bx = a.boxes[b];
    PairSums s;
    if constexpr (LANES > 1)
        s = lane_pair_sums<SHIFTED_FORCE, LANES, false, true>(a, bx, i, valid, sub, a.cache[a.glob->phase]);
    else
        s = block_pair_sums<SHIFTED_FORCE, false, false, true>(st, &map, a, bx, i, valid,
                                                               a.cache[a.glob->phase], block0);
    if (!valid || sub != 0u) return;
    const double v[3] = {canonical_velocity(a, bx, b, i, 0, s.ax), canonical_velocity(a, bx, b, i, 1, s.ay),
                         canonical_velocity(a, bx, b, i, 2, s.az)};
    a.vel4[i] = make_float4((float)v[0], (float)v[1], (float)v[2], (float)s.near);
    const uint32_t id = a.id[i];
    if (id >= count) {
        atomicCAS(&a.glob->fault, 0u, kFaultBadId);
        return;
    }
    double2* p = reinterpret_cast<double2*>(out) + 3 * (size_t)id;
    p[0] = make_double2(a.x[i], a.x[(size_t)a.seg + i]);
    p[1] = make_double2(a.x[2 * (size_t)a.seg + i], v[0]);
    p[2] = make_double2(v[1], v[2]);
}

// ---- steps on canonical velocities: Nose-Hoover (lennard_jones.wgsl:309-397)
// and the heat exchange (lennard_jones.wgsl:732-893); host order
// lennard_jones.rs:1108-1138 ----
// One box. A step runs begin (Nose-Hoover's pending end-half scale s2 of the
// last step and this step's start-half scale s1, the half kick, the drift),
// the decision and rebuild, then canon_force (forces, the closing half kick,
// and the end-of-step sums: the kinetic energy for Nose-Hoover, the slab sums
// for the exchange; the block that finishes last turns them into the
// thermostat update or the exchange coefficients), then for the exchange
// hex_apply. The stored velocity is canonical (before Nose-Hoover's s2).

// begin: every thread takes the start half step from the same state, so all
// of them compute the same s1; the box's first thread stores the result.
__global__ void __launch_bounds__(kBlock) begin_kernel(Arena a) {
    chain_next();
    chain_wait();
    count_kernel(a);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < a.nslots;
    const uint32_t phase = a.glob->phase;
    const uint32_t b = valid ? box_of_slot(a, i) : 0u;
    const Box& bx = a.boxes[b];
    float disp2 = 0.0f;
    if (valid) {
        double s2 = 1.0, s1 = 1.0;  // exact no-ops without Nose-Hoover
        if (bx.thermostat == 2) {
            const Thermo& t = a.nh[b];
            double xi = t.xi_m, eta = t.eta_m, ke = t.ke_m;
            s2 = t.scale;
            s1 = nh_half(bx, xi, eta, ke);
            if (i == bx.first) {
                a.nh[b].xi_s = xi;
                a.nh[b].eta_s = eta;
            }
        }
        const float4 f = a.acc[i];
        const float acc[3] = {f.x, f.y, f.z};
        const uint4 snap = a.snap[i];
        const uint32_t sw[3] = {snap.x, snap.y, snap.z};
        uint32_t enc[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const size_t q = (size_t)k * a.seg + i;
            // the two half steps' scalings in turn, then the half kick
            const double v = a.v[q] * s2 * s1 + (double)acc[k] * bx.half_dt;
            const double x = wrap(a.x[q] + v * bx.dt, bx.box[k]);
            a.x[q] = x;
            a.v[q] = v;
            enc[k] = encode(x, bx.enc[k]);
            const float d = decode_diff(enc[k], sw[k], bx.dec[k]);
            disp2 = __fmaf_rn(d, d, disp2);
        }
        a.cache[phase ^ 1u][i] = make_uint4(enc[0], enc[1], enc[2], 0u);
    }
    note_displacement(a, valid, b, disp2);
    if (i == 0) a.glob->pending = 1u;
}

// The exchange slab of height z (f32, as the reference): 0 hot, 1 cold, 2 neither.
__device__ __forceinline__ int hex_slab(const Box& bx, double z) {
    const float zf = (float)z;
    if (zf >= bx.hex_slabs[0] && zf < bx.hex_slabs[1]) return 0;
    if (zf >= bx.hex_slabs[2] && zf < bx.hex_slabs[3]) return 1;
    return 2;
}

// The exchange's per-slab scale and eHEX/a correction coefficients from the
// slab sums (lennard_jones.wgsl:804-856), in f64; clears the sums.
__device__ void hex_coefficients(const Box& bx, Exchange* h) {
    const double one = 4294967296.0;
    const double es = (double)bx.energy_scale, ms = (double)bx.momentum_scale;
    const double dt = bx.dt, dt3 = dt * dt * dt;
    for (int sl = 0; sl < 2; sl++) {
        long long raw[9];
        for (int k = 0; k < 9; k++) {
            raw[k] = (long long)h->sums[sl][k];
            h->sums[sl][k] = 0ull;
        }
        const double m = (double)raw[0] / one;
        double p[3], f[3];
        for (int k = 0; k < 3; k++) {
            p[k] = (double)raw[1 + k] / one / ms;
            f[k] = (double)raw[6 + k] / one / ms;
        }
        const double v2 = (double)raw[4] / one / es, fv = (double)raw[5] / one / es;
        double com[3] = {0.0, 0.0, 0.0}, mf[3] = {0.0, 0.0, 0.0};
        double sm1 = 0.0, cv = 0.0, cf = 0.0;
        if (m > 0.0) {
            for (int k = 0; k < 3; k++) {
                com[k] = p[k] / m;
                mf[k] = f[k] / m;
            }
            // kinetic energy about the centre of mass
            const double kinetic = 0.5 * v2 - 0.5 * (p[0] * p[0] + p[1] * p[1] + p[2] * p[2]) / m;
            const double energy = (sl == 0 ? 1.0 : -1.0) * bx.hex_energy;
            const double flux = energy / dt;
            const double x = energy / kinetic;
            sm1 = x / (1.0 + sqrt(1.0 + x));  // sqrt(1 + x) - 1
            const double power = fv - (f[0] * com[0] + f[1] * com[1] + f[2] * com[2]);
            cv = dt3 * flux / (2.0 * kinetic * kinetic) * (flux / 48.0 + power / 6.0);
            cf = dt3 * flux / (12.0 * kinetic);
        }
        for (int k = 0; k < 3; k++) {
            h->com[sl][k] = com[k];
            h->mean_f[sl][k] = mf[k];
        }
        h->s_minus_1[sl] = sm1;
        h->c_v[sl] = cv;
        h->c_f[sl] = cf;
    }
}

// Sum of a 64-bit integer over the warp, in every lane.
__device__ __forceinline__ long long warp_sum(long long x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// canon_force: forces from the list, stored; the closing half kick (not for
// kPrime); the end-of-step sums in 32.32 fixed point, added per block, and in
// the last block to finish the Nose-Hoover update or the exchange
// coefficients.
// The sums go through warp shuffles, one shared word per warp: shared memory
// has no 64-bit add, so one atomicAdd per particle is a compare-and-swap loop
// in which the whole block takes turns on one address (the exchange's pass
// took 45 us that way at 2,462 atoms, 16.4 us so; Nose-Hoover's 18.5 us at
// 15,600 atoms, 12.9 us so).
template <bool SHIFTED_FORCE, int PASS, int LANES>
__global__ void __launch_bounds__(kForceThreads) canon_force_kernel(Arena a,
                                                                    const __grid_constant__ CUtensorMap map) {
    chain_next();
    count_kernel(a);
    constexpr int kWarps = kForceThreads / 32;
    __shared__ __align__(128) Stage st;
    __shared__ long long s_sum[kWarps][2][9];
    __shared__ int s_last;
    const uint32_t i = blockIdx.x * (kForceThreads / LANES) + threadIdx.x / LANES;
    const bool valid = i < a.nslots && threadIdx.x % LANES == 0u;  // lane 0 keeps the particle
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const Box& bx = a.boxes[0];
    double v[3] = {0.0, 0.0, 0.0};
    if (valid) {
#pragma unroll
        for (int k = 0; k < 3; k++) v[k] = a.v[(size_t)k * a.seg + i];
    }
    const int sl = PASS == kExchange && valid ? hex_slab(bx, a.x[2 * (size_t)a.seg + i]) : 2;
    PairSums s;
    if constexpr (LANES > 1)
        s = lane_pair_sums<SHIFTED_FORCE, LANES>(a, bx, i, i < a.nslots, threadIdx.x % LANES,
                                                 a.cache[a.glob->phase]);
    else
        s = block_pair_sums<SHIFTED_FORCE, false>(st, &map, a, bx, i, valid, a.cache[a.glob->phase]);
    const float acc[3] = {s.ax, s.ay, s.az};
    if (valid) {
        a.acc[i] = make_float4(acc[0], acc[1], acc[2], 0.0f);
        if (PASS != kPrime) {
#pragma unroll
            for (int k = 0; k < 3; k++) {
                v[k] += (double)acc[k] * bx.half_dt;
                a.v[(size_t)k * a.seg + i] = v[k];
            }
        }
    }
    if (PASS == kKick) return;
    const double es = (double)bx.energy_scale, ms = (double)bx.momentum_scale;
    if (PASS == kExchange) {
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const unsigned in = __ballot_sync(0xffffffffu, sl == k);
            if (in == 0u) {
                // most warps hold no particle of a slab
                if (lane < 9u) s_sum[warp][k][lane] = 0ll;
                continue;
            }
            long long raw[8];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                raw[c] = fixed_raw_f64(v[c] * ms);
                raw[5 + c] = fixed_raw_f64((double)acc[c] * ms);
            }
            raw[3] = fixed_raw_f64((v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) * es);
            raw[4] = fixed_raw_f64(
                ((double)acc[0] * v[0] + (double)acc[1] * v[1] + (double)acc[2] * v[2]) * es);
            if (lane == 0) s_sum[warp][k][0] = (long long)__popc(in) << 32;
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const long long t = warp_sum(sl == k ? raw[c] : 0ll);
                if (lane == 0) s_sum[warp][k][1 + c] = t;
            }
        }
    } else {
        const long long t =
            warp_sum(valid ? fixed_raw_f64(0.5 * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) * es) : 0ll);
        if (lane == 0) s_sum[warp][0][0] = t;
    }
    __syncthreads();
    if (threadIdx.x < (PASS == kExchange ? 18u : 1u)) {
        const uint32_t sl = threadIdx.x / 9u, k = threadIdx.x % 9u;
        long long t = 0;
        for (int w = 0; w < kWarps; w++) t += s_sum[w][sl][k];
        unsigned long long* to = PASS == kExchange ? &a.hex->sums[sl][k] : &a.nh->ke_raw;
        if (t) atomicAdd(to, (unsigned long long)t);
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t* done = PASS == kExchange ? &a.hex->blocks_done : &a.nh->blocks_done;
        __threadfence();
        s_last = atomicAdd(done, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!s_last || threadIdx.x != 0) return;
    // every other block's sums are in
    __threadfence();
    if (PASS == kExchange) {
        a.hex->blocks_done = 0u;
        hex_coefficients(bx, a.hex);
        return;
    }
    Thermo* t = a.nh;
    const long long total = (long long)atomicExch(&t->ke_raw, 0ull);
    t->blocks_done = 0u;
    double ke = (double)total / 4294967296.0 / (double)bx.energy_scale;
    if (PASS == kPrime) {
        t->ke_m = ke;
        t->scale = 1.0;
        return;
    }
    double xi = t->xi_s, eta = t->eta_s;
    const double s2 = nh_half(bx, xi, eta, ke);
    t->xi_m = xi;
    t->eta_m = eta;
    t->ke_m = ke;
    t->scale = s2;
}

// hex_apply (lennard_jones.wgsl:858-893): in each slab, the position
// correction -dt^3 E_i from the velocity before scaling, then
// v <- v + (s - 1)(v - v_com); the moved positions go back into the current
// position copy.
__global__ void __launch_bounds__(kBlock) hex_apply_kernel(Arena a) {
    chain_next();
    chain_wait();
    count_kernel(a);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.nslots) return;
    const Box& bx = a.boxes[0];
    const int sl = hex_slab(bx, a.x[2 * (size_t)a.seg + i]);
    if (sl == 2) return;
    const Exchange& h = *a.hex;
    const float4 f = a.acc[i];
    const float acc[3] = {f.x, f.y, f.z};
    uint32_t enc[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const size_t q = (size_t)k * a.seg + i;
        const double v = a.v[q];
        const double rel = v - h.com[sl][k];
        const double shift = h.c_v[sl] * rel - h.c_f[sl] * ((double)acc[k] - h.mean_f[sl][k]);
        const double x = wrap(a.x[q] - shift, bx.box[k]);
        a.x[q] = x;
        a.v[q] = v + h.s_minus_1[sl] * rel;
        enc[k] = encode(x, bx.enc[k]);
    }
    a.cache[a.glob->phase][i] = make_uint4(enc[0], enc[1], enc[2], 0u);
}

// Canonical velocities back to half a kick behind, with the stored forces.
__global__ void __launch_bounds__(kBlock) half_kick_back_kernel(Arena a) {
    count_kernel(a);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.nslots) return;
    const Box& bx = a.boxes[0];
    const float4 f = a.acc[i];
    a.v[i] -= (double)f.x * bx.half_dt;
    a.v[a.seg + i] -= (double)f.y * bx.half_dt;
    a.v[2 * (size_t)a.seg + i] -= (double)f.z * bx.half_dt;
}

// ---- FP32 calibration: eight independent FMA chains per thread, so the
// FMA pipes stay full; 2 flops per FMA ----
__global__ void __launch_bounds__(kBlock) fp32_peak_kernel(float* out, int iters) {
    float x[8];
#pragma unroll
    for (int k = 0; k < 8; k++) x[k] = (float)(threadIdx.x + k) * 1e-3f;
    const float m = 0.999999f, c = 1e-6f;
    for (int it = 0; it < iters; it++) {
#pragma unroll
        for (int k = 0; k < 8; k++) x[k] = fmaf(x[k], m, c);
    }
    float t = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; k++) t += x[k];
    if (t == 12345.678f) out[blockIdx.x] = t;  // keeps the chains live
}

// ---- the noise stream as the step kernel draws it, for known-answer checks:
// Philox-4x32-10 of each (counter, key), and the Langevin noise of
// (id = ctr.x, step = ctr.y + 2^32 ctr.z, seed = key.x) ----
__global__ void __launch_bounds__(kBlock) philox_check_kernel(const uint4* __restrict__ ctr,
                                                              const uint2* __restrict__ key,
                                                              uint32_t n, uint4* __restrict__ out,
                                                              float4* __restrict__ noise) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint4 c = ctr[k];
    const uint2 q = key[k];
    out[k] = philox4x32_10(c, q);
    float xi[3];
    langevin_noise(c.x, (unsigned long long)c.y | ((unsigned long long)c.z << 32), q.x, xi);
    noise[k] = make_float4(xi[0], xi[1], xi[2], 0.0f);
}

cudaError_t launch_philox_check(const uint4* ctr, const uint2* key, uint32_t n, uint4* out,
                                float4* noise, cudaStream_t s) {
    philox_check_kernel<<<blocks_for(n), kBlock, 0, s>>>(ctr, key, n, out, noise);
    return after_launch();
}

// ---- launchers ----
static unsigned particle_blocks(const Arena& a) {
    return blocks_for(a.nslots, kForceThreads);
}

// With the list streamed from global memory the force kernels use no shared
// memory to speak of; ask for the largest L1 (it caches the gathers).
#ifndef VLJ_L1_CARVEOUT
#define VLJ_L1_CARVEOUT 4  // shared-memory carve-out hint, percent of the maximum (tuned)
#endif
template <class K>
static void prefer_l1(K kernel) {
#if VLJ_LIST_STREAM
    cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, VLJ_L1_CARVEOUT);
#else
    (void)kernel;
#endif
}

static void prefer_l1_once() {
    static bool done = false;
    if (done) return;
    done = true;
    prefer_l1(prime_kernel<true>);
    prefer_l1(prime_kernel<false>);
}

cudaError_t launch_prime(const Arena& a, const CUtensorMap& map, bool shifted_force,
                         cudaStream_t s) {
    prefer_l1_once();
    if (shifted_force)
        prime_kernel<true><<<particle_blocks(a), kForceThreads, 0, s>>>(a, map);
    else
        prime_kernel<false><<<particle_blocks(a), kForceThreads, 0, s>>>(a, map);
    return after_launch();
}

// Lanes per particle of a force pass over n particles: as many as keep the
// grid within VLJ_LANE_THREADS_PER_SM threads an SM. There a lane more
// shortens the chain a warp waits for; past that the warps already cover each
// other's waits, and the split's shuffles and padded rounds cost more. Pass
// time inside a graph with 1 / 2 / 4 / 8 lanes (us): 1,000 atoms 8.9 / 13.6 /
// 7.7 / 6.2; 2,462 (exchange) 15.9 / 12.3 / 10.5 / 9.8; 15,600 (Nose-Hoover)
// 17.6 / 9.5 / 9.3 / 10.8; 32,768 at rho 0.4 10.1 / 9.4 / 10.0 / 13.1; 64,000
// 15.2 / 17.8 / 21.7 / 29.6; 256,000 43 / 55 / 71 / 111.
static int lanes_for(uint32_t n) {
#ifdef VLJ_LANES_FORCE
    return VLJ_LANES_FORCE;
#endif
    const uint64_t room = (uint64_t)sm_count() * VLJ_LANE_THREADS_PER_SM;
    for (int lanes = 8; lanes > 1; lanes /= 2)
        if ((uint64_t)n * (unsigned)lanes <= room) return lanes;
    return 1;
}

// The same, unless a test asks for a number of lanes.
static int lanes_of(const Arena& a, uint32_t n) { return a.step_lanes ? (int)a.step_lanes : lanes_for(n); }

template <bool SF, int LANES, int THREADS>
static void launch_lanes(const Arena& a, cudaStream_t s, cudaGraphConditionalHandle next) {
    static bool carved = false;
    if (!carved) {
        carved = true;
        prefer_l1(step_kernel_lanes<SF, LANES, THREADS>);
    }
    step_kernel_lanes<SF, LANES, THREADS>
        <<<blocks_for(a.nslots, THREADS / LANES), THREADS, 0, s>>>(a, next);
}

template <bool SF, int THREADS>
static void launch_step_lanes(const Arena& a, int lanes, cudaStream_t s,
                              cudaGraphConditionalHandle next) {
    if (lanes == 8) launch_lanes<SF, 8, THREADS>(a, s, next);
    else if (lanes == 4) launch_lanes<SF, 4, THREADS>(a, s, next);
    else launch_lanes<SF, 2, THREADS>(a, s, next);
}

template <int THREADS>
static cudaError_t launch_step_kernel(const Arena& a, const CUtensorMap& map, bool shifted_force,
                                      cudaStream_t s, cudaGraphConditionalHandle next, bool heat) {
    static bool carved = false;
    if (!carved) {
        carved = true;
        prefer_l1(step_kernel<true, false, THREADS>);
        prefer_l1(step_kernel<false, false, THREADS>);
        prefer_l1(step_kernel<true, true, THREADS>);
        prefer_l1(step_kernel<false, true, THREADS>);
    }
#if VLJ_LIST_STREAM
    const int lanes = heat ? 1 : lanes_of(a, a.nslots);
    if (lanes > 1) {
        if (shifted_force) launch_step_lanes<true, THREADS>(a, lanes, s, next);
        else launch_step_lanes<false, THREADS>(a, lanes, s, next);
        return after_launch();
    }
#endif
    const unsigned blocks = blocks_for(a.nslots, THREADS);
    Arena r = a;
#if VLJ_STEP_REMAP
    static int per_sm = 0;
    if (!per_sm &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, step_kernel<true, false, THREADS>,
                                                      THREADS, 0) != cudaSuccess)
        per_sm = 0;
    r.remap_sms = (uint32_t)sm_count();
    r.remap_per_sm = (uint32_t)per_sm;
#endif
    if (shifted_force) {
        if (heat) step_kernel<true, true, THREADS><<<blocks, THREADS, 0, s>>>(r, map, next);
        else step_kernel<true, false, THREADS><<<blocks, THREADS, 0, s>>>(r, map, next);
    } else {
        if (heat) step_kernel<false, true, THREADS><<<blocks, THREADS, 0, s>>>(r, map, next);
        else step_kernel<false, false, THREADS><<<blocks, THREADS, 0, s>>>(r, map, next);
    }
    return after_launch();
}

template <bool SF, bool HEAT>
static cudaError_t launch_tile_step(const Arena& a, cudaStream_t s, cudaGraphConditionalHandle next) {
    const size_t smem = (size_t)a.tile_cap * sizeof(uint4);
    static size_t allowed = 0;  // dynamic shared memory the kernel was opened up to
    if (smem > allowed) {
        cudaError_t e = cudaFuncSetAttribute(tile_step_kernel<SF, HEAT>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        cudaFuncSetAttribute(tile_step_kernel<SF, HEAT>,
                             cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        allowed = smem;
    }
    tile_step_kernel<SF, HEAT><<<a.bricks, a.tile_threads, smem, s>>>(a, next);
    return after_launch();
}

cudaError_t launch_step(const Arena& a, const CUtensorMap& map, bool shifted_force,
                        cudaStream_t s, unsigned long long next_decision, bool heat) {
    prefer_l1_once();
    const cudaGraphConditionalHandle next = (cudaGraphConditionalHandle)next_decision;
    if (a.list16 && a.tile_threads) {
        if (shifted_force)
            return heat ? launch_tile_step<true, true>(a, s, next)
                        : launch_tile_step<true, false>(a, s, next);
        return heat ? launch_tile_step<false, true>(a, s, next)
                    : launch_tile_step<false, false>(a, s, next);
    }
#if VLJ_LIST_STREAM
    switch (a.step_threads) {
        case 64: return launch_step_kernel<64>(a, map, shifted_force, s, next, heat);
        case 256: return launch_step_kernel<256>(a, map, shifted_force, s, next, heat);
        default: return launch_step_kernel<kForceThreads>(a, map, shifted_force, s, next, heat);
    }
#else
    return launch_step_kernel<kForceThreads>(a, map, shifted_force, s, next, heat);
#endif
}

template <bool SF, int LANES>
static void measure_lanes(const Arena& a, const CUtensorMap& map, cudaStream_t s) {
    static bool carved = false;
    if (!carved) {
        carved = true;
        prefer_l1(measure_kernel<SF, LANES>);
    }
    measure_kernel<SF, LANES><<<blocks_for(a.nslots, kForceThreads / LANES), kForceThreads, 0, s>>>(a, map);
}

template <bool SF>
static void measure(const Arena& a, const CUtensorMap& map, cudaStream_t s) {
#if VLJ_LIST_STREAM
    switch (lanes_of(a, a.nslots)) {
        case 8: return measure_lanes<SF, 8>(a, map, s);
        case 4: return measure_lanes<SF, 4>(a, map, s);
        case 2: return measure_lanes<SF, 2>(a, map, s);
        default: break;
    }
#endif
    measure_lanes<SF, 1>(a, map, s);
}

cudaError_t launch_measure(const Arena& a, const CUtensorMap& map, bool shifted_force, cudaStream_t s) {
    if (shifted_force) measure<true>(a, map, s);
    else measure<false>(a, map, s);
    return after_launch();
}

template <bool SF, int LANES>
static void read_lanes(const Arena& a, const CUtensorMap& map, uint32_t first, uint32_t count, double* out,
                       cudaStream_t s) {
    static bool carved = false;
    if (!carved) {
        carved = true;
        prefer_l1(read_kernel<SF, LANES>);
    }
    const uint32_t before = LANES == 1 ? first % kForceThreads : 0u;
    read_kernel<SF, LANES><<<blocks_for((uint64_t)before + count, kForceThreads / LANES), kForceThreads, 0, s>>>(
        a, map, first, count, out);
}

template <bool SF>
static void read(const Arena& a, const CUtensorMap& map, uint32_t first, uint32_t count, double* out,
                 cudaStream_t s) {
#if VLJ_LIST_STREAM
    switch (lanes_of(a, count)) {
        case 8: return read_lanes<SF, 8>(a, map, first, count, out, s);
        case 4: return read_lanes<SF, 4>(a, map, first, count, out, s);
        case 2: return read_lanes<SF, 2>(a, map, first, count, out, s);
        default: break;
    }
#endif
    read_lanes<SF, 1>(a, map, first, count, out, s);
}

cudaError_t launch_read(const Arena& a, const CUtensorMap& map, bool shifted_force, uint32_t first,
                        uint32_t count, double* out, cudaStream_t s) {
    if (shifted_force) read<true>(a, map, first, count, out, s);
    else read<false>(a, map, first, count, out, s);
    return after_launch();
}

cudaError_t launch_begin(const Arena& a, cudaStream_t s) {
    const cudaError_t e = launch_chained(begin_kernel, dim3(blocks_for(a.nslots)), kBlock, s, a);
    return e != cudaSuccess ? e : after_launch();
}

template <bool SF, int PASS, int LANES>
static void canon_force_lanes(const Arena& a, const CUtensorMap& map, cudaStream_t s) {
    static bool carved = false;
    if (!carved) {
        carved = true;
        prefer_l1(canon_force_kernel<SF, PASS, LANES>);
    }
    canon_force_kernel<SF, PASS, LANES>
        <<<blocks_for(a.nslots, kForceThreads / LANES), kForceThreads, 0, s>>>(a, map);
}

template <bool SF, int PASS>
static void canon_force_pass(const Arena& a, const CUtensorMap& map, cudaStream_t s) {
#if VLJ_LIST_STREAM
    switch (lanes_of(a, a.nslots)) {
        case 8: return canon_force_lanes<SF, PASS, 8>(a, map, s);
        case 4: return canon_force_lanes<SF, PASS, 4>(a, map, s);
        case 2: return canon_force_lanes<SF, PASS, 2>(a, map, s);
        default: break;
    }
#endif
    canon_force_lanes<SF, PASS, 1>(a, map, s);
}

template <bool SF>
static void canon_force(const Arena& a, const CUtensorMap& map, CanonPass pass, cudaStream_t s) {
    switch (pass) {
        case kPrime: return canon_force_pass<SF, kPrime>(a, map, s);
        case kNoseHoover: return canon_force_pass<SF, kNoseHoover>(a, map, s);
        case kExchange: return canon_force_pass<SF, kExchange>(a, map, s);
        case kKick: return canon_force_pass<SF, kKick>(a, map, s);
    }
}

cudaError_t launch_canon_force(const Arena& a, const CUtensorMap& map, bool shifted_force,
                               CanonPass pass, cudaStream_t s) {
    prefer_l1_once();
    if (shifted_force)
        canon_force<true>(a, map, pass, s);
    else
        canon_force<false>(a, map, pass, s);
    return after_launch();
}

cudaError_t launch_hex_apply(const Arena& a, cudaStream_t s) {
    const cudaError_t e = launch_chained(hex_apply_kernel, dim3(blocks_for(a.nslots)), kBlock, s, a);
    return e != cudaSuccess ? e : after_launch();
}

cudaError_t launch_half_kick_back(const Arena& a, cudaStream_t s) {
    half_kick_back_kernel<<<blocks_for(a.nslots), kBlock, 0, s>>>(a);
    return after_launch();
}

cudaError_t launch_fp32_peak(float* out, int blocks, int iters, cudaStream_t s) {
    fp32_peak_kernel<<<blocks, kBlock, 0, s>>>(out, iters);
    return after_launch();
}

}  // namespace vlj
