// kpax_env.cu — obstacle grid build and the kernel-level batch entry points.
//
// The reference keeps a fixed 16-slot list per 5 m cell and rebuilds it with atomics every
// iteration (spatialHash.cu:9-67, KPAX.cu:306), silently dropping entries past 16 in nondeterministic order.  Here
// the grid is compressed sparse rows (count -> scan -> fill), holds every (cell, obstacle)
// pair and is built once per plan.  Query verdicts equal the brute-force isMotionValid
// (collisionCheck.cu:49-62) for every box: the cell map is monotone, so any strictly
// overlapping obstacle shares at least one cell with the box.
#include <stdio.h>
#include <algorithm>
#include <string.h>

#include <mutex>
#include <new>

#include "kpax_internal.h"

namespace kpax {

std::atomic<uint64_t> g_launches{0};

namespace {

__device__ __forceinline__ void obstacle_cells(const Grid& g, const float4& lo, const float4& hi, int c0[3], int c1[3])
{
    c0[0] = grid_coord(g, lo.x), c0[1] = grid_coord(g, lo.y), c0[2] = grid_coord(g, lo.z);
    c1[0] = grid_coord(g, hi.x), c1[1] = grid_coord(g, hi.y), c1[2] = grid_coord(g, hi.z);
}

// Cell (x, y, z) of the k-th cell of an obstacle's cell box [c0, c1].
__device__ __forceinline__ int box_cell(const Grid& g, const int c0[3], const int c1[3], int k)
{
    const int nx = c1[0] - c0[0] + 1, ny = c1[1] - c0[1] + 1;
    const int x = c0[0] + k % nx, y = c0[1] + (k / nx) % ny, z = c0[2] + k / (nx * ny);
    return x + g.dim * (y + g.dim * z);
}

// Cells of an obstacle's cell box: none when it is inverted in a dimension (the product of two negative
// extents is positive, and box_cell would name cells outside the grid).
__device__ __forceinline__ int box_cells(const int c0[3], const int c1[3])
{
    const int nx = c1[0] - c0[0] + 1, ny = c1[1] - c0[1] + 1, nz = c1[2] - c0[2] + 1;
    return nx > 0 && ny > 0 && nz > 0 ? nx * ny * nz : 0;
}

// One warp per obstacle: pack n x 6 floats into float4 pairs and count (cell, obstacle) pairs.
__global__ void k_env_count(Grid g, const float* __restrict__ obs, uint32_t n, float4* __restrict__ packed,
                            uint32_t* __restrict__ counts)
{
    const uint32_t o = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if(o >= n) return;
    const float* b = obs + (size_t)6 * o;
    const float4 lo = make_float4(b[0], b[1], b[2], 0.0f), hi = make_float4(b[3], b[4], b[5], 0.0f);
    if(lane == 0) packed[2 * o] = lo, packed[2 * o + 1] = hi;
    int c0[3], c1[3];
    obstacle_cells(g, lo, hi, c0, c1);
    const int total = box_cells(c0, c1);
    for(int k = lane; k < total; k += 32) atomicAdd(counts + box_cell(g, c0, c1, k), 1u);
}

// Exclusive scan of counts[0, n) in place (single CTA of 1024 threads; each thread scans 8
// consecutive counts per pass, read and written as two 16-byte vectors where the pass is full and
// both arrays start 16-byte aligned, one count at a time otherwise); counts[n] = total; cursor
// gets a copy of the offsets.
constexpr int kEnvScanItems = 8;
__global__ void __launch_bounds__(1024) k_env_scan(uint32_t* __restrict__ counts, uint32_t n, uint32_t* __restrict__ cursor)
{
    __shared__ uint32_t s_warp[32];
    __shared__ uint32_t s_carry;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool vec = ((reinterpret_cast<uintptr_t>(counts) | reinterpret_cast<uintptr_t>(cursor)) & 15u) == 0;
    if(threadIdx.x == 0) s_carry = 0;
    __syncthreads();
    for(uint32_t base = 0; base < n; base += 1024 * kEnvScanItems) {
        const uint32_t i0 = base + threadIdx.x * kEnvScanItems;
        const bool full = vec && i0 + kEnvScanItems <= n;
        uint32_t v[kEnvScanItems], sum = 0;
        if(full) {
            const uint4 a = *reinterpret_cast<const uint4*>(counts + i0), b = *reinterpret_cast<const uint4*>(counts + i0 + 4);
            v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
        } else {
#pragma unroll
            for(int j = 0; j < kEnvScanItems; ++j) v[j] = i0 + j < n ? counts[i0 + j] : 0u;
        }
#pragma unroll
        for(int j = 0; j < kEnvScanItems; ++j) sum += v[j];
        uint32_t x = sum;
#pragma unroll
        for(int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
            if(lane >= d) x += y;
        }
        if(lane == 31) s_warp[warp] = x;
        __syncthreads();
        if(warp == 0) {
            uint32_t w = s_warp[lane];
#pragma unroll
            for(int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, w, d);
                if(lane >= d) w += y;
            }
            s_warp[lane] = w;
        }
        __syncthreads();
        uint32_t e[kEnvScanItems], acc = s_carry + (warp ? s_warp[warp - 1] : 0u) + x - sum;
#pragma unroll
        for(int j = 0; j < kEnvScanItems; ++j) e[j] = acc, acc += v[j];
        if(full) {
            const uint4 a = make_uint4(e[0], e[1], e[2], e[3]), b = make_uint4(e[4], e[5], e[6], e[7]);
            *reinterpret_cast<uint4*>(counts + i0) = a, *reinterpret_cast<uint4*>(counts + i0 + 4) = b;
            *reinterpret_cast<uint4*>(cursor + i0) = a, *reinterpret_cast<uint4*>(cursor + i0 + 4) = b;
        } else {
#pragma unroll
            for(int j = 0; j < kEnvScanItems; ++j)
                if(i0 + j < n) counts[i0 + j] = e[j], cursor[i0 + j] = e[j];
        }
        __syncthreads();
        if(threadIdx.x == 0) s_carry += s_warp[31];
        __syncthreads();
    }
    if(threadIdx.x == 0) counts[n] = s_carry;
}

__global__ void k_env_fill(Grid g, const float4* __restrict__ packed, uint32_t n, uint32_t* __restrict__ cursor,
                           uint32_t* __restrict__ ent)
{
    const uint32_t o = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if(o >= n) return;
    int c0[3], c1[3];
    obstacle_cells(g, packed[2 * o], packed[2 * o + 1], c0, c1);
    const int total = box_cells(c0, c1);
    for(int k = lane; k < total; k += 32) ent[atomicAdd(cursor + box_cell(g, c0, c1, k), 1u)] = o;
}

// The three passes in one CTA with the counts in shared memory, for grids and obstacle counts that one
// SM gets through sooner than the launches of three kernels and a memset take.  Rows of x-neighbouring cells
// are dealt out to the threads, so that a box over the whole grid keeps them as busy as many small ones.
// Entries are filled in when they fit `cap`; otherwise `cursor` holds the offsets for k_env_fill.  More
// than env_build_pairs(n) (cell, obstacle) pairs are left to the other kernels: `off` then holds zeros and
// the number of pairs, which is known before any is counted.
// The three kernels give each obstacle a warp on one of many SMs, so their time is the largest box's; this
// one's is the pairs'.  B200, the allocation-free batch with 1021 segments on a 9261-cell grid, host us,
// three kernels / one: 20 boxes of 5 m (160 pairs) 41 / 33, 45 m (15477) 62 / 45, 90 m (69232) 119 / 71; one
// over the whole grid 155 / 37; 60 boxes of 30 m (17550) 50 / 45, 45 m (46597) 65 / 59, 60 m (89860) 78 / 85;
// 256 of 10 m (6420) 44 / 36, 20 m (27667) 53 / 56, 45 m (184267) 61 / 154.  More than 256 of 1 to 5 m: 300
// 56 / 52, 1000 58 / 88 with eight threads an obstacle.
constexpr int kEnvBuildBS = 1024;
constexpr uint32_t kEnvBuildCells = 12000;  // 48 KB of shared memory with the rest (22^3 cells: 46 KB)
constexpr uint32_t kEnvBuildObstacles = 256;
__host__ __device__ constexpr uint32_t env_build_pairs(uint32_t n) { return n <= 40u ? 0xFFFFFFFFu : n <= 80u ? 1u << 15 : 1u << 14; }
inline bool env_build_once(uint32_t cells, uint32_t n) { return cells <= kEnvBuildCells && n <= kEnvBuildObstacles; }

__global__ void __launch_bounds__(kEnvBuildBS) k_env_build(Grid g, const float* __restrict__ obs, uint32_t n, uint32_t cells,
                                                           float4* __restrict__ packed, uint32_t* __restrict__ off,
                                                           uint32_t* __restrict__ cursor, uint32_t* __restrict__ ent, uint32_t cap)
{
    extern __shared__ uint32_t s_cell[];  // counts, then offsets, then the next free entry
    __shared__ uint32_t s_warp[32];
    // of each obstacle: the rows before its own, its first cell, its extents in x and y
    __shared__ uint32_t s_row[kEnvBuildObstacles], s_cell0[kEnvBuildObstacles], s_ext[kEnvBuildObstacles];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    // exclusive prefix of the block's values, and their sum
    auto block_scan = [&](uint32_t v, uint32_t& total) {
        auto warp_scan = [&](uint32_t a) {
#pragma unroll
            for(int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, a, d);
                if(lane >= (uint32_t)d) a += y;
            }
            return a;
        };
        const uint32_t x = warp_scan(v);
        if(lane == 31u) s_warp[warp] = x;
        __syncthreads();
        if(warp == 0) s_warp[lane] = warp_scan(s_warp[lane]);
        __syncthreads();
        const uint32_t below = (warp ? s_warp[warp - 1] : 0u) + x - v;
        total = s_warp[31];
        __syncthreads();
        return below;
    };
    for(uint32_t i = tid; i < cells; i += kEnvBuildBS) s_cell[i] = 0u;
    uint32_t own_rows = 0, own_pairs = 0;
    if(tid < n) {
        const float* b = obs + (size_t)6 * tid;
        const float4 lo = make_float4(b[0], b[1], b[2], 0.0f), hi = make_float4(b[3], b[4], b[5], 0.0f);
        packed[2 * tid] = lo, packed[2 * tid + 1] = hi;
        int c0[3], c1[3];
        obstacle_cells(g, lo, hi, c0, c1);
        own_pairs = (uint32_t)box_cells(c0, c1);
        if(own_pairs) own_rows = (uint32_t)((c1[1] - c0[1] + 1) * (c1[2] - c0[2] + 1));
        s_cell0[tid] = (uint32_t)(c0[0] + g.dim * (c0[1] + g.dim * c0[2]));
        s_ext[tid] = (uint32_t)(c1[0] - c0[0] + 1) | ((uint32_t)(c1[1] - c0[1] + 1) << 16);
    }
    uint32_t rows, pairs;
    const uint32_t row0 = block_scan(own_rows, rows);
    if(tid < n) s_row[tid] = row0;
    block_scan(own_pairs, pairs);  // its barriers cover s_row and s_cell as well
    if(pairs > env_build_pairs(n)) {
        for(uint32_t i = tid; i <= cells; i += kEnvBuildBS) off[i] = i < cells ? 0u : pairs;
        return;
    }
    auto each_cell = [&](auto f) {
        for(uint32_t r = tid; r < rows; r += kEnvBuildBS) {
            uint32_t o = 0;  // the last obstacle whose rows start at or before r
#pragma unroll
            for(uint32_t d = kEnvBuildObstacles / 2; d > 0; d >>= 1)
                if(o + d < n && s_row[o + d] <= r) o += d;
            const uint32_t q = r - s_row[o], nx = s_ext[o] & 0xFFFFu, ny = s_ext[o] >> 16, z = q / ny, y = q - z * ny;
            const uint32_t c = s_cell0[o] + g.dim * (y + g.dim * z);
            for(uint32_t x = 0; x < nx; ++x) f(o, c + x);
        }
    };
    each_cell([&](uint32_t, uint32_t c) { atomicAdd(s_cell + c, 1u); });
    __syncthreads();
    const uint32_t per = (cells + kEnvBuildBS - 1) / kEnvBuildBS | 1u;  // odd: no bank conflicts
    const uint32_t i0 = min(tid * per, cells), i1 = min(i0 + per, cells);
    uint32_t sum = 0, total;
    for(uint32_t i = i0; i < i1; ++i) sum += s_cell[i];
    uint32_t acc = block_scan(sum, total);
    for(uint32_t i = i0; i < i1; ++i) {
        const uint32_t v = s_cell[i];
        s_cell[i] = acc, acc += v;
    }
    __syncthreads();
    for(uint32_t i = tid; i < cells; i += kEnvBuildBS) {
        off[i] = s_cell[i];
        if(total > cap) cursor[i] = s_cell[i];
    }
    if(tid == 0) off[cells] = total;
    if(total > cap) return;
    __syncthreads();
    each_cell([&](uint32_t o, uint32_t c) { ent[atomicAdd(s_cell + c, 1u)] = o; });
}

inline uint32_t warp_blocks(uint32_t n) { return (uint32_t)(((uint64_t)n * 32 + 255) / 256); }

// ---------------------------------------------------------------- batch kernels

// CTAs of the batch kernels: 256 threads, four per SM (64 registers), for the 6-state models; the
// quadrotor's step keeps over 100 values, and at 64 registers its spills cost more than the warps
// gain (30011 segments in the building scene 70 us spilling, 53 us at 128 registers; 2^20 555 -> 448 us).
// With a query per step (K == 1) the waits for lookups prevail: 2^19 of 0.4 s steps 413 us at 64 registers,
// 506 at 128.
// The kept states of a group (kSaveFloats) stay below the 48 KB of static shared memory.
template <int M, int K>
constexpr int kBatchBS = M == KPAX_MODEL_QUADROTOR && K > 1 ? 128 : 256;
constexpr int kBatchBlocks = 4;
template <int M, int BS, int K>
constexpr int kSaveFloats = K > 1 ? K * ModelDims<M>::SD * BS : 4;

template <int M, int K>
__global__ void __launch_bounds__((kBatchBS<M, K>), kBatchBlocks) k_propagate_batch(KParams p, Grid g, const float* __restrict__ parents,
                                                         const float* __restrict__ draws, uint32_t stream_id, uint32_t n,
                                                         float* __restrict__ rows, uint8_t* __restrict__ valid,
                                                         int32_t* __restrict__ steps_out)
{
    constexpr int SD = ModelDims<M>::SD, CD = ModelDims<M>::CD, S = SD + CD + 1;
    constexpr int BS = kBatchBS<M, K>;
    __shared__ __align__(16) float s_save[kSaveFloats<M, BS, K>];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    float s[SD], u[6], c[4], rc[4];
#pragma unroll
    for(int k = 0; k < SD; ++k) s[k] = __ldg(parents + (size_t)i * SD + k);
    if(draws) {
#pragma unroll
        for(int k = 0; k < 5; ++k) u[k] = __ldg(draws + (size_t)i * 5 + k);
        u[5] = 0.0f;
    } else {
        child_draws(p, stream_id, 0u, i, u);
    }
    const int steps = draw_controls(p, u, c);
    int done = 0;
    const bool ok = propagate<M, K>(p, g, s, c, steps, done, s_save + threadIdx.x * SD, BS);
    row_controls<M>(c, rc);
    float* dst = rows + (size_t)i * S;
#pragma unroll
    for(int k = 0; k < SD; ++k) dst[k] = s[k];
#pragma unroll
    for(int k = 0; k < CD; ++k) dst[SD + k] = rc[k];
    dst[SD + CD] = __fmul_rn(p.h, (float)steps);  // STEP_SIZE * propagationDuration
    valid[i] = ok ? 1 : 0;
    if(steps_out) steps_out[i] = done;
}

// Large batches run in phases so that lanes do not idle behind their warp's longest segment: the
// head runs every segment for its first kHeadSteps steps and finishes the segments that end there; the
// others are appended, state and controls, to a compact list, which the tail carries to the end with
// full warps.  Both run the same per-step code in the same order, so rows, verdicts and step counts
// equal the one-pass kernel's.
// What bounds the kernels is instruction issue (Dubins, 2^20 segments: 70-77 % of the issue slots, 24 of
// 32 lanes), so a phase must save more steps and walks than its appends and reloads cost.  A head of one
// query group asks for no more queries than one pass would; only the quadrotor, whose step costs most,
// gains by dropping its dead sooner.  B200, us, one pass / head of 2 / of 5 / of 2 and a middle phase:
// Dubins 2^22, 200 obstacles 615 / 625 / 579 / 639, 1500 obstacles 859 / 637 / 633 / 656;
// quadrotor 2^21, 200 obstacles 1302 / 1191 / 1173 / 1201, 2000 obstacles 1418 / 582 / 661 / 579.
template <int M, int K>
constexpr int kHeadSteps = M == KPAX_MODEL_QUADROTOR || K == 1 ? 2 : K;
// The phases need a few waves of CTAs to fill the chip twice (one pass / two phases, us: Dubins 2^18, 200
// obstacles 58 / 66, 2^19 93 / 96, with 1500 obstacles 130 / 113; quadrotor 2^18, 200 obstacles 181 / 182,
// with 2000 208 / 125), and segments of more than two query groups: those of ten steps leave the tail
// too little (double integrator 2^22, 20 obstacles 235 / 266, 200 obstacles 263 / 291).  With a query per
// step the quadrotor's steps are worth it from ten on (quad-ref, 200 obstacles, one pass / phases: 2^18
// 91 / 94, 2^19 169 / 140, 2^21 638 / 466).
template <int M, int K>
constexpr uint32_t kPhasedMin = K > 1 ? 2048u * kBatchBS<M, K> : 1u << 18;
template <int M, int K>
inline bool phased(const KParams& p, uint32_t n)
{
    return n >= kPhasedMin<M, K> && (p.nsteps > 2 * kGroup || (K == 1 && M == KPAX_MODEL_QUADROTOR));
}
// With a query per step a middle phase up to 3/5 of the longest segment keeps the tail's lanes full at no
// further query (quadrotor steps of 0.4 s, 2^21, no obstacles 1482 us without it, 1248 with it).
template <int K>
constexpr bool kMiddle = K == 1;
// Segments per round of the phases (bounds the survivor lists' scratch).  Each round pays the
// latency of its longest segment in every phase, so rounds are as large as the scratch allows.
constexpr uint32_t kPhaseChunk = 1u << 24;

struct LiveList {
    uint32_t* count;
    uint32_t* idx;
    int32_t* steps;  // unused (null) for fixed-step models
    float* ctl;      // CD per entry
    float* state;    // SD per entry
};
constexpr size_t kCountBytes = 256;  // the counts of both lists, 128 bytes apart

template <int M>
__device__ __forceinline__ void write_segment(const KParams& p, uint32_t i, const float* s, const float* c, int steps, bool ok,
                                              int done, float* __restrict__ rows, uint8_t* __restrict__ valid,
                                              int32_t* __restrict__ steps_out)
{
    constexpr int SD = ModelDims<M>::SD, CD = ModelDims<M>::CD, S = SD + CD + 1;
    float rc[4];
    row_controls<M>(c, rc);
    float* dst = rows + (size_t)i * S;
#pragma unroll
    for(int k = 0; k < SD; ++k) dst[k] = s[k];
#pragma unroll
    for(int k = 0; k < CD; ++k) dst[SD + k] = rc[k];
    dst[SD + CD] = __fmul_rn(p.h, (float)steps);
    valid[i] = ok ? 1 : 0;
    if(steps_out) steps_out[i] = done;
}

// Appends the warp's live segments to `live` (one atomic per warp); called by all 32 lanes.
template <int SD, int CD>
__device__ __forceinline__ void append_live(const LiveList& live, bool alive, int lane, uint32_t i, int steps, const float* c,
                                            const float* s)
{
    const uint32_t m = __ballot_sync(0xffffffffu, alive);
    if(!m) return;
    const int leader = __ffs(m) - 1;
    uint32_t base = 0;
    if(lane == leader) base = atomicAdd(live.count, (uint32_t)__popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if(alive) {
        const uint32_t j = base + __popc(m & ((1u << lane) - 1u));
        live.idx[j] = i;
        if(live.steps) live.steps[j] = steps;
#pragma unroll
        for(int k = 0; k < CD; ++k) live.ctl[(size_t)j * CD + k] = c[k];
#pragma unroll
        for(int k = 0; k < SD; ++k) live.state[(size_t)j * SD + k] = s[k];
    }
}

// Segments i of one round (pointers offset to the round's first segment; i0 = that segment's index
// in the batch, which keys its draws).
template <int M, int K>
__global__ void __launch_bounds__((kBatchBS<M, K>), kBatchBlocks) k_propagate_head(KParams p, Grid g, const float* __restrict__ parents,
                                                        const float* __restrict__ draws, uint32_t stream_id, uint32_t n,
                                                        uint32_t i0, float* __restrict__ rows, uint8_t* __restrict__ valid,
                                                        int32_t* __restrict__ steps_out, LiveList live)
{
    constexpr int SD = ModelDims<M>::SD, CD = ModelDims<M>::CD;
    constexpr int BS = kBatchBS<M, K>, kHead = kHeadSteps<M, K>, kQuery = K > 1 ? kHead : 1;
    __shared__ __align__(16) float s_save[kSaveFloats<M, BS, kQuery>];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    bool alive = false;
    float s[SD], c[4];
    int steps = 0;
    if(i < n) {
        float u[6];
#pragma unroll
        for(int k = 0; k < SD; ++k) s[k] = __ldg(parents + (size_t)i * SD + k);
        if(draws) {
#pragma unroll
            for(int k = 0; k < 5; ++k) u[k] = __ldg(draws + (size_t)i * 5 + k);
            u[5] = 0.0f;
        } else {
            child_draws(p, stream_id, 0u, i0 + i, u);
        }
        steps = draw_controls(p, u, c);
        const auto k = segment_consts<M>(p, c);
        const StepParams sp = step_params(p);
        int done = 0;
        const bool ok = run_steps<M, kQuery>(sp, g, s, c, k, min(steps, kHead), done, s_save + threadIdx.x * SD, BS);
        alive = ok && done < steps;
        if(!alive) write_segment<M>(p, i, s, c, steps, ok, done, rows, valid, steps_out);
    }
    append_live<SD, CD>(live, alive, lane, i, steps, c, s);
}

// Segments of `live` from step `from` on: to their end (kLast), or to step `until` with those that go on
// appended to `next`.
template <int M, int K, bool kLast>
__global__ void __launch_bounds__((kBatchBS<M, K>), kBatchBlocks) k_propagate_tail(KParams p, Grid g, float* __restrict__ rows,
                                                        uint8_t* __restrict__ valid, int32_t* __restrict__ steps_out,
                                                        LiveList live, int from, int until, LiveList next)
{
    constexpr int SD = ModelDims<M>::SD, CD = ModelDims<M>::CD;
    constexpr int BS = kBatchBS<M, K>;
    __shared__ __align__(16) float s_save[kSaveFloats<M, BS, K>];
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x, count = *live.count;
    if(kLast ? j >= count : blockIdx.x * blockDim.x >= count) return;  // appends need whole warps
    const bool in = kLast || j < count;
    const uint32_t e = in ? j : 0u;
    const uint32_t i = live.idx[e];
    const int steps = live.steps ? live.steps[e] : p.nsteps;
    float s[SD], c[4];
#pragma unroll
    for(int k = 0; k < 4; ++k) c[k] = k < CD ? live.ctl[(size_t)e * CD + k] : 0.0f;
#pragma unroll
    for(int k = 0; k < SD; ++k) s[k] = live.state[(size_t)e * SD + k];
    const auto kc = segment_consts<M>(p, c);
    const StepParams sp = step_params(p);
    int done = from;
    const int end = kLast ? steps : in ? min(steps, until) : 0;
    const bool ok = run_steps<M, K>(sp, g, s, c, kc, end, done, s_save + threadIdx.x * SD, BS);
    const bool alive = !kLast && in && ok && done < steps;
    if(in && !alive) write_segment<M>(p, i, s, c, steps, ok, done, rows, valid, steps_out);
    if constexpr(!kLast) append_live<SD, CD>(next, alive, threadIdx.x & 31, i, steps, c, s);
}

// The phases over rounds of kPhaseChunk segments; the lists' counts are cleared before every round.
template <int M, int K>
void launch_phases(const KParams& p, const Grid& g, const float* parents, const float* draws, uint32_t stream_id, uint32_t n,
                   float* rows, uint8_t* valid, int32_t* steps_out, const LiveList& live, const LiveList& second, cudaStream_t s)
{
    const int SD = p.sd, S = p.S;
    for(uint32_t o = 0; o < n; o += kPhaseChunk) {
        const uint32_t m = std::min(kPhaseChunk, n - o), bs = kBatchBS<M, K>, blocks = (m + bs - 1) / bs;
        float* r = rows + (size_t)o * S;
        uint8_t* v = valid + o;
        int32_t* st = steps_out ? steps_out + o : nullptr;
        int from = kHeadSteps<M, K>;
        cudaMemsetAsync(live.count, 0, kCountBytes, s);
        k_propagate_head<M, K><<<blocks, bs, 0, s>>>(p, g, parents + (size_t)o * SD, draws ? draws + (size_t)o * 5 : nullptr,
                                                   stream_id, m, o, r, v, st, live);
        if constexpr(kMiddle<K>) {
            const int until = std::max(from + 1, p.nsteps * 3 / 5);
            k_propagate_tail<M, K, false><<<blocks, bs, 0, s>>>(p, g, r, v, st, live, from, until, second);
            from = until;
        }
        k_propagate_tail<M, K, true><<<blocks, bs, 0, s>>>(p, g, r, v, st, kMiddle<K> ? second : live, from, 0, LiveList{});
        count_launch(kMiddle<K> ? 3 : 2);
    }
}

__global__ void k_collide_batch(Grid g, const float* __restrict__ bbmin, const float* __restrict__ bbmax, uint32_t n,
                                uint8_t* __restrict__ free_out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    const float lo[3] = {bbmin[3 * i], bbmin[3 * i + 1], bbmin[3 * i + 2]};
    const float hi[3] = {bbmax[3 * i], bbmax[3 * i + 1], bbmax[3 * i + 2]};
    free_out[i] = box_free(g, lo, hi) ? 1 : 0;
}

// Large batches of queries with the whole grid in shared memory: a cell's record is its first entry and
// the one past its last (16 bits each), entries are 16-bit obstacle indices, obstacles (lo, hi) pairs per
// dimension.  The queries' cells are scattered, and a gather of 32 scattered words takes 32 wavefronts
// from L1 but about four from shared memory; what bounds it is the issue of divergent lookups (a walk cell by
// cell: 13 of 32 lanes active, 78 % issue).  Cells of a row lie behind one another in the entries, so a lane
// walks rows.  Copying the grid costs every CTA 3-5 us, so it pays from 2^21 boxes on.
// B200, 2^22 boxes, us (global / shared by cells / by rows): boxes of up to 0.2 m, 300 obstacles 52 / 45 / 41,
// 1000 80 / 62 / 58, 2000 103 / 82 / 78; of up to 3 m 84 / 86 / 70, 115 / 100 / 87, 121 / 109 / 102; of up to
// 20 m 263 / 238 / 147, 150 / 129 / 99, 105 / 94 / 84.
constexpr int kCollideBS = 1024;
constexpr uint32_t kCollideSharedMin = 1u << 21, kCollideSharedEnt = 4096;  // with few entries most cells are empty: 2^21 boxes among 20 obstacles 29 / 30 us
constexpr size_t kCollideMaxSmem = 224 * 1024;
inline size_t collide_smem(uint32_t cells, uint32_t n_ent, uint32_t n_obs)
{
    return (4 * (size_t)cells + 2 * (size_t)n_ent + 7) / 8 * 8 + 24 * (size_t)n_obs;
}

__global__ void __launch_bounds__(kCollideBS, 2) k_collide_shared(Grid g, uint32_t cells, uint32_t n_ent, uint32_t n_obs,
                                                               const float* __restrict__ bbmin, const float* __restrict__ bbmax,
                                                               uint32_t n, uint8_t* __restrict__ free_out)
{
    extern __shared__ __align__(16) uint8_t s_grid[];
    uint32_t* s_cell = reinterpret_cast<uint32_t*>(s_grid);
    uint16_t* s_ent = reinterpret_cast<uint16_t*>(s_cell + cells);
    float2* s_obs = reinterpret_cast<float2*>(s_grid + (4 * (size_t)cells + 2 * (size_t)n_ent + 7) / 8 * 8);
    for(uint32_t i = threadIdx.x; i < cells; i += kCollideBS) s_cell[i] = __ldg(g.off + i) | (__ldg(g.off + i + 1) << 16);
    for(uint32_t i = threadIdx.x; i < n_ent; i += kCollideBS) s_ent[i] = (uint16_t)__ldg(g.ent + i);
    for(uint32_t i = threadIdx.x; i < n_obs; i += kCollideBS) {
        const float4 a = __ldg(g.obs + 2 * i), m = __ldg(g.obs + 2 * i + 1);
        s_obs[i] = make_float2(a.x, m.x), s_obs[n_obs + i] = make_float2(a.y, m.y), s_obs[2 * n_obs + i] = make_float2(a.z, m.z);
    }
    __syncthreads();
    auto query = [&](const float* lo, const float* hi) -> bool {
        const int x0 = grid_coord(g, lo[0]), y0 = grid_coord(g, lo[1]), z0 = grid_coord(g, lo[2]);
        const int x1 = grid_coord(g, hi[0]), y1 = grid_coord(g, hi[1]), z1 = grid_coord(g, hi[2]);
        const int row = x1 - x0, plane = y1 - y0;
        int gy = plane, gz = z1 - z0;
        if((row | plane | gz) < 0) return true;  // an inverted box has no cells
        // the walk over the box's rows of cells, whose entries lie behind one another, as one loop: a lane
        // whose row is done steps to its next one
        uint32_t c = x0 + g.dim * (y0 + g.dim * z0), k = s_cell[c] & 0xFFFFu, e = s_cell[c + row] >> 16;
        for(;;) {
            if(k < e) {
                const uint32_t o = s_ent[k++];
                const float2 a = s_obs[o], b = s_obs[n_obs + o], d = s_obs[2 * n_obs + o];
                if(hi[0] > a.x && a.y > lo[0] && hi[1] > b.x && b.y > lo[1] && hi[2] > d.x && d.y > lo[2]) return false;
            } else {
                if(gy-- > 0) c += g.dim;
                else if(gy = plane, gz-- > 0) c += g.dim * g.dim - g.dim * plane;
                else break;
                k = s_cell[c] & 0xFFFFu, e = s_cell[c + row] >> 16;
            }
        }
        return true;
    };
    // a warp takes 32 consecutive boxes at a time, so that its lanes' corners share cache lines; the last stride
    // would pass 2^32 where n is near it
    const uint32_t stride = gridDim.x * kCollideBS;
    for(uint32_t i = blockIdx.x * kCollideBS + threadIdx.x; i < n; i += stride) {
        const float lo[3] = {__ldcs(bbmin + 3 * (size_t)i), __ldcs(bbmin + 3 * (size_t)i + 1), __ldcs(bbmin + 3 * (size_t)i + 2)};
        const float hi[3] = {__ldcs(bbmax + 3 * (size_t)i), __ldcs(bbmax + 3 * (size_t)i + 1), __ldcs(bbmax + 3 * (size_t)i + 2)};
        free_out[i] = query(lo, hi) ? 1 : 0;
        if(n - i <= stride) break;
    }
}

__global__ void k_region_batch(KParams p, const float* __restrict__ states, uint32_t n, int32_t* __restrict__ r1,
                               int32_t* __restrict__ r2)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    float s[12];
    for(int k = 0; k < p.sd; ++k) s[k] = states[(size_t)i * p.sd + k];
    const int a = region_r1<12>(p, s);
    r1[i] = a;
    if(r2) r2[i] = region_r2<12>(p, s, a);
}

__global__ void k_sincos_pair(const float* __restrict__ x, uint32_t n, float* __restrict__ out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    float s, c, s2, c2;
    sincos_checked(x[i], &s, &c);
    sincosf(x[i], &s2, &c2);
    out[4 * i] = s, out[4 * i + 1] = c, out[4 * i + 2] = s2, out[4 * i + 3] = c2;
}

}  // namespace

// The grid's offsets by two kernels, from counts at zero.
static kpax_status env_count(const Grid& g, const float* d_obstacles, uint32_t n, uint32_t cells, float4* packed, uint32_t* off,
                             uint32_t* cursor, cudaStream_t stream)
{
    k_env_count<<<warp_blocks(n), 256, 0, stream>>>(g, d_obstacles, n, packed, off);
    KPAX_CHECK_LAUNCH();
    k_env_scan<<<1, 1024, 0, stream>>>(off, cells, cursor);
    KPAX_CHECK_LAUNCH();
    count_launch(2);
    return KPAX_OK;
}

kpax_status Env::build_start(const KParams& p, const float* d_obstacles, uint32_t n, cudaStream_t stream)
{
    cell = p.cell;
    wmin = p.wmin;
    dim = p.gdim;
    const uint32_t cells = (uint32_t)dim * dim * dim;
    if(cells != n_cells) {
        if(d_off) cudaFree(d_off), d_off = nullptr;
        if(d_cursor) cudaFree(d_cursor), d_cursor = nullptr;
        KPAX_CUDA(cudaMalloc(&d_off, sizeof(uint32_t) * (cells + 1)));
        KPAX_CUDA(cudaMalloc(&d_cursor, sizeof(uint32_t) * cells));
        n_cells = cells;
    }
    if(!h_total) KPAX_CUDA(cudaMallocHost(&h_total, sizeof(uint32_t)));
    if(n > obs_cap) {
        if(d_obs) cudaFree(d_obs), d_obs = nullptr;
        KPAX_CUDA(cudaMalloc(&d_obs, sizeof(float4) * 2 * n));
        obs_cap = n;
    }
    n_obs = n;
    if(!d_ent) {
        KPAX_CUDA(cudaMalloc(&d_ent, sizeof(uint32_t) * 1024));
        ent_cap = 1024;
    }
    if(!d_obs) {
        KPAX_CUDA(cudaMalloc(&d_obs, sizeof(float4) * 2));
        obs_cap = 1;
    }
    filled = false;
    if(n && env_build_once(cells, n)) {
        k_env_build<<<1, kEnvBuildBS, sizeof(uint32_t) * cells, stream>>>(view(), d_obstacles, n, cells, d_obs, d_off, d_cursor, d_ent, ent_cap);
        KPAX_CHECK_LAUNCH();
        count_launch(1);
        filled = true;
    } else {
        KPAX_CUDA(cudaMemsetAsync(d_off, 0, sizeof(uint32_t) * (cells + 1), stream));
        if(n) {
            kpax_status st = env_count(view(), d_obstacles, n, cells, d_obs, d_off, d_cursor, stream);
            if(st != KPAX_OK) return st;
        }
    }
    *h_total = 0;
    if(n) KPAX_CUDA(cudaMemcpyAsync(h_total, d_off + cells, sizeof(uint32_t), cudaMemcpyDeviceToHost, stream));
    return KPAX_OK;
}

kpax_status Env::build_finish(const float* d_obstacles, cudaStream_t stream)
{
    n_ent = *h_total;
    if(filled && n_ent > env_build_pairs(n_obs)) {
        filled = false;
        kpax_status st = env_count(view(), d_obstacles, n_obs, n_cells, d_obs, d_off, d_cursor, stream);
        if(st != KPAX_OK) return st;
    }
    if(n_ent > ent_cap) {
        filled = false;
        if(d_ent) cudaFree(d_ent), d_ent = nullptr, ent_cap = 0;
        const uint32_t want = n_ent + n_ent / 4 + 1024;
        KPAX_CUDA(cudaMalloc(&d_ent, sizeof(uint32_t) * want));
        ent_cap = want;
    }
    if(n_obs && !filled) {
        k_env_fill<<<warp_blocks(n_obs), 256, 0, stream>>>(view(), d_obs, n_obs, d_cursor, d_ent);
        KPAX_CHECK_LAUNCH();
        count_launch(1);
    }
    return KPAX_OK;
}

kpax_status Env::build(const KParams& p, const float* d_obstacles, uint32_t n, cudaStream_t stream)
{
    kpax_status st = build_start(p, d_obstacles, n, stream);
    if(st != KPAX_OK) return st;
    if(n) KPAX_CUDA(cudaStreamSynchronize(stream));
    return build_finish(d_obstacles, stream);
}

void Env::release()
{
    if(d_obs) cudaFree(d_obs);
    if(d_off) cudaFree(d_off);
    if(d_cursor) cudaFree(d_cursor);
    if(d_ent) cudaFree(d_ent);
    if(d_live) cudaFree(d_live), d_live = nullptr, live_cap = 0;
    if(h_total) cudaFreeHost(h_total);
    d_obs = nullptr, d_off = d_cursor = d_ent = h_total = nullptr;
    obs_cap = ent_cap = n_cells = n_ent = n_obs = 0;
}

kpax_status launch_propagate(const KParams& p, const Grid& g, const float* parents, const float* draws, uint32_t stream_id,
                             uint32_t n, float* rows, uint8_t* valid, int32_t* steps, cudaStream_t stream)
{
    if(!n) return KPAX_OK;
    by_model(p.model, grouped(p) ? kGroup : 1, [&](auto m, auto k) {
        constexpr int M = decltype(m)::value, K = decltype(k)::value;
        constexpr uint32_t bs = kBatchBS<M, K>;
        k_propagate_batch<M, K><<<(n + bs - 1) / bs, bs, 0, stream>>>(p, g, parents, draws, stream_id, n, rows, valid, steps);
    });
    KPAX_CHECK_LAUNCH();
    count_launch();
    return KPAX_OK;
}

}  // namespace kpax

using namespace kpax;

extern "C" {

uint64_t kpax_kernel_launches(void) { return g_launches.load(); }

kpax_status kpax_test_sincos(const float* d_x, uint32_t n, float* d_out, void* stream)
{
    if(n && (!d_x || !d_out)) return set_error("kpax_test_sincos: null argument"), KPAX_EINVAL;
    if(!n) return KPAX_OK;
    k_sincos_pair<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(d_x, n, d_out);
    KPAX_CHECK_LAUNCH();
    return KPAX_OK;
}

// FP32 issue-rate microkernel: every thread advances kChains independent FMA chains `iters` times
// (2 FLOP per FMA); the values stay bounded (|a| < 1) and are folded into one store the compiler
// cannot drop.  The measured rate is the denominator of the propagation kernels' roofline.
constexpr int kFmaChains = 8;
__global__ void __launch_bounds__(512) k_fma_peak(float* __restrict__ out, uint32_t iters, float a, float b)
{
    float x[kFmaChains];
#pragma unroll
    for(int j = 0; j < kFmaChains; ++j) x[j] = (float)(threadIdx.x + j) * 1e-3f;
    for(uint32_t i = 0; i < iters; i += 16) {
#pragma unroll
        for(int u = 0; u < 16; ++u)
#pragma unroll
            for(int j = 0; j < kFmaChains; ++j) x[j] = fmaf(x[j], a, b);
    }
    float s = 0.0f;
#pragma unroll
    for(int j = 0; j < kFmaChains; ++j) s += x[j];
    if(s == -1.0f) out[blockIdx.x * blockDim.x + threadIdx.x] = s;  // never true; keeps the chains live
}

kpax_status kpax_fp32_peak(uint32_t iters, double* h_tflops, double* h_ms, void* stream)
{
    if(!h_tflops || iters < 16) return set_error("kpax_fp32_peak: need h_tflops and iters >= 16"), KPAX_EINVAL;
    iters = iters / 16 * 16;
    int dev = 0, sms = 0;
    KPAX_CUDA(cudaGetDevice(&dev));
    KPAX_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const uint32_t blocks = (uint32_t)sms * 4u, threads = 512;  // 2048 threads per SM
    cudaStream_t s = (cudaStream_t)stream;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    KPAX_CUDA(cudaEventCreate(&e0));
    KPAX_CUDA(cudaEventCreate(&e1));
    float ms = 0.0f;
    for(int rep = 0; rep < 2; ++rep) {  // the first launch warms up
        cudaEventRecord(e0, s);
        k_fma_peak<<<blocks, threads, 0, s>>>(nullptr, iters, 0.99999f, 1e-6f);
        cudaEventRecord(e1, s);
        count_launch();
    }
    cudaError_t err = cudaEventSynchronize(e1);
    if(err == cudaSuccess) err = cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if(err != cudaSuccess) return set_error("kpax_fp32_peak: %s", cudaGetErrorString(err)), KPAX_ECUDA;
    const double flop = 2.0 * kFmaChains * (double)iters * blocks * threads;
    *h_tflops = ms > 0.0f ? flop / (ms * 1e-3) / 1e12 : 0.0;
    if(h_ms) *h_ms = ms;
    return KPAX_OK;
}

kpax_status kpax_env_create(const kpax_config* cfg, const float* d_obstacles, uint32_t n_obs, void* stream, kpax_env** out)
{
    NvtxRange range("kpax_env_create");
    if(!cfg || !out || (n_obs && !d_obstacles)) return set_error("kpax_env_create: null argument"), KPAX_EINVAL;
    *out = nullptr;
    kpax_env* e = new(std::nothrow) kpax_env();
    if(!e) return set_error("kpax_env_create: host allocation failed"), KPAX_ENOMEM;
    kpax_status st = derive_params(*cfg, &e->params);
    if(st == KPAX_OK) st = e->env.build(e->params, d_obstacles, n_obs, (cudaStream_t)stream);
    if(st == KPAX_OK) {
        cudaError_t err = cudaStreamSynchronize((cudaStream_t)stream);
        if(err != cudaSuccess) set_error("kpax_env_create: %s", cudaGetErrorString(err)), st = KPAX_ECUDA;
    }
    if(st != KPAX_OK) {
        e->env.release();
        delete e;
        return st;
    }
    *out = e;
    return KPAX_OK;
}

kpax_status kpax_env_destroy(kpax_env* e)
{
    if(!e) return KPAX_OK;
    e->env.release();
    if(e->d_occ) cudaFree(e->d_occ);
    delete e;
    return KPAX_OK;
}

kpax_status kpax_env_stats(kpax_env* e, uint32_t* n_cells, uint32_t* n_entries)
{
    if(!e) return set_error("kpax_env_stats: null env"), KPAX_EINVAL;
    if(n_cells) *n_cells = e->env.n_cells;
    if(n_entries) *n_entries = e->env.n_ent;
    return KPAX_OK;
}

kpax_status kpax_propagate_batch(const kpax_config* cfg, kpax_env* env, const float* d_parents, const float* d_draws,
                                 uint32_t draw_stream, uint32_t n, float* d_rows, uint8_t* d_valid, int32_t* d_steps,
                                 void* stream)
{
    NvtxRange range("kpax_propagate_batch");
    if(!cfg || !env || (n && (!d_parents || !d_rows || !d_valid)))
        return set_error("kpax_propagate_batch: null argument"), KPAX_EINVAL;
    KParams p;
    kpax_status st = derive_params(*cfg, &p);
    if(st != KPAX_OK) return st;
    if(p.gdim != env->env.dim || p.cell != env->env.cell || p.wmin != env->env.wmin)
        return set_error("kpax_propagate_batch: env was built for another workspace grid"), KPAX_EINVAL;
    const int group = grouped(p) ? kGroup : 1;
    const bool two = by_model(p.model, group, [&](auto m, auto k) { return phased<decltype(m)::value, decltype(k)::value>(p, n); });
    if(!two)
        return launch_propagate(p, env->env.view(), d_parents, d_draws, draw_stream, n, d_rows, d_valid, d_steps,
                                (cudaStream_t)stream);
    // phases: the live lists of a round live in the env's scratch, grown on demand (their counts, then each
    // list's index, step-count (drawn durations only), control and state arrays)
    Env& e = env->env;
    auto align = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t m = std::min(n, kPhaseChunk);
    const size_t l_steps = align(4ull * m), l_ctl = l_steps + (p.fixed_steps ? 0 : align(4ull * m)),
                 l_state = l_ctl + align(4ull * p.cd * m), l_bytes = l_state + align(4ull * p.sd * m);
    const size_t bytes = kCountBytes + (group == 1 && kMiddle<1> ? 2 : 1) * l_bytes;
    if(bytes > e.live_cap) {
        if(e.d_live) cudaFree(e.d_live), e.d_live = nullptr, e.live_cap = 0;
        KPAX_CUDA(cudaMalloc(&e.d_live, bytes));
        e.live_cap = bytes;
    }
    auto list = [&](int k) {
        char *count = static_cast<char*>(e.d_live) + 128 * k, *l = static_cast<char*>(e.d_live) + kCountBytes + k * l_bytes;
        return LiveList{reinterpret_cast<uint32_t*>(count), reinterpret_cast<uint32_t*>(l),
                        p.fixed_steps ? nullptr : reinterpret_cast<int32_t*>(l + l_steps), reinterpret_cast<float*>(l + l_ctl),
                        reinterpret_cast<float*>(l + l_state)};
    };
    cudaStream_t s = (cudaStream_t)stream;
    const Grid g = e.view();
    by_model(p.model, group, [&](auto m, auto k) {
        launch_phases<decltype(m)::value, decltype(k)::value>(p, g, d_parents, d_draws, draw_stream, n, d_rows, d_valid, d_steps, list(0), list(1), s);
    });
    KPAX_CHECK_LAUNCH();
    return KPAX_OK;
}

kpax_status kpax_collide_batch(kpax_env* env, const float* d_bbmin, const float* d_bbmax, uint32_t n, uint8_t* d_free,
                               void* stream)
{
    if(!env || (n && (!d_bbmin || !d_bbmax || !d_free))) return set_error("kpax_collide_batch: null argument"), KPAX_EINVAL;
    if(!n) return KPAX_OK;
    const Env& e = env->env;
    const size_t smem = collide_smem(e.n_cells, e.n_ent, e.n_obs);
    if(n >= kCollideSharedMin && e.n_ent >= kCollideSharedEnt && e.n_ent < 65536u && e.n_obs <= 65536u && smem <= kCollideMaxSmem) {
        int dev = 0, sms = 0;
        KPAX_CUDA(cudaGetDevice(&dev));
        KPAX_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        // the limit belongs to the kernel: every call sets the same one, whatever its own grid needs
        KPAX_CUDA(cudaFuncSetAttribute(k_collide_shared, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCollideMaxSmem));
        const uint32_t grid = (uint32_t)sms * (smem <= kCollideMaxSmem / 2 ? 2u : 1u);
        k_collide_shared<<<grid, kCollideBS, smem, (cudaStream_t)stream>>>(e.view(), e.n_cells, e.n_ent, e.n_obs, d_bbmin, d_bbmax, n, d_free);
        KPAX_CHECK_LAUNCH();
        count_launch();
        return KPAX_OK;
    }
    k_collide_batch<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(env->env.view(), d_bbmin, d_bbmax, n, d_free);
    KPAX_CHECK_LAUNCH();
    count_launch();
    return KPAX_OK;
}

kpax_status kpax_region_batch(const kpax_config* cfg, const float* d_states, uint32_t n, int32_t* d_r1, int32_t* d_r2,
                              void* stream)
{
    if(!cfg || (n && (!d_states || !d_r1))) return set_error("kpax_region_batch: null argument"), KPAX_EINVAL;
    KParams p;
    kpax_status st = derive_params(*cfg, &p);
    if(st != KPAX_OK) return st;
    if(!n) return KPAX_OK;
    k_region_batch<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(p, d_states, n, d_r1, d_r2);
    KPAX_CHECK_LAUNCH();
    count_launch();
    return KPAX_OK;
}

}  // extern "C"

// ---------------------------------------------------------------- allocation-free propagation
// kpax_propagate_batch_noalloc builds the obstacle grid in a fixed device array instead of
// memory from cudaMalloc, for callers that must not allocate device memory while they run: a
// planner called from a robot's real-time control cycle (cudaMalloc can synchronise the device
// and take unbounded time) or a host application that reserves all device memory up front for
// its own pool.  The array below lives in every GPU that loads this library, until exit.
namespace {

constexpr uint32_t kNoAllocMaxObstacles = 4096;
constexpr uint32_t kNoAllocMaxCells = 1u << 17;    // e.g. a 50^3 grid
constexpr uint32_t kNoAllocMaxEntries = 1u << 18;  // (cell, obstacle) pairs

struct NoAllocScratch {
    float4 obs[2 * kNoAllocMaxObstacles];
    uint32_t off[kNoAllocMaxCells + 4];  // cells + 1, padded so that cursor starts 16-byte aligned
    uint32_t cursor[kNoAllocMaxCells];
    uint32_t ent[kNoAllocMaxEntries];
};

// In host code this name is only a stand-in for the device array; kernels get the address
// from cudaGetSymbolAddress below.
static __device__ __align__(256) NoAllocScratch g_noalloc_scratch;

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
NoAllocScratch* g_noalloc_addr[kNoAllocMaxDevices] = {};

// Device address of the scratch array on the current device, looked up once per device.
kpax_status noalloc_scratch(NoAllocScratch** out)
{
    int dev = 0;
    KPAX_CUDA(cudaGetDevice(&dev));
    if(dev < 0 || dev >= kNoAllocMaxDevices) return set_error("device ordinal %d not supported", dev), KPAX_EINVAL;
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if(!g_noalloc_addr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if(e != cudaSuccess || !p)
            return set_error("cudaGetSymbolAddress(scratch) failed: %s", cudaGetErrorString(e)), KPAX_ECUDA;
        g_noalloc_addr[dev] = (NoAllocScratch*)p;
    }
    *out = g_noalloc_addr[dev];
    return KPAX_OK;
}

}  // namespace

extern "C" kpax_status kpax_propagate_batch_noalloc(const kpax_config* cfg, const float* d_obstacles, uint32_t n_obs,
                                                    const float* d_parents, const float* d_draws, uint32_t draw_stream,
                                                    uint32_t n, float* d_rows, uint8_t* d_valid, int32_t* d_steps,
                                                    void* stream)
{
    if(!cfg || (n_obs && !d_obstacles) || (n && (!d_parents || !d_rows || !d_valid)))
        return set_error("kpax_propagate_batch_noalloc: null argument"), KPAX_EINVAL;
    KParams p;
    kpax_status st = derive_params(*cfg, &p);
    if(st != KPAX_OK) return st;
    const uint32_t cells = (uint32_t)p.gdim * p.gdim * p.gdim;
    if(n_obs > kNoAllocMaxObstacles)
        return set_error("kpax_propagate_batch_noalloc: %u obstacles exceed the limit of %u", n_obs, kNoAllocMaxObstacles),
               KPAX_ECAPACITY;
    if(cells > kNoAllocMaxCells)
        return set_error("kpax_propagate_batch_noalloc: %u grid cells exceed the limit of %u", cells, kNoAllocMaxCells),
               KPAX_ECAPACITY;
    NoAllocScratch* s = nullptr;
    if((st = noalloc_scratch(&s)) != KPAX_OK) return st;
    cudaStream_t cs = (cudaStream_t)stream;
    const Grid g{s->obs, s->off, s->ent, p.wmin, 1.0f / p.cell, p.gdim};
    const bool once = n_obs && env_build_once(cells, n_obs);
    if(once) {
        k_env_build<<<1, kEnvBuildBS, sizeof(uint32_t) * cells, cs>>>(g, d_obstacles, n_obs, cells, s->obs, s->off, s->cursor, s->ent, kNoAllocMaxEntries);
        KPAX_CHECK_LAUNCH();
        count_launch(1);
    } else {
        // the array keeps the previous call's grid: the counts must start from zero
        KPAX_CUDA(cudaMemsetAsync(s->off, 0, sizeof(uint32_t) * (cells + 1), cs));
        if(n_obs) {
            if((st = env_count(g, d_obstacles, n_obs, cells, s->obs, s->off, s->cursor, cs)) != KPAX_OK) return st;
        }
    }
    if(n_obs) {
        uint32_t total = 0;
        KPAX_CUDA(cudaMemcpyAsync(&total, s->off + cells, sizeof(uint32_t), cudaMemcpyDeviceToHost, cs));
        KPAX_CUDA(cudaStreamSynchronize(cs));
        if(total > kNoAllocMaxEntries)
            return set_error("kpax_propagate_batch_noalloc: %u (cell, obstacle) pairs exceed the limit of %u", total,
                             kNoAllocMaxEntries),
                   KPAX_ECAPACITY;
        if(once && total > env_build_pairs(n_obs) &&
           (st = env_count(g, d_obstacles, n_obs, cells, s->obs, s->off, s->cursor, cs)) != KPAX_OK)
            return st;
        if(!once || total > env_build_pairs(n_obs)) {
            k_env_fill<<<warp_blocks(n_obs), 256, 0, cs>>>(g, s->obs, n_obs, s->cursor, s->ent);
            KPAX_CHECK_LAUNCH();
            count_launch(1);
        }
    }
    return launch_propagate(p, g, d_parents, d_draws, draw_stream, n, d_rows, d_valid, d_steps, cs);
}
