// kpax_device.cuh — device building blocks of the expansion step.
//
// Rounding contract with the CPU oracle (oracle/kpax_oracle.c):
//  - control draws, step counts, region ids, cell ids, goal distance and scores are computed
//    with explicitly rounded intrinsics (__fadd_rn/__fmul_rn/__fdiv_rn) so no multiply-add is
//    fused; they are bit-identical to the oracle for identical inputs;
//  - the double-integrator step is written the same way, so DI segments are bit-identical;
//  - Dubins and quadrotor RK4 use a branch-free sine/cosine (sincos_fast, within a few ulp of
//    CUDA's sincosf), tan as sin times the reciprocal cosine and the PTX approximate square root
//    and reciprocal, and spell out every rounding and fused multiply-add (so a step gives the same
//    bits in every kernel it is inlined into); they match the oracle within the propagation
//    tolerance.
#pragma once
#include <stdint.h>

#include "kpax_params.h"

namespace kpax {

// ------------------------------------------------------------------ Philox4x32-10
// Salmon et al., SC'11.  ctr = {index, iter, sub-stream, stream}, key = seed.
struct U4 {
    uint32_t x, y, z, w;
};

__device__ __forceinline__ U4 philox(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, uint32_t k0, uint32_t k1)
{
#pragma unroll
    for(int r = 0; r < 10; ++r) {
        uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
        uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
        uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
        c0 = n0, c1 = lo1, c2 = n2, c3 = lo0;
        k0 += 0x9E3779B9u, k1 += 0xBB67AE85u;
    }
    return {c0, c1, c2, c3};
}

// ((x >> 8) + 1) * 2^-24: exact, in (0, 1].
__device__ __forceinline__ float u01(uint32_t x) { return __uint2float_rn((x >> 8) + 1u) * 5.9604644775390625e-8f; }

// The six uniforms of a child: controls c0..c3, duration, frontier draw.
__device__ __forceinline__ void child_draws(const KParams& p, uint32_t stream, uint32_t iter, uint32_t index, float u[6])
{
    U4 a = philox(index, iter, 0u, stream, p.seed_lo, p.seed_hi);
    U4 b = philox(index, iter, 1u, stream, p.seed_lo, p.seed_hi);
    u[0] = u01(a.x), u[1] = u01(a.y), u[2] = u01(a.z), u[3] = u01(a.w);
    u[4] = u01(b.x), u[5] = u01(b.y);
}

__device__ __forceinline__ float reactivate_draw(const KParams& p, uint32_t stream, uint32_t iter, uint32_t index)
{
    return u01(philox(index, iter, 2u, stream, p.seed_lo, p.seed_hi).x);
}

// Goal-progress pruning of an accepted child (prune_updateFrontier_kernel, PruneKPAX.cu:466-498):
// kept when the Philox stream-5 uniform is below clamp(explorationBias + goalBias *
// clamp((d_parent - d_child) / progressScale + 1/2, 0, 1), EPSILON, 1).
__device__ __forceinline__ bool prune_keep(const KParams& p, float d_parent, float d_child, uint32_t stream, uint32_t iter,
                                           uint32_t index)
{
    const float prog = fminf(fmaxf(__fadd_rn(__fdiv_rn(__fsub_rn(d_parent, d_child), p.prune_scale), 0.5f), 0.0f), 1.0f);
    const float prob = fminf(fmaxf(__fadd_rn(p.prune_expl_bias, __fmul_rn(p.prune_goal_bias, prog)), p.eps), 1.0f);
    return u01(philox(index, iter, 5u, stream, p.seed_lo, p.seed_hi).x) < prob;
}

// ------------------------------------------------------------------ sine / cosine
// Branch-free sin and cos of one argument for |x| <= kTrigFastMax: Cody-Waite reduction by pi/2
// with pi/2 split in three parts (1.5703125 + 4.837512969970703125e-4 + 7.54978995489188216e-8),
// then the single-precision minimax polynomials of the Cephes library (S. L. Moshier, sinf.c /
// cosf.c) on [-pi/4, pi/4] and the quadrant map.  Straight-line code, so several calls interleave;
// outside the range the caller falls back to CUDA's sincosf.  Error bound checked against
// sincosf in tests/test_gpu_kernels.py.
constexpr float kTrigFastMax = 8192.0f;

__device__ __forceinline__ void sincos_fast(float x, float* sn, float* cs)
{
    // nearest integer of x * 2 / pi by adding 1.5 * 2^23, whose low mantissa bits then hold it
    const float t = __fadd_rn(__fmul_rn(x, 0.636619772367581343f), 12582912.0f);
    const float n = __fsub_rn(t, 12582912.0f);
    const uint32_t q = __float_as_uint(t);
    float r = fmaf(n, -1.5703125f, x);
    r = fmaf(n, -4.837512969970703125e-4f, r);
    r = fmaf(n, -7.54978995489188216e-8f, r);
    const float z = r * r;
    const float ps = fmaf(fmaf(fmaf(-1.9515295891e-4f, z, 8.3321608736e-3f), z, -1.6666654611e-1f), z * r, r);
    const float pc = fmaf(fmaf(fmaf(2.443315711809948e-5f, z, -1.388731625493765e-3f), z, 4.166664568298827e-2f), z * z,
                          fmaf(-0.5f, z, 1.0f));
    const bool odd = (q & 1u) != 0u;
    const float a = odd ? pc : ps, b = odd ? ps : pc;
    *sn = __uint_as_float(__float_as_uint(a) ^ ((q & 2u) << 30));
    *cs = __uint_as_float(__float_as_uint(b) ^ (((q + 1u) & 2u) << 30));
}

__device__ __forceinline__ void sincos_checked(float x, float* sn, float* cs)
{
    sincos_fast(x, sn, cs);
    if(!(fabsf(x) <= kTrigFastMax)) sincosf(x, sn, cs);  // huge or non-finite arguments
}

// (sin, cos) of up to four arguments on a path that a step rarely takes: one copy of the code for all,
// so that it does not crowd the step's instructions.  Each as sincos_checked; `huge_only` leaves the
// arguments within kTrigFastMax as they are.
template <int N>
__device__ __forceinline__ void sincos_rare(const float (&x)[N], float* sc, bool huge_only)
{
#pragma unroll 1
    for(int d = 0; d < N; ++d) {
        float v = x[0], s, c;
#pragma unroll
        for(int j = 1; j < N; ++j) v = d == j ? x[j] : v;
        if(huge_only && fabsf(v) <= kTrigFastMax) continue;
        sincos_checked(v, &s, &c);
#pragma unroll
        for(int j = 0; j < N; ++j) {
            sc[2 * j] = d == j ? s : sc[2 * j];
            sc[2 * j + 1] = d == j ? c : sc[2 * j + 1];
        }
    }
}

// N arguments with one test for the common case (a NaN or infinity fails it).
template <int N>
__device__ __forceinline__ void sincos_all(const float (&x)[N], float* sc)
{
    bool fast = true;
#pragma unroll
    for(int d = 0; d < N; ++d) {
        sincos_fast(x[d], &sc[2 * d], &sc[2 * d + 1]);
        fast = fast && fabsf(x[d]) <= kTrigFastMax;
    }
    if(!fast) sincos_rare(x, sc, true);
}

// sin and cos of a0 + d from s0 = sin(a0), c0 = cos(a0) by the angle-sum identity, with the
// Taylor series of sin(d) to d^7 and cos(d) - 1 to d^8: for |d| <= kShiftMax the truncation error
// is below 2e-11, so the result is within a few ulp of sin/cos of the rounded sum a0 + d.  The RK4
// stages evaluate the attitude at a0 + (h/2) k and a0 + h k; this replaces three of every four
// full evaluations per angle and step.
constexpr float kShiftMax = 0.25f;
struct ShiftCoef {
    float sd, cm;  // sin(d) and cos(d) - 1
};

__device__ __forceinline__ ShiftCoef shift_coef(float d)
{
    const float d2 = d * d;
    return {fmaf(d * d2, fmaf(d2, fmaf(d2, -1.0f / 5040.0f, 1.0f / 120.0f), -1.0f / 6.0f), d),
            d2 * fmaf(d2, fmaf(d2, fmaf(d2, 1.0f / 40320.0f, -1.0f / 720.0f), 1.0f / 24.0f), -0.5f)};
}

__device__ __forceinline__ void sincos_apply(float s0, float c0, ShiftCoef k, float* sn, float* cs)
{
    *sn = fmaf(s0, k.cm, fmaf(c0, k.sd, s0));
    *cs = fmaf(c0, k.cm, fmaf(-s0, k.sd, c0));
}

__device__ __forceinline__ void sincos_shift(float s0, float c0, float d, float* sn, float* cs)
{
    sincos_apply(s0, c0, shift_coef(d), sn, cs);
}

// Square root and reciprocal by the PTX approximations sqrt.approx.f32 / rcp.approx.f32 (about one
// ulp, against the half ulp of the correctly rounded forms, which cost a Newton step and a
// special-case branch each): the quadrotor right-hand side takes two roots and one reciprocal
// per stage on its dependency chain.
__device__ __forceinline__ float sqrt_approx(float x)
{
    float y;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float rcp_approx(float x)
{
    float y;
    asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Two FP32 values per instruction (fma.rn.f32x2 and friends of sm_100a): each half rounds as the scalar
// operation does.  The quadrotor's step is bound by its instruction count (559 of 800 instructions per
// step on the FMA pipes); its element-wise updates take half as many this way: 2^20 segments without
// obstacles 701 -> 663 us, 2^16 62.2 -> 58.2 us.
typedef unsigned long long F2;

__device__ __forceinline__ F2 f2(float lo, float hi)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ F2 f2(float x) { return f2(x, x); }
__device__ __forceinline__ float2 unpack(F2 v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// float -> int with the reference's device semantics (saturating, NaN -> 0).
__device__ __forceinline__ int f2i(float x) { return __float2int_rz(x); }
__device__ __forceinline__ int clampi(int v, int lo, int hi) { return min(max(v, lo), hi); }

// ------------------------------------------------------------------ regions (Graph.cu:99-205)
// state s: the first 3 + cdim + vdim floats are read.  The attitude and velocity digits are
// visited with compile-time state indices (j < SD, predicated on the runtime dimensions) so the
// state stays in registers; the mixed-radix ids are the same integers as the reference's loops.
template <int SD>
__device__ __forceinline__ int region_r1(const KParams& p, const float* s)
{
    int w = 0, f = 1;
#pragma unroll
    for(int i = 2; i >= 0; --i) {
        int idx = f2i(__fdiv_rn(__fmul_rn((float)p.W1, __fsub_rn(s[i], p.wmin)), p.wspan));
        w += f * clampi(idx, 0, p.W1 - 1);
        f *= p.W1;
    }
    if(p.w_only) return w;
    int a = 0, v = 0;
    const int ce = 3 + p.cdim, ve = ce + p.vdim;
    if(p.C1 > 1) {  // digit i = j - 3, the last one least significant
#pragma unroll
        for(int j = 3; j < SD; ++j) {
            if(j < ce) {
                const float x = s[j];
                int idx = 0;
                for(int k = 0; k < p.C1 - 1; ++k) idx += (x >= p.cthr1[k]);
                a = a * p.C1 + idx;
            }
        }
    }
    if(p.V1 > 1) {
#pragma unroll
        for(int j = 3; j < SD; ++j) {
            if(j >= ce && j < ve) {
                int idx = f2i(__fdiv_rn(__fmul_rn((float)p.V1, __fsub_rn(s[j], p.vmin_r)), p.vspan));
                v = v * p.V1 + clampi(idx, 0, p.V1 - 1);
            }
        }
    }
    return w * p.r1_mulW + a * p.r1_mulA + v;
}

// getSubRegion (Graph.cu:155-205).  The R1 min corner is W_MIN + i*W_R1_SIZE (float),
// C_MIN + i*C_R1_SIZE (double, tabulated) and V_MIN + i*V_R1_SIZE (float), as Graph.cu:69-95.
// The R1 id's cell digits are decoded as they are consumed, least significant first.  In compat
// mode the id is decoded the way initializeRegions_kernel lays out its table (Graph.cu:58-96:
// workspace part fastest, C_R1^2 attitude cells, then velocity); otherwise in getRegion's order
// (workspace part slowest).
template <int SD>
__device__ __forceinline__ int region_r2(const KParams& p, const float* s, int r1)
{
    int wr, ar, vr;
    if(p.compat) {
        const int W3 = p.W1 * p.W1 * p.W1;
        wr = r1 % W3;
        ar = (r1 / W3) % (p.C1 * p.C1);
        vr = (r1 / (W3 * p.C1 * p.C1)) % p.V1;
    } else {
        wr = r1 / p.r1_mulW;
        const int rem = r1 - wr * p.r1_mulW;
        ar = rem / p.r1_mulA;
        vr = rem - ar * p.r1_mulA;
    }
    int w = 0, f = 1;
#pragma unroll
    for(int i = 2; i >= 0; --i) {
        const int dw = wr % p.W1;
        wr /= p.W1;
        const float m = __fadd_rn(p.wmin, __fmul_rn((float)dw, p.w1size));
        int idx = f2i(__fdiv_rn(__fmul_rn((float)p.W2, __fsub_rn(s[i], m)), p.w1size));
        w += f * clampi(idx, 0, p.W2 - 1);
        f *= p.W2;
    }
    int a = 0, v = 0;
    const int ce = 3 + p.cdim, ve = ce + p.vdim;
    if(p.C2 > 1) {
        f = 1;
#pragma unroll
        for(int j = SD - 1; j >= 3; --j) {
            if(j < ce) {
                const int da = ar % p.C1;
                ar /= p.C1;
                const float x = __fmul_rn((float)p.C2, __fsub_rn(s[j], p.cmin_tab[da]));
                int idx = 0;
                for(int k = 0; k < p.C2 - 1; ++k) idx += (x >= p.cthr2[k]);
                a += f * idx;
                f *= p.C2;
            }
        }
    }
    if(p.V2 > 1) {
        f = 1;
#pragma unroll
        for(int j = SD - 1; j >= 3; --j) {
            if(j >= ce && j < ve) {
                const int dv = vr % p.V1;
                vr /= p.V1;
                const float m = __fadd_rn(p.vmin_r, __fmul_rn((float)dv, p.v1size));
                int idx = f2i(__fdiv_rn(__fmul_rn((float)p.V2, __fsub_rn(s[j], m)), p.v1size));
                v += f * clampi(idx, 0, p.V2 - 1);
                f *= p.V2;
            }
        }
    }
    return r1 * p.P + (w * p.r2_mulW + a * p.r2_mulA + v);
}

// ------------------------------------------------------------------ spatial hash
// CSR grid over the workspace cube; obstacles as float4 pairs (min xyz, max xyz).
struct Grid {
    const float4* __restrict__ obs;
    const uint32_t* __restrict__ off;  // cells + 1
    const uint32_t* __restrict__ ent;
    float wmin, inv_cell;  // 1 / GRID_CELL_SIZE
    int dim;
};

// Cell of a coordinate.  Any non-decreasing map gives the brute-force verdict as long as the
// build and the query use the same one; a multiply by the reciprocal replaces the reference's
// division (spatialHash.cuh:236-246), which can move a point on a cell face by one cell.
__device__ __forceinline__ int grid_coord(const Grid& g, float x)
{
    return clampi(f2i(__fmul_rn(__fsub_rn(x, g.wmin), g.inv_cell)), 0, g.dim - 1);
}

// isMotionValidSpatialHash (spatialHash.cu:145-194) with isBroadPhaseValid (collisionCheck.cu:3-10):
// true when no obstacle overlaps the box strictly in all three dimensions.
// The box's cells are x0..x1, y0..y1, z0..z1.
__device__ __forceinline__ bool box_free_cells(const Grid& g, const float lo[3], const float hi[3], int x0, int y0, int z0,
                                               int x1, int y1, int z1)
{
    for(int gz = z0; gz <= z1; ++gz)
        for(int gy = y0; gy <= y1; ++gy)
            for(int gx = x0; gx <= x1; ++gx) {
                const int c = gx + g.dim * (gy + g.dim * gz);
                const uint32_t b = __ldg(g.off + c), e = __ldg(g.off + c + 1);
                for(uint32_t k = b; k < e; ++k) {
                    const uint32_t o = __ldg(g.ent + k);
                    const float4 a = __ldg(g.obs + 2 * o), m = __ldg(g.obs + 2 * o + 1);
                    if(hi[0] > a.x && m.x > lo[0] && hi[1] > a.y && m.y > lo[1] && hi[2] > a.z && m.z > lo[2]) return false;
                }
            }
    return true;
}

__device__ __forceinline__ bool box_free(const Grid& g, const float lo[3], const float hi[3])
{
    return box_free_cells(g, lo, hi, grid_coord(g, lo[0]), grid_coord(g, lo[1]), grid_coord(g, lo[2]), grid_coord(g, hi[0]),
                          grid_coord(g, hi[1]), grid_coord(g, hi[2]));
}

// The swept box of one step, p0 -> p1.  cells: the cell coordinates of p0 on entry, replaced by p1's (a
// step's end is the next one's start).  The cell map is non-decreasing, so the box's cells are the range of
// its two corners' cells.
__device__ __forceinline__ bool step_free(const Grid& g, const float p0[3], const float p1[3], int cells[3])
{
    float lo[3], hi[3];
    int c0[3], c1[3];
#pragma unroll
    for(int d = 0; d < 3; ++d) {
        lo[d] = fminf(p0[d], p1[d]), hi[d] = fmaxf(p0[d], p1[d]);
        const int c = grid_coord(g, p1[d]);
        c0[d] = min(cells[d], c), c1[d] = max(cells[d], c);
        cells[d] = c;
    }
    return box_free_cells(g, lo, hi, c0[0], c0[1], c0[2], c1[0], c1[1], c1[2]);
}

// First of `limit` consecutive swept boxes, box j from pos(j) to pos(j + 1), that an obstacle
// overlaps, or `limit` when all are free.  lo / hi: the hull of the boxes.  One walk over the cells
// of the hull finds the obstacles that overlap it, and only those are tested against the boxes, so
// the dependent lookups (offsets, entry, obstacle) are paid once per group of steps instead of at
// every step.  A box's cells lie inside its hull's (the cell map is non-decreasing) and an obstacle
// that overlaps a box overlaps the hull, so the answer is the per-box query's.
template <class F>
__device__ __forceinline__ int first_hit(const Grid& g, const float lo[3], const float hi[3], int limit, F pos)
{
    const int x0 = grid_coord(g, lo[0]), y0 = grid_coord(g, lo[1]), z0 = grid_coord(g, lo[2]);
    const int x1 = grid_coord(g, hi[0]), y1 = grid_coord(g, hi[1]), z1 = grid_coord(g, hi[2]);
    for(int gz = z0; gz <= z1; ++gz)
        for(int gy = y0; gy <= y1; ++gy)
            for(int gx = x0; gx <= x1; ++gx) {
                const int c = gx + g.dim * (gy + g.dim * gz);
                const uint32_t b = __ldg(g.off + c), e = __ldg(g.off + c + 1);
                for(uint32_t k = b; k < e; ++k) {
                    const uint32_t o = __ldg(g.ent + k);
                    const float4 a = __ldg(g.obs + 2 * o), m = __ldg(g.obs + 2 * o + 1);
                    if(hi[0] > a.x && m.x > lo[0] && hi[1] > a.y && m.y > lo[1] && hi[2] > a.z && m.z > lo[2]) {
                        float q[3] = {pos(0, 0), pos(0, 1), pos(0, 2)};
                        for(int j = 0; j < limit; ++j) {
                            const float r[3] = {pos(j + 1, 0), pos(j + 1, 1), pos(j + 1, 2)};
                            if(fmaxf(q[0], r[0]) > a.x && m.x > fminf(q[0], r[0]) && fmaxf(q[1], r[1]) > a.y &&
                               m.y > fminf(q[1], r[1]) && fmaxf(q[2], r[2]) > a.z && m.z > fminf(q[2], r[2]))
                                limit = j;
                            q[0] = r[0], q[1] = r[1], q[2] = r[2];
                        }
                        if(limit == 0) return 0;
                    }
                }
            }
    return limit;
}

// x * 0 is +-0 for a finite x and NaN for an infinite or NaN one, so the sum of those products is
// 0 exactly when every value is finite (n even).
__device__ __forceinline__ bool finite_all(const float* s, int n)
{
    F2 a = f2(0.0f);
#pragma unroll
    for(int i = 0; i + 1 < n; i += 2) a = fma2(f2(s[i], s[i + 1]), f2(0.0f), a);
    const float2 v = unpack(a);
    return __fadd_rn(v.x, v.y) == 0.0f;
}

// ------------------------------------------------------------------ controls
// statePropagatorSpatialHash.cu:74-77 / 141-144 / 236-241: c = MIN + u * (MAX - MIN);
// steps = 1 + (int)(u * N) (N + 1 when u == 1, as in the reference).
__device__ __forceinline__ int draw_controls(const KParams& p, const float u[6], float c[4])
{
#pragma unroll
    for(int i = 0; i < 4; ++i) c[i] = __fadd_rn(p.clo[i], __fmul_rn(u[i], p.crng[i]));
    return p.fixed_steps ? p.nsteps : 1 + f2i(__fmul_rn(u[4], (float)p.nsteps));
}

// ------------------------------------------------------------------ models
// One integration step per model with the reference's bounds checks; the swept box's collision
// query, the reference's last check of a step, is made by run_steps for groups of steps.  The output
// row holds the state after the failing step, as the reference's break does.

// The configuration values a step reads, copied to registers once per segment (the planner keeps
// its KParams in shared memory).
struct StepParams {
    float h, hh, h6, vmin, vmax, ws_lo, ws_hi, pitch_lo, pitch_hi;
};

__device__ __forceinline__ StepParams step_params(const KParams& p)
{
    return {p.h, p.hh, p.h6, p.vmin, p.vmax, p.ws_lo, p.ws_hi, p.pitch_lo, p.pitch_hi};
}

// Double integrator, statePropagatorSpatialHash.cu:72-134 (x += h(5v + 2ah)/6, not textbook RK4).  The terms
// that depend on the segment's acceleration only (a*h/2, a*h and the velocity increment
// (a + 2a + 2a + a)*h/6) are computed once per segment, with the same rounded operations.
struct DIConsts {
    float ah2[3], ah[3], dv[3];
};

__device__ __forceinline__ DIConsts di_consts(const KParams& p, const float* c)
{
    DIConsts k;
#pragma unroll
    for(int d = 0; d < 3; ++d) {
        const float a = c[d];
        k.ah[d] = __fmul_rn(a, p.h);
        k.ah2[d] = __fdiv_rn(k.ah[d], 2.0f);
        const float asum = __fadd_rn(__fadd_rn(__fadd_rn(a, __fmul_rn(2.0f, a)), __fmul_rn(2.0f, a)), a);
        k.dv[d] = __fdiv_rn(__fmul_rn(asum, p.h), 6.0f);
    }
    return k;
}

// One step from s in place; false when the step fails a check (velocity box, workspace, finite).
__device__ __forceinline__ bool step_di(const StepParams& p, float* s, const DIConsts& k)
{
    const float h = p.h;
#pragma unroll
    for(int d = 0; d < 3; ++d) {
        const float v = s[3 + d];
        // (v + (v + 2*(v + a*h/2) + (v + a*h))) * h / 6
        const float t1 = __fadd_rn(v, k.ah2[d]);
        const float t2 = __fadd_rn(v, k.ah[d]);
        const float sum = __fadd_rn(v, __fadd_rn(__fadd_rn(v, __fmul_rn(2.0f, t1)), t2));
        s[d] = __fadd_rn(s[d], __fdiv_rn(__fmul_rn(sum, h), 6.0f));
        s[3 + d] = __fadd_rn(v, k.dv[d]);  // v + (a + 2a + 2a + a) * h / 6
    }
    if(s[3] < p.vmin || s[3] > p.vmax || s[4] < p.vmin || s[4] > p.vmax || s[5] < p.vmin || s[5] > p.vmax) return false;
    if(s[0] < p.ws_lo || s[0] > p.ws_hi || s[1] < p.ws_lo || s[1] > p.ws_hi || s[2] < p.ws_lo || s[2] > p.ws_hi) return false;
    return finite_all(s, 6);
}

// Dubins airplane, statePropagatorSpatialHash.cu:139-229; c = (a, yawRate, pitchRate).  One step
// from s in place; false when the step fails a check (speed, pitch range, workspace, finite).
// The stage angle increments of a Dubins segment are its fixed rates times h/2 and h, so their
// sine / cosine series are evaluated once per segment.
struct DubinsShifts {
    bool shift;  // all four increments within kShiftMax
    ShiftCoef p1, y1, p2, y2;
};

__device__ __forceinline__ DubinsShifts dubins_shifts(const KParams& p, const float* c)
{
    const float h = p.h, hh = p.hh, yr = c[1], pr = c[2];
    return {fmaxf(fabsf(__fmul_rn(h, pr)), fabsf(__fmul_rn(h, yr))) <= kShiftMax, shift_coef(__fmul_rn(hh, pr)),
            shift_coef(__fmul_rn(hh, yr)), shift_coef(__fmul_rn(h, pr)), shift_coef(__fmul_rn(h, yr))};
}

__device__ __forceinline__ bool step_dubins(const StepParams& p, float* s, const float* c, const DubinsShifts& k)
{
    const float h = p.h, hh = p.hh, h6 = p.h6;
    const float a = c[0], yr = c[1], pr = c[2];
    const float yaw = s[3], pitch = s[4], v = s[5];
    float sp0, cp0, sy0, cy0, sp1, cp1, sy1, cy1, sp2, cp2, sy2, cy2;
    {
        const float x[2] = {pitch, yaw};
        float sc[4];
        sincos_all(x, sc);
        sp0 = sc[0], cp0 = sc[1], sy0 = sc[2], cy0 = sc[3];
    }
    if(k.shift) {
        sincos_apply(sp0, cp0, k.p1, &sp1, &cp1);
        sincos_apply(sy0, cy0, k.y1, &sy1, &cy1);
        sincos_apply(sp0, cp0, k.p2, &sp2, &cp2);
        sincos_apply(sy0, cy0, k.y2, &sy2, &cy2);
    } else {
        const float x[4] = {__fmaf_rn(hh, pr, pitch), __fmaf_rn(hh, yr, yaw), __fmaf_rn(h, pr, pitch), __fmaf_rn(h, yr, yaw)};
        float sc[8] = {};
        sincos_rare(x, sc, false);
        sp1 = sc[0], cp1 = sc[1], sy1 = sc[2], cy1 = sc[3], sp2 = sc[4], cp2 = sc[5], sy2 = sc[6], cy2 = sc[7];
    }
    // every rounding written out (as the quadrotor's): the same bits wherever the step is inlined
    const float vm = __fmaf_rn(hh, a, v), ve = __fmaf_rn(h, a, v);
    const float vmc = __fmul_rn(vm, cp1), vc0 = __fmul_rn(v, cp0), vc2 = __fmul_rn(ve, cp2);
    const float mx = __fmul_rn(vmc, cy1), my = __fmul_rn(vmc, sy1), mz = __fmul_rn(vm, sp1);
    // (k1 + 2 (k2 + k3)) + k4 with k2 = k3 (the reference's stage sum; 2 x is exact)
    s[0] = __fmaf_rn(h6, __fmaf_rn(vc2, cy2, __fmaf_rn(2.0f, __fadd_rn(mx, mx), __fmul_rn(vc0, cy0))), s[0]);
    s[1] = __fmaf_rn(h6, __fmaf_rn(vc2, sy2, __fmaf_rn(2.0f, __fadd_rn(my, my), __fmul_rn(vc0, sy0))), s[1]);
    s[2] = __fmaf_rn(h6, __fmaf_rn(ve, sp2, __fmaf_rn(2.0f, __fadd_rn(mz, mz), __fmul_rn(v, sp0))), s[2]);
    s[3] = __fmaf_rn(h, yr, yaw);
    s[4] = __fmaf_rn(h, pr, pitch);
    s[5] = __fmaf_rn(h6, __fadd_rn(__fmaf_rn(2.0f, __fadd_rn(a, a), a), a), v);
    if(s[5] < p.vmin || s[5] > p.vmax || s[4] < p.pitch_lo || s[4] > p.pitch_hi) return false;
    if(s[0] < p.ws_lo || s[0] > p.ws_hi || s[1] < p.ws_lo || s[1] > p.ws_hi || s[2] < p.ws_lo || s[2] > p.ws_hi) return false;
    return finite_all(s, 6);
}

// Quadrotor right-hand side, statePropagator.cu:325-370, in its two halves: the kinematics
// (position and Euler-angle rates, xd[0..5]) read the attitude's sines and cosines and the body
// velocities and rates; the dynamics (velocity and rate derivatives, xd[6..11]) read sin/cos of
// roll and pitch, the velocities, rates and controls.  Model constants NU 10e-3, MU 2e-6, IX 1,
// IY 1, IZ 2, GRAVITY -9.81, MASS 1 (config.h:300-308).  Every operation is written out (explicit
// roundings and fused multiply-adds), so the result does not depend on how the compiler contracts
// the expressions where the step is inlined.
struct QuadTrig {
    float sf, cf, st, ct, sp, cp;  // sin / cos of roll, pitch, yaw
};
struct QuadRates {
    float u, v, w, p, q, r;  // body velocities and rates
};

__device__ __forceinline__ void quad_kin(float* xd, const QuadTrig& t, const QuadRates& b)
{
    const float sec = rcp_approx(t.ct);  // tan(theta) = sin * sec, 1/cos(theta) = sec
    const float sfst = __fmul_rn(t.sf, t.st), cfst = __fmul_rn(t.cf, t.st);
    const float r01 = __fmaf_rn(sfst, t.cp, -__fmul_rn(t.cf, t.sp)), r02 = __fmaf_rn(cfst, t.cp, __fmul_rn(t.sf, t.sp));
    const float r11 = __fmaf_rn(sfst, t.sp, __fmul_rn(t.cf, t.cp)), r12 = __fmaf_rn(cfst, t.sp, -__fmul_rn(t.sf, t.cp));
    xd[0] = __fmaf_rn(r02, b.w, __fmaf_rn(r01, b.v, __fmul_rn(__fmul_rn(t.ct, t.cp), b.u)));
    xd[1] = __fmaf_rn(r12, b.w, __fmaf_rn(r11, b.v, __fmul_rn(__fmul_rn(t.ct, t.sp), b.u)));
    xd[2] = __fmaf_rn(__fmul_rn(t.cf, t.ct), b.w, __fmaf_rn(__fmul_rn(t.sf, t.ct), b.v, -__fmul_rn(t.st, b.u)));
    const float qr = __fmaf_rn(b.q, t.sf, __fmul_rn(b.r, t.cf));
    xd[3] = __fmaf_rn(qr, __fmul_rn(t.st, sec), b.p);
    xd[4] = __fmaf_rn(b.q, t.cf, -__fmul_rn(b.r, t.sf));
    xd[5] = __fmul_rn(qr, sec);
}

__device__ __forceinline__ void quad_dyn(float* xd, float sf, float cf, float st, float ct, const QuadRates& b, const float* c)
{
    const float NU = 10e-3f, MU = 2e-6f, G = -9.81f;
    const float XYZ = __fmul_rn(-NU, sqrt_approx(__fmaf_rn(b.w, b.w, __fmaf_rn(b.v, b.v, __fmul_rn(b.u, b.u)))));
    const float gct = __fmul_rn(G, ct);
    xd[0] = __fmaf_rn(XYZ, b.u, __fmaf_rn(-G, st, __fmaf_rn(b.r, b.v, -__fmul_rn(b.q, b.w))));
    xd[1] = __fmaf_rn(XYZ, b.v, __fmaf_rn(gct, sf, __fmaf_rn(b.p, b.w, -__fmul_rn(b.r, b.u))));
    xd[2] = __fadd_rn(__fmaf_rn(XYZ, b.w, __fmaf_rn(gct, cf, __fmaf_rn(b.q, b.u, -__fmul_rn(b.p, b.v)))), c[0]);
    const float LMN = __fmul_rn(-MU, sqrt_approx(__fmaf_rn(b.r, b.r, __fmaf_rn(b.q, b.q, __fmul_rn(b.p, b.p)))));
    xd[3] = __fadd_rn(__fmaf_rn(LMN, b.p, -__fmul_rn(b.q, b.r)), c[1]);  // (IY - IZ)/IX = -1, 1/IX = 1
    xd[4] = __fadd_rn(__fmaf_rn(LMN, b.q, __fmul_rn(b.p, b.r)), c[2]);   // (IZ - IX)/IY = 1,  1/IY = 1
    // (IX - IY)/IZ = 0 (the product still carries a non-finite rate), 1/IZ = 0.5
    xd[5] = __fmaf_rn(0.5f, c[3], __fmaf_rn(0.5f, __fmul_rn(LMN, b.r), __fmul_rn(0.0f, __fmul_rn(b.p, b.q))));
}

// The first RK4 stage is evaluated at x0 + 1 * 0: the state is x0 + 0 (which only turns -0 into
// +0) and the angle-sum shift by 0 reduces to sin + 0 and cos.  trig0: (sin, cos) of the three
// Euler angles of x0.
__device__ __forceinline__ QuadTrig quad_first_trig(const float* trig0)
{
    return {__fadd_rn(trig0[0], 0.0f), trig0[1], __fadd_rn(trig0[2], 0.0f), trig0[3], __fadd_rn(trig0[4], 0.0f), trig0[5]};
}

__device__ __forceinline__ QuadRates quad_first_rates(const float* v0)
{
    return {__fadd_rn(v0[0], 0.0f), __fadd_rn(v0[1], 0.0f), __fadd_rn(v0[2], 0.0f),
            __fadd_rn(v0[3], 0.0f), __fadd_rn(v0[4], 0.0f), __fadd_rn(v0[5], 0.0f)};
}

// The attitude at a0 + delta * ka (later stages): sin and cos by the angle-sum shift of trig0;
// large attitude increments or non-finite values are evaluated at the rounded angles.
__device__ __forceinline__ QuadTrig quad_stage_trig(const float* a0, const float* trig0, const float* ka, float delta)
{
    QuadTrig t;
    const float d0 = __fmul_rn(delta, ka[0]), d1 = __fmul_rn(delta, ka[1]), d2 = __fmul_rn(delta, ka[2]);
    if(fmaxf(fabsf(d0), fmaxf(fabsf(d1), fabsf(d2))) <= kShiftMax) {
        sincos_shift(trig0[0], trig0[1], d0, &t.sf, &t.cf);
        sincos_shift(trig0[2], trig0[3], d1, &t.st, &t.ct);
        sincos_shift(trig0[4], trig0[5], d2, &t.sp, &t.cp);
    } else {
        const float x[3] = {__fadd_rn(a0[0], d0), __fadd_rn(a0[1], d1), __fadd_rn(a0[2], d2)};
        float sc[6] = {};
        sincos_rare(x, sc, false);
        t = {sc[0], sc[1], sc[2], sc[3], sc[4], sc[5]};
    }
    return t;
}

__device__ __forceinline__ QuadRates quad_stage_rates(const float* v0, const float* kv, float delta)
{
    const F2 d = f2(delta);
    const float2 a = unpack(fma2(d, f2(kv[0], kv[1]), f2(v0[0], v0[1]))), b = unpack(fma2(d, f2(kv[2], kv[3]), f2(v0[2], v0[3]))),
                 c = unpack(fma2(d, f2(kv[4], kv[5]), f2(v0[4], v0[5])));
    return {a.x, a.y, b.x, b.y, c.x, c.y};
}

__device__ __forceinline__ void quad_trig0(const float* a0, float* trig0)
{
    const float x[3] = {a0[0], a0[1], a0[2]};
    sincos_all(x, trig0);
}

// The per-step bounds checks of each half (velocity box; workspace; finite).
// A box check of three values by their minimum and maximum: fminf / fmaxf pass over a NaN that the
// six comparisons would let through as well, and the finite check rejects it either way, so the
// verdict is the comparisons'.
__device__ __forceinline__ bool in_box3(const float* v, float lo, float hi)
{
    return !(fminf(fminf(v[0], v[1]), v[2]) < lo || fmaxf(fmaxf(v[0], v[1]), v[2]) > hi);
}

__device__ __forceinline__ bool quad_dyn_ok(const StepParams& p, const float* v)
{
    return in_box3(v, p.vmin, p.vmax) && finite_all(v, 6);
}

__device__ __forceinline__ bool quad_kin_ok(const StepParams& p, const float* x)
{
    return in_box3(x, p.ws_lo, p.ws_hi) && finite_all(x, 6);
}

// Quadrotor RK4, statePropagatorSpatialHash.cu:234-308: four stages, the stage sum in the
// reference's order ((k1 + 2k2) + 2k3) + k4.  One step from s in place; false when the step fails
// a check (velocity box, workspace, finite).
__device__ __forceinline__ bool step_quad(const StepParams& p, float* s, const float* c)
{
    const float h = p.h, hh = p.hh, h6 = p.h6;
    float k[12], trig0[6];
    F2 acc[6];
    quad_trig0(s + 3, trig0);
    {
        const QuadTrig t = quad_first_trig(trig0);
        const QuadRates b = quad_first_rates(s + 6);
        quad_kin(k, t, b);
        quad_dyn(k + 6, t.sf, t.cf, t.st, t.ct, b, c);
    }
#pragma unroll
    for(int j = 0; j < 6; ++j) acc[j] = f2(k[2 * j], k[2 * j + 1]);
#pragma unroll 1
    for(int stage = 1; stage < 4; ++stage) {
        const float delta = stage == 3 ? h : hh, w = stage == 3 ? 1.0f : 2.0f;
        const QuadTrig t = quad_stage_trig(s + 3, trig0, k + 3, delta);
        const QuadRates b = quad_stage_rates(s + 6, k + 6, delta);
        quad_kin(k, t, b);
        quad_dyn(k + 6, t.sf, t.cf, t.st, t.ct, b, c);
#pragma unroll
        for(int j = 0; j < 6; ++j) acc[j] = fma2(f2(w), f2(k[2 * j], k[2 * j + 1]), acc[j]);
    }
#pragma unroll
    for(int j = 0; j < 6; ++j) {
        const float2 v = unpack(fma2(f2(h6), acc[j], f2(s[2 * j], s[2 * j + 1])));
        s[2 * j] = v.x, s[2 * j + 1] = v.y;
    }
    return quad_dyn_ok(p, s + 6) && quad_kin_ok(p, s);
}

// Per-segment constants of a model's step (the double integrator's acceleration terms, the Dubins
// stage shifts; nothing for the quadrotor).
struct NoSegmentConsts {};
template <int M>
__device__ __forceinline__ auto segment_consts(const KParams& p, const float* c)
{
    if constexpr(M == KPAX_MODEL_DUBINS_AIRPLANE) return dubins_shifts(p, c);
    else if constexpr(M == KPAX_MODEL_DOUBLE_INTEGRATOR) return di_consts(p, c);
    else return NoSegmentConsts{};
}

template <int M, class K>
__device__ __forceinline__ bool model_step(const StepParams& p, float* s, const float* c, const K& k)
{
    if constexpr(M == KPAX_MODEL_DOUBLE_INTEGRATOR) return step_di(p, s, k);
    else if constexpr(M == KPAX_MODEL_DUBINS_AIRPLANE) return step_dubins(p, s, c, k);
    else return step_quad(p, s, c);
}

template <int M>
struct ModelDims;
template <>
struct ModelDims<KPAX_MODEL_DOUBLE_INTEGRATOR> {
    static constexpr int SD = 6, CD = 3;
};
template <>
struct ModelDims<KPAX_MODEL_DUBINS_AIRPLANE> {
    static constexpr int SD = 6, CD = 3;
};
template <>
struct ModelDims<KPAX_MODEL_QUADROTOR> {
    static constexpr int SD = 12, CD = 4;
};

template <int SD>
__device__ __forceinline__ void save_state(float* dst, const float* s)
{
    if constexpr(SD == 12) {
#pragma unroll
        for(int q = 0; q < 3; ++q)
            reinterpret_cast<float4*>(dst)[q] = make_float4(s[4 * q], s[4 * q + 1], s[4 * q + 2], s[4 * q + 3]);
    } else {
#pragma unroll
        for(int q = 0; q < SD / 2; ++q) reinterpret_cast<float2*>(dst)[q] = make_float2(s[2 * q], s[2 * q + 1]);
    }
}

template <int SD>
__device__ __forceinline__ void take_state(const float* src, float* s)
{
    if constexpr(SD == 12) {
#pragma unroll
        for(int q = 0; q < 3; ++q) {
            const float4 v = reinterpret_cast<const float4*>(src)[q];
            s[4 * q] = v.x, s[4 * q + 1] = v.y, s[4 * q + 2] = v.z, s[4 * q + 3] = v.w;
        }
    } else {
#pragma unroll
        for(int q = 0; q < SD / 2; ++q) {
            const float2 v = reinterpret_cast<const float2*>(src)[q];
            s[2 * q] = v.x, s[2 * q + 1] = v.y;
        }
    }
}

// Runs a segment from step `done` up to step `end` (in place), checking every step like the
// reference; returns false when a step fails, and leaves the number of steps executed (the failing
// one included) in `done`.
//
// K > 1: steps are taken in groups of up to K.  The group is integrated with the bounds checks only, each
// step's state kept in `save`, then one walk over the obstacles near the group's hull finds its first
// colliding step (first_hit), and a segment that collides takes the state after that step back from
// `save`.  The lookups of a query are a chain of dependent loads walked at the pace of the warp's slowest
// lane, so the fewer walks the better; K is bounded by the shared memory of the states.  B200, groups of
// five against a query per step: expansion of 2^16 quadrotor children in the building scene 83.2 -> 67.3
// us, 2^14 children 67 -> 57 us, Dubins in the forest 27.0 -> 22.7 us; 2^22 Dubins segments 848 -> 672 us;
// the double integrator, whose expansion is mostly its fixed part, 18 us either way.  save: this thread's
// SD floats of the first step of the block's K x `threads` x SD (a warp's 16- or 8-byte accesses to them
// are conflict-free).
// K == 1: a query per step, nothing kept (save is not used): see grouped().
template <int M, int K, class C>
__device__ __forceinline__ bool run_steps(const StepParams& p, const Grid& g, float* s, const float* c, const C& k, int end,
                                          int& done, float* save, int threads)
{
    constexpr int SD = ModelDims<M>::SD;
    if constexpr(K == 1) {
        int cells[3] = {grid_coord(g, s[0]), grid_coord(g, s[1]), grid_coord(g, s[2])};
        while(done < end) {
            const float p0[3] = {s[0], s[1], s[2]};
            ++done;
            if(!model_step<M>(p, s, c, k) || !step_free(g, p0, s, cells)) return false;
        }
        return true;
    }
    const int stride = threads * SD;
    while(done < end) {
        const int m = min(K, end - done);
        const float p0[3] = {s[0], s[1], s[2]};
        float lo[3] = {p0[0], p0[1], p0[2]}, hi[3] = {p0[0], p0[1], p0[2]};
        int n = 0;  // steps of the group within bounds
        bool ok = true;
#pragma unroll 1
        while(n < m) {
            ok = model_step<M>(p, s, c, k);
            save_state<SD>(save + n * stride, s);
            if(!ok) break;
#pragma unroll
            for(int d = 0; d < 3; ++d) lo[d] = fminf(lo[d], s[d]), hi[d] = fmaxf(hi[d], s[d]);
            ++n;
        }
        const int hit = n ? first_hit(g, lo, hi, n, [&](int j, int d) { return j ? save[(j - 1) * stride + d] : p0[d]; }) : 0;
        if(hit < n) {
            take_state<SD>(save + hit * stride, s);
            ok = false;
        }
        if(!ok) {
            done += hit + 1;
            return false;
        }
        done += m;
    }
    return true;
}

// Propagates `steps` steps from s (in place) and returns validity; `done` receives the number of
// steps executed (the failing one included).
template <int M, int K>
__device__ __forceinline__ bool propagate(const KParams& p, const Grid& g, float* s, const float* c, int steps, int& done,
                                          float* save, int threads)
{
    const auto k = segment_consts<M>(p, c);
    const StepParams sp = step_params(p);
    const Grid gl = g;  // register copy of the grid's pointers and cell map
    done = min(0, steps);  // a caller's draws may ask for no step
    return run_steps<M, K>(sp, gl, s, c, k, steps, done, save, threads);
}

// Controls as stored in the row: Dubins stores (yawRate, pitchRate, a) (statePropagatorSpatialHash.cu:223-225).
template <int M>
__device__ __forceinline__ void row_controls(const float* c, float* out)
{
    if constexpr(M == KPAX_MODEL_DUBINS_AIRPLANE) {
        out[0] = c[1], out[1] = c[2], out[2] = c[0], out[3] = 0.0f;
    } else {
#pragma unroll
        for(int i = 0; i < 4; ++i) out[i] = c[i];
    }
}

}  // namespace kpax
