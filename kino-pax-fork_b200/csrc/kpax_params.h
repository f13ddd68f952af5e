// kpax_params.h — launch parameters derived once on the host from a kpax_config.
//
// Everything a kernel needs about the dynamics, the checks and the region grid is here,
// precomputed so that device code does only float arithmetic.  The reference evaluates a
// few tests in double because its macros are double literals (C_MIN/C_MAX = +-M_PI,
// DUBINS_AIRPLANE_MIN/MAX_PITCH = +-M_PI/3, config.h:231-232, 280-281); those tests are
// replaced by float thresholds that give the identical verdict for every float input
// (see kpax_config.cpp).
#pragma once
#include <stdint.h>

#include "kpax.h"

namespace kpax {

constexpr int kMaxThr = 15;  // attitude split lengths are limited to 16

struct KParams {
    int model, sd, cd, S;   // state dim, control dim, sample dim (S = sd + cd + 1)
    float h, hh, h6;        // STEP_SIZE, 0.5f*STEP_SIZE, STEP_SIZE/6.0f
    int nsteps, fixed_steps;
    float ws_lo, ws_hi;     // workspace check bounds of the model
    float vmin, vmax;
    float pitch_lo, pitch_hi;  // p < pitch_lo  <=>  (double)p < MIN_PITCH, etc.
    float clo[4], crng[4];     // control ranges in draw order: c = clo + u * crng
    // region grid (Graph.cu:99-205)
    int W1, C1, V1, W2, C2, V2, cdim, vdim, w_only;
    float wmin, wspan, vmin_r, vspan, w1size, v1size;
    float cthr1[kMaxThr];   // attitude R1 index = #{k : c >= cthr1[k]}
    float cthr2[kMaxThr];   // attitude R2 index = #{k : C2*(c - m) >= cthr2[k]}
    int r1_mulW, r1_mulA, r2_mulW, r2_mulA, P, num_r1;
    int compat;             // R1 min corners decoded as initializeRegions_kernel does (w fastest)
    float cmin_tab[kMaxThr + 1];  // (float)(C_MIN + i * C_R1_SIZE), evaluated in double
    uint32_t r2_words;      // ceil(num_r1 * P / 32)
    // spatial hash (spatialHash.cuh:9-13)
    float cell;
    int gdim;
    // planner
    float goal_thresh, eps, vol;
    uint32_t cap, budget, per_entry, root_repeat, sparse_repeat;
    int sparse_thr;
    uint32_t seed_lo, seed_hi;
    // goal-progress pruning (PruneKPAX)
    int prune;
    float prune_goal_bias, prune_expl_bias, prune_scale;
};

// Steps per collision query where queries are grouped: 5 divides the presets' 10, 20 and 25 steps, and the
// kept states (120 KB of shared memory at 512 quadrotor children per SM) leave the grid over 100 KB of L1.
constexpr int kGroup = 5;

// Whether steps share collision queries in groups (run_steps).  A group's hull is walked over all its cells,
// and the steps behind a colliding one are wasted, so groups pay while they stay about as small as a grid
// cell: when kGroup steps at the speed bound go at most a cell far, or 5/4 of one where speeds spread around
// zero (the Dubins airplane flies near its bound).  Longer steps get a query each.
// B200, groups / query per step: the presets (0.5 to 3 m in 5 m cells) gain, see run_steps; the quadrotor's
// 3 m in 2.5 m cells, 300 iterations of 2^16 children, 22.3 / 23.4 ms; quad-ref (15 m in 5 m cells), 100
// iterations 8.3 / 6.2 ms, with steps three times as long 7.5 / 2.3 ms.  Segments, 5 m cells, 2000 obstacles:
// 30011 of the quadrotor, 6 m a group 58 / 70 us, 60 m 243 / 31; 2^19 of Dubins, 5 m 120 / 116, 6 m 145 / 119,
// 10 m 139 / 106; 2^19 of the double integrator, 6 m 91 / 86 (30011: 27 / 29), 12.5 m 156 / 92.
inline bool grouped(const KParams& p)
{
    const float v = p.vmax > -p.vmin ? p.vmax : -p.vmin;
    const float reach = p.model == KPAX_MODEL_DUBINS_AIRPLANE ? 1.0f : 1.25f;
    return (float)kGroup * p.h * v <= reach * p.cell;
}

// Derive parameters; returns KPAX_OK or KPAX_EINVAL with a message in kpax_last_error().
kpax_status derive_params(const kpax_config& cfg, KParams* out);
void set_error(const char* fmt, ...);

}  // namespace kpax
