// dem_rollout.cu — per-rollout costs of a batch of planner rollouts.
//
// One CTA per rollout q, after dem_rollout_segment has stepped every rollout's
// ship and ice window:
//   * the reference planner's four unweighted cost components
//     (medea_ice_ship/jax_mbd_planner.py:_make_raw_components_fn, :569-665) of
//     the pose path eta0, eta_1 .. eta_H, in float32 as the planner runs them:
//     costmap integral (bilinear query :128-168 at the hull centre and four
//     box corners, maximum, trapezoid rule over segment lengths), path length,
//     exponentially discounted goal distance, and jerk of the normalised
//     controls; the optional goal-line truncation (:621-637) masks waypoints
//     after the first crossing;
//   * the kinetic energy the rollout transferred to its ice window,
//     sum_e 0.5 m_e (|v_e(H)|^2 - |v_e(0)|^2) over the window's elements, in
//     double with a fixed summation order (run to run identical).
// What bounds it: for a planner's thousands of short rollouts, the five bilinear
// queries of every waypoint, so the terms run one thread per waypoint of a group
// of rollouts (neighbours in memory, so that a step's poses and controls are read
// as a row); the products of the sums over waypoints are terms too, and the sums
// themselves run in waypoint order, a warp per rollout with a sum per lane, so
// that a chain holds nothing but additions.  (One rollout a CTA and its four sums,
// with their square roots and divisions, on one thread: 76 us for 8192 rollouts of
// 64 steps, 27 now.)
// The per-waypoint values can be written out on the way, which saves a second
// pass over the poses and queries (14 us for the same rollouts).
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "dem_b200.h"

namespace {

constexpr int kRcThreads = 128;
constexpr int kRcGroupThreads = 256;
constexpr int kRcMaxHorizon = 2000;
constexpr int kRcArrays = 8;  // floats of shared memory per waypoint of a rollout (80 KB at the longest horizon)

struct RcArgs {
    int Q, H, rows, cols, use_hull, has_truncate, has_jerk, has_ke;
    float xo, yo, res, oob, hl, hw, gx, gy, trunc_y, tau;
    float ac[3], as[3];
    int group_log2;  // rollouts of a CTA
};

// Words of a rollout's arrays: 4 beyond a multiple of 32, so that the lanes of a
// warp, eight rollouts by four waypoints, fall on different banks.
__host__ __device__ constexpr int rc_stride(int W) { return (kRcArrays * W + 31) / 32 * 32 + 4; }

// jnp.max semantics: NaN wins
__device__ __forceinline__ float max_nan(float a, float b) { return (a > b || a != a) ? a : b; }

// _make_query (jax_mbd_planner.py:128-168) in float32
__device__ __forceinline__ float query(const RcArgs& c, const float* __restrict__ g, float x, float y) {
    const float cf = (x - c.xo) / c.res - 0.5f;
    const float rf = (y - c.yo) / c.res - 0.5f;
    const int r0 = (int)floorf(rf), c0 = (int)floorf(cf);
    const float fr = rf - (float)r0, fc = cf - (float)c0;
    const int r0c = min(max(r0, 0), c.rows - 1), r1c = min(max(r0 + 1, 0), c.rows - 1);
    const int c0c = min(max(c0, 0), c.cols - 1), c1c = min(max(c0 + 1, 0), c.cols - 1);
    const float oob = (c0 < 0 || c0 + 1 >= c.cols) ? c.oob : 0.0f;
    const float g00 = __ldg(g + (size_t)r0c * c.cols + c0c), g01 = __ldg(g + (size_t)r0c * c.cols + c1c);
    const float g10 = __ldg(g + (size_t)r1c * c.cols + c0c), g11 = __ldg(g + (size_t)r1c * c.cols + c1c);
    const float val = g00 * (1.0f - fr) * (1.0f - fc) + g01 * (1.0f - fr) * fc + g10 * fr * (1.0f - fc) + g11 * fr * fc;
    return val + oob;
}

// a waypoint's cost: the query at the hull centre and its four box corners,
// maximum (NaN wins), or at the centre alone without a hull
__device__ __forceinline__ float waypoint_cost(const RcArgs& c, const float* __restrict__ grid, float x, float y,
                                               float psi) {
    if (!c.use_hull) return query(c, grid, x, y);
    const float cs = cosf(psi), sn = sinf(psi);
    const float dxb[5] = {0.0f, c.hl, c.hl, -c.hl, -c.hl};
    const float dyb[5] = {0.0f, c.hw, -c.hw, c.hw, -c.hw};
    float w = 0.0f;
    for (int k = 0; k < 5; ++k) {
        const float wx = x + cs * dxb[k] - sn * dyb[k];
        const float wy = y + sn * dxb[k] + cs * dyb[k];
        const float v = query(c, grid, wx, wy);
        w = (k == 0) ? v : max_nan(w, v);
    }
    return w;
}

template <typename T>
__global__ void __launch_bounds__(kRcGroupThreads) rollout_cost_kernel(
    const RcArgs c, const int* __restrict__ sys_start, const T* __restrict__ eta0, const T* __restrict__ eta_hist,
    const T* __restrict__ u, const float* __restrict__ grid, const T* __restrict__ masses, const T* __restrict__ v0,
    const T* __restrict__ v1, double* __restrict__ out, float* __restrict__ wcost) {
    extern __shared__ float sm[];
    const int H = c.H, W = H + 1, stride = rc_stride(W), R = 1 << c.group_log2, q0 = blockIdx.x * R;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* dsc = sm + R * stride;  // (W) undiscounted weights exp(-t / tau)
    // a rollout's sums in the order of the lanes that run them, then the waypoints
    enum { kCost, kLength, kGoal, kJerk, kWp, kX, kY, kMask };
    auto arr = [&](int r, int k) { return sm + r * stride + k * W; };
    __shared__ double s_ke[kRcThreads];
    __shared__ float s_dsum;
    for (int t = threadIdx.x; t < W; t += blockDim.x) dsc[t] = expf(-(float)t / c.tau);
    for (int i = threadIdx.x; i < W * R; i += blockDim.x) {
        const int t = i >> c.group_log2, r = i & (R - 1), q = q0 + r;
        if (q >= c.Q) continue;
        const T* p = (t == 0) ? eta0 + 3 * (size_t)q : eta_hist + 3 * ((size_t)(t - 1) * c.Q + q);
        const float x = (float)p[0], y = (float)p[1], psi = (float)p[2];
        float j = 0.0f;
        if (c.has_jerk && t < H) {
            for (int k = 0; k < 3; ++k) {
                const float a = ((float)u[3 * ((size_t)t * c.Q + q) + k] - c.ac[k]) / c.as[k];
                const float b = ((float)u[3 * ((size_t)(t + 1 < H ? t + 1 : t) * c.Q + q) + k] - c.ac[k]) / c.as[k];
                const float du = b - a;
                j = j + du * du;
            }
        }
        const float w = waypoint_cost(c, grid, x, y, psi);
        const float gdx = x - c.gx, gdy = y - c.gy;
        arr(r, kWp)[t] = w;
        arr(r, kX)[t] = x;
        arr(r, kY)[t] = y;
        arr(r, kGoal)[t] = sqrtf(gdx * gdx + gdy * gdy + 1e-4f);
        arr(r, kJerk)[t] = j;
    }
    // kinetic energy transferred to the window (double, fixed order; one rollout a CTA)
    if (c.has_ke) {
        double ke = 0.0;
        const int e0 = sys_start[q0], e1 = sys_start[q0 + 1];
        for (int e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
            const double m = (double)masses[e];
            const double a0 = (double)v0[2 * (size_t)e], b0 = (double)v0[2 * (size_t)e + 1];
            const double a1 = (double)v1[2 * (size_t)e], b1 = (double)v1[2 * (size_t)e + 1];
            ke += 0.5 * m * ((a1 * a1 + b1 * b1) - (a0 * a0 + b0 * b0));
        }
        s_ke[threadIdx.x] = ke;
    }
    __syncthreads();
    if (warp == 0 && lane == 0) {
        float dsum = 0.0f;
#pragma unroll 8
        for (int t = 0; t < W; ++t) dsum = dsum + dsc[t];
        s_dsum = dsum;
    }
    if (c.has_truncate && lane == 0) {
        // goal-line truncation: waypoint t counts while max(y_0 .. y_{t-1}) < truncate_y
        for (int r = warp; r < R && q0 + r < c.Q; r += blockDim.x >> 5) {
            const float* ty = arr(r, kY);
            float* mk = arr(r, kMask);
            float cum = -1e9f;
            mk[0] = (cum < c.trunc_y) ? 1.0f : 0.0f;
            for (int t = 0; t < H; ++t) {
                cum = (t == 0) ? ty[0] : max_nan(cum, ty[t]);
                mk[t + 1] = (cum < c.trunc_y) ? 1.0f : 0.0f;
            }
        }
    }
    if (c.has_ke)
        for (int s = blockDim.x / 2; s > 0; s >>= 1) {
            if (threadIdx.x < s) s_ke[threadIdx.x] += s_ke[threadIdx.x + s];
            __syncthreads();
        }
    __syncthreads();
    const float dsum = s_dsum;
    for (int i = threadIdx.x; i < W * R; i += blockDim.x) {
        const int t = i >> c.group_log2, r = i & (R - 1);
        if (q0 + r >= c.Q) continue;
        arr(r, kGoal)[t] = (dsc[t] / dsum) * arr(r, kGoal)[t];
        if (t < H) {
            const float *tx = arr(r, kX) + t, *ty = arr(r, kY) + t, *wp = arr(r, kWp) + t, *mk = arr(r, kMask) + t;
            const float m0 = c.has_truncate ? mk[0] : 1.0f, m1 = c.has_truncate ? mk[1] : 1.0f;
            const float dx = tx[1] - tx[0], dy = ty[1] - ty[0];
            const float seg = sqrtf(dx * dx + dy * dy + 1e-8f);
            arr(r, kLength)[t] = seg * m0;
            arr(r, kCost)[t] = 0.5f * (wp[0] * m0 + wp[1] * m1) * seg;
        }
    }
    __syncthreads();
    for (int r = warp; r < R && q0 + r < c.Q; r += blockDim.x >> 5) {
        const int q = q0 + r;
        if (wcost)
            for (int t = lane; t < H; t += 32) wcost[(size_t)q * H + t] = arr(r, kWp)[t + 1];
        if (lane < 4) {
            const float* v = arr(r, lane);
            const int n = lane == kGoal ? W : lane == kJerk ? H - 1 : H;
            float sum = 0.0f;
#pragma unroll 8
            for (int t = 0; t < n; ++t) sum = sum + v[t];
            if (lane == kJerk) sum = c.has_jerk ? sum / (float)(3 * (H - 1)) : 0.0f;
            out[5 * (size_t)q + lane] = (double)sum;
        } else if (lane == 4) {
            out[5 * (size_t)q + 4] = c.has_ke ? s_ke[0] : 0.0;
        }
    }
}

// one thread per (step, rollout): out[q, t] = the cost of the pose after step t
template <typename T>
__global__ void __launch_bounds__(kRcThreads) waypoint_cost_kernel(RcArgs c, const T* __restrict__ eta_hist,
                                                                   const float* __restrict__ grid,
                                                                   float* __restrict__ out) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= (long long)c.Q * c.H) return;
    const int t = (int)(i / c.Q), q = (int)(i % c.Q);
    const T* p = eta_hist + 3 * (size_t)i;
    out[(size_t)q * c.H + t] = waypoint_cost(c, grid, (float)p[0], (float)p[1], (float)p[2]);
}

// the costmap geometry of the cost arguments, as the planner's float32 query sees it
bool grid_args(const DemRolloutCostParams* p, RcArgs& c) {
    if (p->rows < 1 || p->cols < 1 || (long long)p->rows * p->cols >= (1LL << 31) || !(p->resolution > 0.0))
        return false;
    c.rows = p->rows;
    c.cols = p->cols;
    c.use_hull = (p->ship_length > 0.0 && p->ship_beam > 0.0) ? 1 : 0;
    // the planner's Python scalars meet float32 arrays: each is rounded to float
    c.xo = (float)p->x_origin;
    c.yo = (float)p->y_origin;
    c.res = (float)p->resolution;
    c.oob = (float)p->oob_penalty;
    c.hl = (float)(p->ship_length / 2.0);
    c.hw = (float)(p->ship_beam / 2.0);
    return true;
}

template <typename T>
int launch_costs(const RcArgs& c, const int32_t* sys_start, const void* eta0, const void* eta_hist,
                 const void* u, const float* grid, const void* masses, const void* v0, const void* v1, double* out,
                 float* wcost, cudaStream_t st) {
    // Eight rollouts a CTA once that leaves every SM several of them; fewer when the
    // arrays of eight would crowd the SM.  The energy's sum wants a CTA of its own.
    RcArgs g = c;
    const size_t words = rc_stride(c.H + 1);
    g.group_log2 = 0;
    if (!c.has_ke)
        while (g.group_log2 < 3 && c.Q >= (148 * 2) << (g.group_log2 + 1) && (words << (g.group_log2 + 1)) <= 8192)
            ++g.group_log2;
    const int R = 1 << g.group_log2, threads = R > 1 ? kRcGroupThreads : kRcThreads;
    const size_t smem = sizeof(float) * (words * R + c.H + 1);
    // The limit belongs to the kernel, not to the call: always the longest horizon's,
    // so that calls of other threads find room for theirs.
    constexpr int kMost = (int)sizeof(float) * (rc_stride(kRcMaxHorizon + 1) + kRcMaxHorizon + 1);
    if (smem > 46 * 1024 && cudaFuncSetAttribute(rollout_cost_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 kMost) != cudaSuccess)
        return DEM_ERR_CUDA;
    rollout_cost_kernel<T><<<(c.Q + R - 1) / R, threads, smem, st>>>(g, sys_start, (const T*)eta0, (const T*)eta_hist,
                                                                     (const T*)u, grid, (const T*)masses,
                                                                     (const T*)v0, (const T*)v1, out, wcost);
    return cudaGetLastError() == cudaSuccess ? DEM_OK : DEM_ERR_CUDA;
}

}  // namespace

extern "C" int dem_rollout_costs(int32_t dtype, int32_t n_systems, int32_t horizon, const int32_t* system_start,
                                 const void* eta0, const void* eta_hist, const void* controls, const float* grid,
                                 const DemRolloutCostParams* p, const void* masses, const void* vel0,
                                 const void* vel1, double* out, void* stream) {
    return dem_rollout_path_costs(dtype, n_systems, horizon, system_start, eta0, eta_hist, controls, grid, p, masses,
                                  vel0, vel1, out, nullptr, stream);
}

extern "C" int dem_rollout_path_costs(int32_t dtype, int32_t n_systems, int32_t horizon, const int32_t* system_start,
                                      const void* eta0, const void* eta_hist, const void* controls,
                                      const float* grid, const DemRolloutCostParams* p, const void* masses,
                                      const void* vel0, const void* vel1, double* out, float* waypoint_out,
                                      void* stream) {
    if (!p || !out || !eta0 || !eta_hist || !grid || (dtype != DEM_F32 && dtype != DEM_F64)) return DEM_ERR_INVALID;
    if (n_systems < 1 || horizon < 1 || horizon > kRcMaxHorizon) return DEM_ERR_INVALID;
    RcArgs c{};
    if (!grid_args(p, c)) return DEM_ERR_INVALID;
    const bool has_ke = masses || vel0 || vel1;
    if (has_ke && (!masses || !vel0 || !vel1 || !system_start)) return DEM_ERR_INVALID;
    if (controls)
        for (int k = 0; k < 3; ++k)
            if (!(p->action_scale[k] != 0.0) || !std::isfinite(p->action_scale[k])) return DEM_ERR_INVALID;
    c.Q = n_systems;
    c.H = horizon;
    c.has_truncate = p->has_truncate ? 1 : 0;
    c.has_jerk = controls ? 1 : 0;
    c.has_ke = has_ke ? 1 : 0;
    c.gx = (float)p->goal_x;
    c.gy = (float)p->goal_y;
    c.trunc_y = (float)p->truncate_y;
    c.tau = (float)((double)(horizon + 1) / 3.0);
    for (int k = 0; k < 3; ++k) {
        c.ac[k] = (float)p->action_center[k];
        c.as[k] = (float)p->action_scale[k];
    }
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == DEM_F32)
        return launch_costs<float>(c, system_start, eta0, eta_hist, controls, grid, masses, vel0, vel1, out,
                                   waypoint_out, st);
    return launch_costs<double>(c, system_start, eta0, eta_hist, controls, grid, masses, vel0, vel1, out,
                                waypoint_out, st);
}

extern "C" int dem_rollout_waypoint_costs(int32_t dtype, int32_t n_systems, int32_t horizon, const void* eta_hist,
                                          const float* grid, const DemRolloutCostParams* p, float* out,
                                          void* stream) {
    if (!p || !out || !eta_hist || !grid || (dtype != DEM_F32 && dtype != DEM_F64)) return DEM_ERR_INVALID;
    if (n_systems < 1 || horizon < 1 || horizon > kRcMaxHorizon) return DEM_ERR_INVALID;
    RcArgs c{};
    if (!grid_args(p, c)) return DEM_ERR_INVALID;
    c.Q = n_systems;
    c.H = horizon;
    const long long total = (long long)n_systems * horizon;
    const unsigned blocks = (unsigned)((total + kRcThreads - 1) / kRcThreads);
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == DEM_F32)
        waypoint_cost_kernel<float><<<blocks, kRcThreads, 0, st>>>(c, (const float*)eta_hist, grid, out);
    else
        waypoint_cost_kernel<double><<<blocks, kRcThreads, 0, st>>>(c, (const double*)eta_hist, grid, out);
    return cudaGetLastError() == cudaSuccess ? DEM_OK : DEM_ERR_CUDA;
}

// ════════════════════════════════════════════════════════════════════════════
// dem_rollout_ice_terms: per rollout, the hull impulse (sum over the steps of
// the frame's J_cumul_incr = |F_ice_on_ship| dt, jax_simulation.py:692-697)
// and the bonds its ship broke (intact at the start, broken at the end), one
// CTA per rollout with fixed-order sums.
// ════════════════════════════════════════════════════════════════════════════
namespace {

template <typename T>
__global__ void __launch_bounds__(kRcThreads) ice_terms_kernel(int Q, int H, const T* __restrict__ J_hist,
                                                               const int* __restrict__ bond_start,
                                                               const uint8_t* __restrict__ intact0,
                                                               const uint8_t* __restrict__ intact1,
                                                               double* __restrict__ out) {
    __shared__ double s_imp[kRcThreads];
    __shared__ long long s_brk[kRcThreads];
    const int q = blockIdx.x;
    double imp = 0.0;
    for (int t = threadIdx.x; t < H; t += blockDim.x) imp += (double)J_hist[(size_t)t * Q + q];
    long long brk = 0;
    if (bond_start) {
        for (int b = bond_start[q] + threadIdx.x; b < bond_start[q + 1]; b += blockDim.x)
            brk += (intact0[b] != 0 && intact1[b] == 0) ? 1 : 0;
    }
    s_imp[threadIdx.x] = imp;
    s_brk[threadIdx.x] = brk;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            s_imp[threadIdx.x] += s_imp[threadIdx.x + w];
            s_brk[threadIdx.x] += s_brk[threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[2 * q] = s_imp[0];
        out[2 * q + 1] = (double)s_brk[0];
    }
}

}  // namespace

extern "C" int dem_rollout_ice_terms(int32_t dtype, int32_t n_systems, int32_t horizon, const void* J_hist,
                                     const int32_t* bond_start, const uint8_t* intact0, const uint8_t* intact1,
                                     double* out, void* stream) {
    if ((dtype != DEM_F32 && dtype != DEM_F64) || n_systems < 1 || horizon < 1 || !J_hist || !out)
        return DEM_ERR_INVALID;
    if (bond_start && (!intact0 || !intact1)) return DEM_ERR_INVALID;
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == DEM_F32)
        ice_terms_kernel<float><<<n_systems, kRcThreads, 0, st>>>(n_systems, horizon, (const float*)J_hist, bond_start,
                                                                  intact0, intact1, out);
    else
        ice_terms_kernel<double><<<n_systems, kRcThreads, 0, st>>>(n_systems, horizon, (const double*)J_hist,
                                                                   bond_start, intact0, intact1, out);
    return cudaGetLastError() == cudaSuccess ? DEM_OK : DEM_ERR_CUDA;
}

// ════════════════════════════════════════════════════════════════════════════
// dem_rollout_sweep_features: what a candidate's rigid-ship path sweeps
// through the plan's ice window, one CTA per candidate.  No counterpart in the
// reference.  An element is hit at the first pose t (0..H) at which its
// centroid, in the frame of that pose, lies inside the hull box grown by the
// element's radius r: |x| < half_len + r and |y| < half_beam + r.  The hit's
// ship velocity is the path's step velocity (pose t - pose t-1) / dt (the
// first step's for t = 0), and v_n its component towards the element's
// centroid, clamped at 0.  Per candidate, in double with fixed-order sums (run
// to run identical):
//   [0] elements hit, [1] their mass, [2] sum 0.5 m |v|^2, [3] sum m v_n,
//   [4] sum m (H + 1 - t) / (H + 1) (early hits weigh more), [5] sum 0.5 m v_n^2,
//   [6] bonds with exactly one end hit, [7] bonds with both ends hit.
// The geometry runs in float32 (cos and sin of the heading rounded from
// double), unfused, as a NumPy float32 evaluation of the same expressions.
//
// What bounds it: the pose tests.  A ship moves little over the poses of a plan,
// so most elements of its window are never near the hull, and those that are
// meet it in few poses.  The whole path and each 32 of its poses have a box, in
// the frame of their first pose, that the hull never leaves; an element outside of
// it (a test per element, a lane each) meets none of them.  A warp then goes
// through the elements that are left, a pose per lane, so that 32 poses cost one
// test and the first hit is the lowest bit of the vote.  A CTA takes eight
// neighbouring candidates, a warp each: their poses are read as rows, and as an
// element's hits are a byte, a bond is looked up once for all of them.
// A candidate's sums have one order, whatever the population: those of the elements
// e, e + 256, ... first, 256 sums, and these in a binary tree, 128 apart first.  A
// warp that has a candidate alone goes through the eight 32s of elements of each 256
// one after another, in the order in which the tree joins their sums, and keeps
// those that wait for their partner in shared memory.
// (A thread per element, pose after pose, one candidate a CTA: 267 us for 8192
// candidates of 64 steps through 450 elements and 1500 bonds; the boxes and votes
// with one candidate a CTA: 85; now 60, 4 of them for the one order of the sums.)
// ════════════════════════════════════════════════════════════════════════════
namespace {

constexpr int kSwThreads = 256;
constexpr int kSwWarps = kSwThreads / 32;
constexpr int kSwFeatures = DEM_SWEEP_FEATURES;
constexpr int kSwSums = 5;  // features 1 to 5; the others are counts
constexpr int kSwMaxElements = DEM_SWEEP_MAX_ELEMENTS;
constexpr int kSwMaxHorizon = DEM_SWEEP_MAX_HORIZON;

struct SwArgs {
    int Q, H, n, nb;
    float hl, hw, inv_dt;
};

// Some poses in the frame of their first (x, y, c, s): the range of their
// positions and the largest |sin| of the heading's change.
struct SwBox {
    float x, y, c, s, lo_x, hi_x, lo_y, hi_y, turn;
};

// False only if the grown hull box (gl, gw) of none of the poses holds (ex, ey).
// In the box's frame the hull of a pose turned by phi reaches gl |cos phi| +
// gw |sin phi| along x and gl |sin phi| + gw |cos phi| along y.  The margin covers
// the rounding of both frames many times; NaN never rejects.
__device__ __forceinline__ bool sw_near(const SwBox& g, float ex, float ey, float gl, float gw) {
    const float dx = ex - g.x, dy = ey - g.y;
    const float lx = g.c * dx + g.s * dy, ly = g.c * dy - g.s * dx;
    const float rx = gl + g.turn * gw, ry = gw + g.turn * gl;
    const float eps = 1e-3f + 1e-5f * (fabsf(dx) + fabsf(dy) + rx + ry);
    return !(lx < g.lo_x - rx - eps || lx > g.hi_x + rx + eps || ly < g.lo_y - ry - eps || ly > g.hi_y + ry + eps);
}

// The box of poses t0 .. t1, by a warp.
__device__ __forceinline__ SwBox sw_box(const float4* pose, int t0, int t1) {
    const float4 o = pose[t0];
    float lo_x = INFINITY, hi_x = -INFINITY, lo_y = INFINITY, hi_y = -INFINITY, turn = 0.0f;
    bool fine = fabsf(o.z) <= 1.0f;
    for (int t = t0 + (threadIdx.x & 31); t <= t1; t += 32) {
        const float4 p = pose[t];
        const float dx = p.x - o.x, dy = p.y - o.y;
        const float lx = o.z * dx + o.w * dy, ly = o.z * dy - o.w * dx, s = fabsf(o.z * p.w - o.w * p.z);
        fine = fine && fabsf(dx) < 1e15f && fabsf(dy) < 1e15f && s <= 2.0f;
        lo_x = fminf(lo_x, lx);
        hi_x = fmaxf(hi_x, lx);
        lo_y = fminf(lo_y, ly);
        hi_y = fmaxf(hi_y, ly);
        turn = fmaxf(turn, s);
    }
    for (int d = 16; d > 0; d >>= 1) {
        lo_x = fminf(lo_x, __shfl_xor_sync(0xffffffffu, lo_x, d));
        hi_x = fmaxf(hi_x, __shfl_xor_sync(0xffffffffu, hi_x, d));
        lo_y = fminf(lo_y, __shfl_xor_sync(0xffffffffu, lo_y, d));
        hi_y = fmaxf(hi_y, __shfl_xor_sync(0xffffffffu, hi_y, d));
        turn = fmaxf(turn, __shfl_xor_sync(0xffffffffu, turn, d));
    }
    // a pose that is not finite, or far beyond any window, leaves the box unbounded
    if (!__all_sync(0xffffffffu, fine))
        return SwBox{0.0f, 0.0f, 1.0f, 0.0f, -INFINITY, INFINITY, -INFINITY, INFINITY, 1.0f};
    return SwBox{o.x, o.y, o.z, o.w, lo_x, hi_x, lo_y, hi_y, turn};
}

// Shared memory of a CTA with G candidates: poses (x, y, cos, sin), sums (the eight
// warps' of one candidate, or three that wait in each of eight warps), boxes, hits.
struct SwLayout {
    size_t sum, box, hit, bytes;
    __host__ __device__ SwLayout(int G, int H, int n) {
        sum = sizeof(float4) * (size_t)G * (H + 1);
        box = sum + sizeof(double) * kSwSums * 32 * (G == 1 ? kSwWarps : 3 * kSwWarps);
        hit = box + (sizeof(SwBox) * (size_t)G * ((H + 32) / 32 + 1) + 15) / 16 * 16;
        bytes = hit + ((size_t)n + 15) / 16 * 16;
    }
};

// One candidate a CTA, or eight, a warp each.
template <typename T, int G>
__global__ void __launch_bounds__(kSwThreads, 4) sweep_kernel(const SwArgs c, const T* __restrict__ eta0,
                                                              const T* __restrict__ hist, const T* __restrict__ pos,
                                                              const T* __restrict__ radii, const T* __restrict__ mass,
                                                              const int* __restrict__ bi, const int* __restrict__ bj,
                                                              float* __restrict__ out) {
    static_assert(G == 1 || G == kSwWarps, "a candidate's sums are a CTA's or a warp's");
    extern __shared__ __align__(16) unsigned char sw_smem[];
    const SwLayout at(G, c.H, c.n);
    float4* pose = reinterpret_cast<float4*>(sw_smem);
    SwBox* box = reinterpret_cast<SwBox*>(sw_smem + at.box);
    unsigned char* hit = sw_smem + at.hit;  // a bit per candidate
    double* sums = reinterpret_cast<double*>(sw_smem + at.sum);
    __shared__ int counts[G][3];  // elements hit, bonds with one end hit and with both
    const int H = c.H, W = H + 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q0 = blockIdx.x * G, groups = (H + 32) / 32;
    for (int i = threadIdx.x; i < W * G; i += kSwThreads) {
        const int t = i / G, r = i % G, q = min(q0 + r, c.Q - 1);
        const T* p = (t == 0) ? eta0 + 3 * (size_t)q : hist + ((size_t)(t - 1) * c.Q + q) * 3;
        double sn, cs;
        sincos((double)p[2], &sn, &cs);
        pose[r * W + t] = make_float4((float)p[0], (float)p[1], (float)cs, (float)sn);
    }
    for (int w = threadIdx.x; w < (c.n + 3) / 4; w += kSwThreads) reinterpret_cast<unsigned*>(hit)[w] = 0u;
    if (threadIdx.x < 3 * G) counts[threadIdx.x / 3][threadIdx.x % 3] = 0;
    __syncthreads();
    // boxes of each 32 poses, then of the path
    for (int i = warp; i < G * (groups + 1); i += kSwWarps) {
        const int r = i / (groups + 1), k = i % (groups + 1);
        const SwBox b = sw_box(pose + r * W, k < groups ? 32 * k : 0, k < groups ? min(32 * k + 31, H) : H);
        if (lane == 0) box[i] = b;
    }
    __syncthreads();
    const int r = G == 1 ? 0 : warp;
    const float4* path = pose + r * W;
    const SwBox* boxes = box + r * (groups + 1);
    // the 32 elements of each 256 that come i-th: the warp's own, or 0, 4, 2, 6, 1, 5, 3, 7
    auto part = [&](int i) { return 32 * (G == 1 ? warp : (int)(__brev((unsigned)i) >> 29)); };
    auto load = [&](int e, float& x, float& y, float& rad) {
        x = y = rad = 0.0f;
        if (e < c.n) {
            x = (float)pos[2 * (size_t)e];
            y = (float)pos[2 * (size_t)e + 1];
            rad = (float)radii[e];
        }
    };
    int met = 0;  // elements hit
    double acc[kSwSums];
    double* wait = sums + (G == 1 ? 0 : warp * 3 * kSwSums * 32);
    float nx, ny, nr;
    load(part(0) + lane, nx, ny, nr);
    for (int i = 0; i < G; ++i) {
        for (int k = 0; k < kSwSums; ++k) acc[k] = 0.0;
        for (int e0 = part(i); e0 < c.n; e0 += kSwThreads) {
            const int e = e0 + lane;
            const float ex = nx, ey = ny, gl = c.hl + nr, gw = c.hw + nr;
            int ahead = e0 + kSwThreads;  // the warp's next elements
            for (int j = i + 1; j < G && ahead >= c.n; ++j) ahead = part(j);
            load(ahead + lane, nx, ny, nr);
            const bool reach = e < c.n && sw_near(boxes[groups], ex, ey, gl, gw);
            if (!__any_sync(0xffffffffu, reach)) continue;
            int th = -1;  // the lane's element: the pose that hits it first
            for (int k = 0; k < groups; ++k) {
                const bool near = reach && th < 0 && sw_near(boxes[k], ex, ey, gl, gw);
                unsigned todo = __ballot_sync(0xffffffffu, near);
                const int t = 32 * k + lane;
                const float4 p = path[min(t, H)];
                while (todo) {
                    const int l = __ffs(todo) - 1;
                    todo &= todo - 1;
                    // every lane takes part in the four shuffles
                    const float lx = __shfl_sync(0xffffffffu, ex, l), ly = __shfl_sync(0xffffffffu, ey, l);
                    const float ll = __shfl_sync(0xffffffffu, gl, l), lw = __shfl_sync(0xffffffffu, gw, l);
                    const float dx = lx - p.x, dy = ly - p.y;
                    const float bx = p.z * dx + p.w * dy;
                    const float by = p.z * dy - p.w * dx;
                    const bool in = fabsf(bx) < ll && fabsf(by) < lw && t <= H;
                    const unsigned v = __ballot_sync(0xffffffffu, in);
                    if (v && lane == l) th = 32 * k + __ffs(v) - 1;
                }
            }
            met += __popc(__ballot_sync(0xffffffffu, th >= 0));
            if (th >= 0) {
                const float4 p = path[th];
                // the first step's velocity at the start pose
                const float4 pa = path[max(th, 1)], pb = path[max(th, 1) - 1];
                const float dx = ex - p.x, dy = ey - p.y;
                const double m = (double)mass[e];
                const double vx = (double)((pa.x - pb.x) * c.inv_dt), vy = (double)((pa.y - pb.y) * c.inv_dt);
                const double dd = sqrt((double)dx * (double)dx + (double)dy * (double)dy);
                const double vn = fmax(0.0, (vx * (double)dx + vy * (double)dy) / fmax(dd, 1e-6));
                acc[0] += m;
                acc[1] += 0.5 * m * (vx * vx + vy * vy);
                acc[2] += m * vn;
                acc[3] += m * (double)(H + 1 - th) / (double)(H + 1);
                acc[4] += 0.5 * m * vn * vn;
                atomicOr(reinterpret_cast<unsigned*>(hit) + (e >> 2), (1u << r) << (8 * (e & 3)));
            }
        }
        if (G > 1) {
            // join the sums that wait for this one, as a binary counter carries
            int b = 0;
            for (; (i >> b) & 1; ++b)
                for (int k = 0; k < kSwSums; ++k) acc[k] = wait[(b * kSwSums + k) * 32 + lane] + acc[k];
            if (b < 3)
                for (int k = 0; k < kSwSums; ++k) wait[(b * kSwSums + k) * 32 + lane] = acc[k];
        }
    }
    auto lanes = [&](double v) {
        for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
        return v;
    };
    if (lane == 0) atomicAdd(&counts[r][0], met);
    if (G > 1) {
        for (int k = 0; k < kSwSums; ++k) {
            const double v = lanes(acc[k]);
            if (lane == 0 && q0 + r < c.Q) out[(size_t)(q0 + r) * kSwFeatures + 1 + k] = (float)v;
        }
    } else {
        for (int k = 0; k < kSwSums; ++k) sums[(warp * kSwSums + k) * 32 + lane] = acc[k];
    }
    __syncthreads();
    if (G == 1 && warp < kSwSums) {
        auto of = [&](int w) { return sums[(w * kSwSums + warp) * 32 + lane]; };
        const double v = lanes(((of(0) + of(4)) + (of(2) + of(6))) + ((of(1) + of(5)) + (of(3) + of(7))));
        if (lane == 0) out[(size_t)q0 * kSwFeatures + 1 + warp] = (float)v;
    }
    constexpr int kAhead = 4;  // bonds whose ends are read before the first is looked up
    for (int b0 = threadIdx.x; b0 < c.nb; b0 += kAhead * kSwThreads) {
        int i[kAhead], j[kAhead];
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            const int b = b0 + k * kSwThreads;
            i[k] = b < c.nb ? bi[b] : -1;
            j[k] = b < c.nb ? bj[b] : -1;
        }
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            if (i[k] < 0 || i[k] >= c.n || j[k] < 0 || j[k] >= c.n) continue;
            const unsigned hi = hit[i[k]], hj = hit[j[k]];
            for (unsigned x = hi | hj; x; x &= x - 1) {  // few: the candidates that hit an end
                const int l = __ffs(x) - 1;
                atomicAdd(&counts[l][1 + (((hi & hj) >> l) & 1u)], 1);
            }
        }
    }
    __syncthreads();
    if (threadIdx.x < 3 * G) {
        const int l = threadIdx.x / 3, k = threadIdx.x % 3;
        if (q0 + l < c.Q) out[(size_t)(q0 + l) * kSwFeatures + (k == 0 ? 0 : 5 + k)] = (float)counts[l][k];
    }
}
static_assert(kSwFeatures == 8 && kSwThreads == 256, "the order of a candidate's sums");

template <typename T, int G>
int launch_sweep(const SwArgs& c, const void* eta0, const void* hist, const void* pos, const void* radii,
                 const void* mass, const int32_t* bi, const int32_t* bj, float* out, cudaStream_t st) {
    const size_t smem = SwLayout(G, c.H, c.n).bytes;
    // the kernel's limit is the largest call's, whatever other threads call
    const int most = (int)SwLayout(G, kSwMaxHorizon, kSwMaxElements).bytes;
    if (smem > 46 * 1024 && cudaFuncSetAttribute(sweep_kernel<T, G>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 most) != cudaSuccess)
        return DEM_ERR_CUDA;
    sweep_kernel<T, G><<<(c.Q + G - 1) / G, kSwThreads, smem, st>>>(c, (const T*)eta0, (const T*)hist, (const T*)pos,
                                                                    (const T*)radii, (const T*)mass, bi, bj, out);
    return cudaGetLastError() == cudaSuccess ? DEM_OK : DEM_ERR_CUDA;
}

// Eight candidates a CTA from the population on whose CTAs fill the SMs: 2368
// candidates in 29 us either way, 4736 in 37 against 52 with one a CTA, 8192 in 60
// against 85; below, 1776 in 27 against 24.5, 1184 in 27 against 18 and 64 in 22
// against 11.
constexpr int kSwGroupFrom = 148 * 16;

}  // namespace

extern "C" int dem_rollout_sweep_features(int32_t dtype, int32_t n_rollouts, int32_t horizon, const void* eta0,
                                          const void* eta_hist, int32_t n, const void* positions, const void* radii,
                                          const void* masses, int32_t n_bonds, const int32_t* bond_i,
                                          const int32_t* bond_j, double half_len, double half_beam, double dt,
                                          float* out, void* stream) {
    if ((dtype != DEM_F32 && dtype != DEM_F64) || n_rollouts < 1 || horizon < 1 || horizon > kSwMaxHorizon)
        return DEM_ERR_INVALID;
    if (n < 0 || n > kSwMaxElements || n_bonds < 0 || !(dt > 0.0) || !(half_len >= 0.0) || !(half_beam >= 0.0))
        return DEM_ERR_INVALID;
    if (!eta0 || !eta_hist || !out || (n > 0 && (!positions || !radii || !masses)) ||
        (n_bonds > 0 && (!bond_i || !bond_j)))
        return DEM_ERR_INVALID;
    SwArgs c{};
    c.Q = n_rollouts;
    c.H = horizon;
    c.n = n;
    c.nb = n_bonds;
    c.hl = (float)half_len;
    c.hw = (float)half_beam;
    c.inv_dt = (float)(1.0 / dt);
    cudaStream_t st = (cudaStream_t)stream;
    const bool group = n_rollouts >= kSwGroupFrom;
    if (dtype == DEM_F32)
        return (group ? launch_sweep<float, 8> : launch_sweep<float, 1>)(c, eta0, eta_hist, positions, radii, masses,
                                                                         bond_i, bond_j, out, st);
    return (group ? launch_sweep<double, 8> : launch_sweep<double, 1>)(c, eta0, eta_hist, positions, radii, masses,
                                                                       bond_i, bond_j, out, st);
}
