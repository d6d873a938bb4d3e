// Per-robot path smoothing by gradient descent on the clearance cost, judged
// by the robot's own collision checker.  Included from robot_kernels.cuh.
#pragma once

#include "clearance_device.cuh"
#include "clearance_eval.cuh"
#include "near_check.cuh"
#include "planner_device.cuh"

namespace prrtc {

// Deterministic block sum (fixed blockDim, fixed order); every thread gets it.
__device__ __forceinline__ double block_sum(double v, double *s_red)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += s_red[w];
    return t;
}

// One block per path.  First `shortcut_rounds` shortcut attempts: a span
// (i, j) of the path, chosen by a hash of (path, round), is replaced by evenly
// spaced points on the straight segment q_i -> q_j when every one of those
// sub-edges is free at granularity / 4 points (a quick filter; the judge below
// checks at full resolution).  Then the path stays in shared memory for all
// `steps` iterations of
//     q_w <- clamp(q_w - step * (cost_weight * dC/dq(q_w) + smooth_weight * (2 q_w - q_{w-1} - q_{w+1})))
// over the interior waypoints (the end points stay where they are).  The
// result is then checked edge by edge with the robot's checker at
// `granularity` points per edge (a + k ((b - a) / g), k = 1..g, as the
// planner interpolates); it is written back only if every point is free, so a
// rejected path is left exactly as it came in.
// Four lanes evaluate a waypoint (clearance_eval.cuh), all threads check points.
template <class Gen>
__host__ __device__ constexpr size_t smooth_eval_offset(int records, int waypoints)
{
    return (records * sizeof(float4) + 2 * sizeof(float) * waypoints * Gen::kDof + 15) & ~(size_t)15;
}

// The check of a point in an environment without a grid, as a called function
// (EveryCheckCtx, device_common.cuh).
template <class Gen>
__device__ __noinline__ bool every_test(const NearCfg<Gen::kDof> c, const EnvView env, volatile int *stop)
{
    EveryCheckCtx ctx{};
    ctx.env = env;
    ctx.stop_flag = stop;
    return Gen::fkcc(c.q, ctx);
}

// One point's check, compiled into both places that ask (as a function of its
// own it is built with 128 registers instead of up to 255: 32 Baxter paths took
// 3.5 instead of 2.9 ms).
template <class Gen>
__device__ __forceinline__ bool point_free(const NearCfg<Gen::kDof> &c, CheckCtx &ctx)
{
    ctx.work = 0;
    return ctx.env.grid ? Gen::fkcc(c.q, ctx) : every_test<Gen>(c, ctx.env, ctx.stop_flag);
}

template <class Gen>
__global__ void __launch_bounds__(256) k_smooth_paths(const ClrLaunch P)
{
    constexpr int D = Gen::kDof;
    extern __shared__ float4 s_dyn[];
    __shared__ int s_bad;
    __shared__ double s_red[8];
    __shared__ unsigned long long s_bar;
    __shared__ EnvGrid s_grid;
    constexpr int NJ = Gen::kFrames - 1, SLOTS = (Gen::kFrames + 2) / 4;
    const int path = blockIdx.x;
    const int W = P.waypoints;
    const ClrEnv pe = P.envs[path];
    const int R = pe.n.records();
    float *s_q = reinterpret_cast<float *>(s_dyn + R);
    float *s_g = s_q + W * D;
    auto *s_eval = reinterpret_cast<clr::EvalScratch<NJ> *>(reinterpret_cast<char *>(s_dyn) + smooth_eval_offset<Gen>(R, W));
    float *gq = P.q + (size_t)path * W * D;
    for (int i = threadIdx.x; i < W * D; i += blockDim.x) s_q[i] = gq[i];
    const EnvGrid *gr = stage_grid(&s_grid, pe.grid, s_dyn, threadIdx.x, blockDim.x);
    stage_env_bulk(s_dyn, pe.rec, R, &s_bar);   // synchronises the block
    const ClrEnv e{s_dyn, pe.n, gr};
    const ClrSmooth s = P.s;
    CheckCtx ctx{EnvView{e.rec, e.n, gr}, 0.0f, &s_bad};
    const int group = threadIdx.x >> 2, groups = blockDim.x >> 2, l = threadIdx.x & 3;
    // every waypoint's cost (returned summed over this thread's) and gradient
    auto evaluate = [&](auto &&store) {
        double cost = 0.0;
        for (int w0 = 0; w0 < W; w0 += groups) {
            const int w = w0 + group;
            double gr[SLOTS];
            const double c = clr::eval<Gen>(s_eval[group], P.M, e, s_q + (w < W ? w : 0) * D, w < W, s.margin, gr);
            if (w < W) {
                if (l == 0) cost += c;
                store(w, gr);
            }
        }
        return cost;
    };
    if (P.cost_before) {   // the cost of the path as given
        const double total = block_sum(evaluate([](int, const double(&)[SLOTS]) {}), s_red);
        if (threadIdx.x == 0) P.cost_before[path] = (float)total;
    }
    const int gs = max(1, s.granularity / 4);
    for (int r = 0; r < s.shortcut_rounds && W > 2; r++) {
        const unsigned h = hash32((unsigned)path * 0x9E3779B1u + (unsigned)r * 0x85EBCA77u + 0x27D4EB2Fu);
        const int span = 2 + (int)(h % (unsigned)min(W - 2, 31));   // 2 .. min(W - 1, 32) segments
        const int i0 = (int)((h >> 8) % (unsigned)(W - span));
        const float *qa = s_q + i0 * D, *qb = s_q + (i0 + span) * D;
        if (threadIdx.x == 0) s_bad = 0;
        __syncthreads();
        // sub-edge m runs from p_m to p_{m+1}, p_m = qa + (m / span) (qb - qa)
        for (int idx = threadIdx.x; idx < span * gs; idx += blockDim.x) {
            if (*(volatile int *)&s_bad) break;
            const int m = idx / gs, k = idx - m * gs + 1;
            NearCfg<D> cfg;
#pragma unroll
            for (int d = 0; d < D; d++) {
                const float delta = qb[d] - qa[d];
                const float a = qa[d] + ((float)m / (float)span) * delta, b = qa[d] + ((float)(m + 1) / (float)span) * delta;
                cfg.q[d] = __fadd_rn(a, __fmul_rn((float)k, __fdiv_rn(__fsub_rn(b, a), (float)gs)));
            }
            if (!point_free<Gen>(cfg, ctx)) s_bad = 1;
        }
        __syncthreads();
        if (s_bad == 0)
            for (int i = threadIdx.x; i < (span - 1) * D; i += blockDim.x) {
                const int m = i / D + 1, d = i - (m - 1) * D;
                s_q[(i0 + m) * D + d] = qa[d] + ((float)m / (float)span) * (qb[d] - qa[d]);
            }
        __syncthreads();
    }
    for (int it = 0; it <= s.steps; it++) {
        const double cost = evaluate([&](int w, const double(&gr)[SLOTS]) {
            if (w == 0 || w == W - 1) return;
#pragma unroll
            for (int t = 0; t < SLOTS; t++)
                if (l + 4 * t < NJ) {
                    const int d = P.M.joints[l + 4 * t].q;
                    s_g[w * D + d] = (float)((double)s.cost_weight * gr[t]) +
                                     s.smooth_weight * (2.0f * s_q[w * D + d] - s_q[(w - 1) * D + d] - s_q[(w + 1) * D + d]);
                }
        });
        if (it == s.steps) {
            const double total = block_sum(cost, s_red);
            if (threadIdx.x == 0 && P.cost_after) P.cost_after[path] = (float)total;
        }
        __syncthreads();
        if (it == s.steps) break;
        for (int i = threadIdx.x + D; i < (W - 1) * D; i += blockDim.x) {
            const int d = i % D;
            s_q[i] = fminf(fmaxf(s_q[i] - s.step * s_g[i], P.lo[d]), P.hi[d]);
        }
        __syncthreads();
    }
    // the judge: every edge at the planner's interpolation points
    if (threadIdx.x == 0) s_bad = 0;
    __syncthreads();
    const float fg = (float)s.granularity;
    const int total = (W - 1) * s.granularity;
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        if (*(volatile int *)&s_bad) break;
        const int ed = idx / s.granularity, k = idx - ed * s.granularity + 1;
        const float *a = s_q + ed * D, *b = a + D;
        NearCfg<D> cfg;
#pragma unroll
        for (int d = 0; d < D; d++) cfg.q[d] = __fadd_rn(a[d], __fmul_rn((float)k, __fdiv_rn(__fsub_rn(b[d], a[d]), fg)));
        if (!point_free<Gen>(cfg, ctx)) s_bad = 1;
    }
    __syncthreads();
    const bool ok = s_bad == 0;
    if (ok)
        for (int i = threadIdx.x; i < W * D; i += blockDim.x) gq[i] = s_q[i];
    if (threadIdx.x == 0) P.accepted[path] = ok ? 1 : 0;
}

}  // namespace prrtc
