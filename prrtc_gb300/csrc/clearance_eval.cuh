// The clearance cost and its adjoint for many configurations at once
// (clearance_device.cuh defines both and holds the one-thread form, which
// this one follows term by term).  Four lanes of a warp share a configuration.
//
// What bounds it: the FP64 pipe does two lanes per clock and SM, so a
// configuration's kinematics, sweep and conversions in FP64 (1700 warp
// instructions for 32 configurations, 16 clocks each) took longer than
// everything else.  Here
//  * the kinematics run in pairs of floats (Dd: 48 bits; T. J. Dekker, "A
//    floating-point technique for extending the available precision", 1971),
//    a frame's three rows on three lanes, sines and cosines by their Taylor
//    series after a reduction by multiples of pi / 2;
//  * leaf spheres and sphere pairs are screened by bounds first: balls around
//    a link's leaves and each leaf by the clearance grid, links' balls, then
//    one link's sphere against the ball around the other's, for pairs;
//  * the few terms that are left run in FP64 as before, and each term's force
//    is applied to the joints that carry it directly, four joints at a time
//    (no force tables, no sweep over joints without forces).
// 4096 Panda paths of 64 waypoints on shelf scenes (k_path_cost_grad): 1.83 ms
// with one thread per waypoint, 0.5 ms so; 1024 of them smoothed 44.6 -> 11.7 ms,
// 32 Baxter paths 61.1 -> 3.7 ms (rows of pairs against the whole other frame
// instead of parts of at most 6 spheres: 12.1 and 4.8 ms; parts of 4: 11.5 and 3.7).  Results differ from the one-thread form's by
// 2e-10 (relative, all outputs), the error against float64 is the same 2.5e-8
// (float32's own).
#pragma once

#include "clearance_device.cuh"

namespace prrtc {

namespace clr {

// ---- pairs of floats: value h + l, |l| <= ulp(h) / 2 ---------------------
struct Dd {
    float h, l;
};
__device__ __forceinline__ Dd dd(float h, float l = 0.0f) { return Dd{h, l}; }
__device__ __forceinline__ Dd quick_sum(float a, float b)   // |a| >= |b|
{
    const float s = __fadd_rn(a, b);
    return Dd{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ Dd two_sum(float a, float b)
{
    const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
    return Dd{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ Dd operator+(Dd x, Dd y)
{
    const Dd s = two_sum(x.h, y.h);
    return quick_sum(s.h, __fadd_rn(s.l, __fadd_rn(x.l, y.l)));
}
__device__ __forceinline__ Dd operator-(Dd x) { return Dd{-x.h, -x.l}; }
__device__ __forceinline__ Dd operator-(Dd x, Dd y) { return x + (-y); }
__device__ __forceinline__ Dd operator*(Dd x, Dd y)
{
    const float p = __fmul_rn(x.h, y.h);
    return quick_sum(p, __fmaf_rn(x.l, y.h, __fmaf_rn(x.h, y.l, __fmaf_rn(x.h, y.h, -p))));
}
__device__ __forceinline__ Dd operator*(Dd x, float f)
{
    const float p = __fmul_rn(x.h, f);
    return quick_sum(p, __fmaf_rn(x.l, f, __fmaf_rn(x.h, f, -p)));
}
__device__ __forceinline__ double to_double(Dd x) { return (double)x.h + (double)x.l; }

// Sine and cosine of |q| <= 100 to 2^-44: q = k pi / 2 + r with pi / 2 in three
// parts (the first two of 16 bits, so k times them is exact; Cody and Waite's
// reduction, see near_sincos), then the
// Taylor series of r, |r| <= pi / 4, up to r^15 / r^16, the coefficients down to
// 1 / 7! and 1 / 8! in pairs.
__device__ __forceinline__ Dd coef(double c) { return Dd{(float)c, (float)(c - (double)(float)c)}; }
__device__ __forceinline__ void sin_cos(float q, Dd *sn, Dd *cs)
{
    const float k = rintf(q * 0.636619772f);
    const float t = __fmaf_rn(-k, 0x1.921ep+0f, q), p2 = -k * 0x1.b544p-16f;   // both exact
    const Dd a = two_sum(t, p2);
    const Dd r = quick_sum(a.h, __fmaf_rn(-k, 0x1.0b4612p-34f, a.l));
    const Dd x = r * r;
    // sin r = r + r x (-1/3! + x (1/5! + x (-1/7! + x (1/9! - ...))))
    float f = __fmaf_rn(x.h, -1.0f / 1307674368000.0f, 1.0f / 6227020800.0f);
    f = __fmaf_rn(x.h, f, -1.0f / 39916800.0f);
    f = __fmaf_rn(x.h, f, 1.0f / 362880.0f);
    Dd s = x * f + coef(-1.0 / 5040.0);
    s = x * s + coef(1.0 / 120.0);
    s = x * s + coef(-1.0 / 6.0);
    s = r + r * (x * s);
    // cos r = 1 + x (-1/2! + x (1/4! + x (-1/6! + x (1/8! - ...))))
    f = __fmaf_rn(x.h, 1.0f / 20922789888000.0f, -1.0f / 87178291200.0f);
    f = __fmaf_rn(x.h, f, 1.0f / 479001600.0f);
    f = __fmaf_rn(x.h, f, -1.0f / 3628800.0f);
    Dd c = x * f + coef(1.0 / 40320.0);
    c = x * c + coef(-1.0 / 720.0);
    c = x * c + coef(1.0 / 24.0);
    c = x * c + coef(-0.5);
    c = dd(1.0f) + x * c;
    const int n = (int)k;
    const Dd u = n & 1 ? c : s, v = n & 1 ? s : c;
    *sn = n & 2 ? -u : u;
    *cs = (n + 1) & 2 ? -v : v;
}

// ---- four lanes, one configuration ---------------------------------------

// A configuration's shared memory.  T: row r of joint j's frame (table
// position j) at hi[12 j + 4 r], the low parts alike; trig: cosine and sine
// (revolute) or the value (prismatic); axes: per joint its axis and origin in
// FP64, filled when the first force comes up.
template <int NJ>
struct alignas(16) EvalScratch {
    float hi[12 * NJ], lo[12 * NJ];
    Dd trig[2 * NJ];
    double axes[6 * NJ];
};

__device__ __forceinline__ float3 place_hi(const float *hi, int j, float4 p)
{
    if (j < 0) return f3(p.x, p.y, p.z);
    const float4 *t = reinterpret_cast<const float4 *>(hi + 12 * j);
    const float4 a = t[0], b = t[1], c = t[2];
    return f3(a.x * p.x + a.y * p.y + a.z * p.z + a.w, b.x * p.x + b.y * p.y + b.z * p.z + b.w,
              c.x * p.x + c.y * p.y + c.z * p.z + c.w);
}

template <int NJ>
__device__ __forceinline__ double3 place_dd(const EvalScratch<NJ> &S, int j, float4 p)
{
    if (j < 0) return d3(p.x, p.y, p.z);
    double v[3];
#pragma unroll
    for (int r = 0; r < 3; r++) {
        const float *h = S.hi + 12 * j + 4 * r, *l = S.lo + 12 * j + 4 * r;
        v[r] = to_double(Dd{h[0], l[0]} * p.x + Dd{h[1], l[1]} * p.y + Dd{h[2], l[2]} * p.z + Dd{h[3], l[3]});
    }
    return d3(v[0], v[1], v[2]);
}

// One obstacle against a leaf sphere: screened in float32 at cf, then in FP64
// at the centre c (placed when the first term is kept).
template <class Centre>
__device__ __forceinline__ void obstacle_term(const float4 *__restrict__ rec, const EnvCounts &n, int k, float3 cf, float r,
                                              float keep, double m, Centre &&centre, double *cost, double3 *g)
{
    if (k < n.ns) {
        const float4 s = rec[k];
        if (-sd_point_f(sub(cf, f3(s.x, s.y, s.z)), r + s.w) > keep)
            point_term(sub(centre(), d3(s.x, s.y, s.z)), (double)r + s.w, m, cost, g);
        return;
    }
    k -= n.ns;
    if (k < n.nc + n.nzc) {
        const bool z = k >= n.nc;
        const float4 a = rec[n.ns + 2 * k], v = rec[n.ns + 2 * k + 1];
        if (-sd_capsule_f(cf, r, a, v, z) > keep) capsule_term(centre(), r, a, v, z, m, cost, g);
        return;
    }
    k -= n.nc + n.nzc;
    const bool z = k >= n.ncb;
    const float4 *p = rec + n.ns + 2 * (n.nc + n.nzc) + 4 * k;
    const float4 c0 = p[0], c1 = p[1], c2 = p[2], c3 = p[3];
    const float3 a1 = f3(c1.x, c1.y, z ? 0.0f : c1.z), a2 = f3(c2.x, c2.y, z ? 0.0f : c2.z),
                 a3 = z ? f3(0.0f, 0.0f, 1.0f) : f3(c3.x, c3.y, c3.z), ce = f3(c0.x, c0.y, c0.z), h = f3(c0.w, c1.w, c2.w);
    if (-sd_box_f(cf, r, ce, a1, a2, a3, h) > keep) box_term(centre(), r, ce, a1, a2, a3, h, m, cost, g);
}

// May sphere (c, r) have an obstacle nearer than r?  By the grid; yes without one.
__device__ __forceinline__ bool env_near(const EnvGrid *g, float3 c, float r)
{
    if (!g) return true;
    const int cell = grid_cell(*g, c.x, c.y, c.z);
    if (cell < 0) return !outside(*g, c.x, c.y, c.z, r);
    const int t = __float2int_ru(r * kGridUnit);
    return t > 255 || (int)__ldg(g->near_ + cell) < t;
}

// Cost and gradient of one configuration per four lanes; every lane of the
// warp calls it, `active` for the configurations that exist.  q: the
// configuration (dof floats).  Returns the cost to all four lanes and, in gr,
// dC/dq of the joints at table positions l, l + 4, ... (l: lane within the
// four).  Configurations out of the kinematics' range (not finite, beyond
// 100 rad in sum) are left to the one-thread form: here, on one of the four
// lanes, or with `left` by the caller, who is told.
template <class Gen>
__device__ double eval(EvalScratch<Gen::kFrames - 1> &S, const ClrModel &M, const ClrEnv &e, const float *q, bool active,
                       float mf, double (&gr)[(Gen::kFrames + 2) / 4], bool *left = nullptr)
{
    constexpr int NJ = Gen::kFrames - 1, SLOTS = (Gen::kFrames + 2) / 4;
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, l = lane & 3, base = lane & ~3;
    const double m = mf;
    double cost = 0.0;
#pragma unroll
    for (int t = 0; t < SLOTS; t++) gr[t] = 0.0;
    float sum = 0.0f;
    if (active)
        for (int d = 0; d < NJ; d++) sum += fabsf(q[d]);
    const bool far = active && !(sum < 100.0f);
    const bool run = active && !far;
    // kinematics
    if (run)
#pragma unroll
        for (int t = 0; t < SLOTS; t++) {
            const int j = l + 4 * t;
            if (j < NJ) {
                const float th = q[M.joints[j].q];
                if (M.joints[j].revolute) {
                    sin_cos(th, &S.trig[2 * j + 1], &S.trig[2 * j]);
                } else {
                    S.trig[2 * j] = dd(th);
                }
            }
        }
    __syncwarp();
    if (run && l < 3) Gen::clr_rows(l, S.trig, S.hi, S.lo);
    __syncwarp();

    // a force gf at c on the sphere whose carrying joints are `chain`, one per
    // lane: each of the four lanes applies it to its own joints
    bool ready = false;
    auto apply = [&](bool have, double3 c, double3 gf, unsigned chain) {
        unsigned pending = __ballot_sync(FULL, have);
        if (!pending) return;
        if (!ready) {
            if (run)
#pragma unroll
                for (int t = 0; t < SLOTS; t++) {
                    const int j = l + 4 * t;
                    if (j < NJ)
#pragma unroll
                        for (int r = 0; r < 3; r++) {
                            S.axes[6 * j + r] = to_double(Dd{S.hi[12 * j + 4 * r + 2], S.lo[12 * j + 4 * r + 2]});
                            S.axes[6 * j + 3 + r] = to_double(Dd{S.hi[12 * j + 4 * r + 3], S.lo[12 * j + 4 * r + 3]});
                        }
                }
            ready = true;
        }
        while (pending) {
            // the first lane of each four that has one
            const unsigned nib = pending >> base & 15u;
            const int src = nib ? base + __ffs(nib) - 1 : lane;
            const double3 c1 = d3(__shfl_sync(FULL, c.x, src), __shfl_sync(FULL, c.y, src), __shfl_sync(FULL, c.z, src));
            const double3 g1 = d3(__shfl_sync(FULL, gf.x, src), __shfl_sync(FULL, gf.y, src), __shfl_sync(FULL, gf.z, src));
            const unsigned ch = __shfl_sync(FULL, chain, src);
            if (nib)
#pragma unroll
                for (int t = 0; t < SLOTS; t++) {
                    const int j = l + 4 * t;
                    if (j < NJ && (ch >> j & 1)) {
                        const double *x = S.axes + 6 * j;
                        const double3 ax = d3(x[0], x[1], x[2]);
                        gr[t] += dot(ax, M.joints[j].revolute ? cross(sub(c1, d3(x[3], x[4], x[5])), g1) : g1);
                    }
                }
            const unsigned b0 = pending & 0x11111111u, r1 = pending & ~(b0 * 15u), b1 = r1 & 0x22222222u,
                           r2 = r1 & ~((b1 >> 1) * 15u), b2 = r2 & 0x44444444u, b3 = r2 & ~((b2 >> 2) * 15u);
            pending &= ~(b0 | b1 | b2 | b3);
        }
    };

    // leaf spheres against the obstacles: the sets that come near any, then
    // their leaves, four at a time
    const EnvGrid *grid = e.grid && e.grid->lo[0] <= e.grid->hi[0] ? e.grid : nullptr;
    const float reach = mf + 2.0f * kScreen, keep = -kScreen - mf;
    for (int p0 = 0; p0 < M.n_leaf_sets; p0 += 32) {   // a bit per set
        unsigned sets = 0;
        for (int s0 = 0; s0 < 32 && p0 + s0 < M.n_leaf_sets; s0 += 4) {
            const int s = p0 + s0 + l;
            bool near = false;
            if (run && s < M.n_leaf_sets) {
                const ClrLeafSet L = M.leaf_sets[s];
                near = env_near(grid, place_hi(S.hi, L.joint, L.ball), L.ball.w + reach);
            }
            sets |= (__ballot_sync(FULL, near) >> base & 15u) << s0;
        }
        int i = 0, n = 0, joint = -1;
        while (true) {
            if (i >= n && sets) {
                const ClrLeafSet L = M.leaf_sets[p0 + __ffs(sets) - 1];
                sets &= sets - 1;
                i = L.first;
                n = L.first + L.n;
                joint = L.joint;
            }
            if (!__any_sync(FULL, i < n)) break;
            bool have = false;
            double3 g = d3(0.0, 0.0, 0.0), c = g;
            if (i + l < n) {
                const float4 s = M.set_leaves[i + l];
                const float3 cf = place_hi(S.hi, joint, s);
                if (env_near(grid, cf, s.w + reach)) {
                    bool placed = false;
                    auto centre = [&]() {
                        if (!placed) c = place_dd(S, joint, s);
                        placed = true;
                        return c;
                    };
                    const int cell = grid ? grid_cell(*grid, cf.x, cf.y, cf.z) : -1;
                    const int t = __float2int_ru((s.w + reach) * kGridUnit);
                    unsigned listed = cell >= 0 && t <= 255 ? listed_below(*grid, cell, t) : 1u << kGridListed;
                    if (listed >> kGridListed) {
                        env_terms(e, cf, s.w, keep, m, centre, &cost, &g);
                    } else {
                        const uint8_t *num = reinterpret_cast<const uint8_t *>(grid->list + 2 * cell + 1);
                        for (; listed; listed &= listed - 1)
                            obstacle_term(e.rec, e.n, __ldg(num + __ffs(listed) - 1), cf, s.w, keep, m, centre, &cost, &g);
                    }
                    have = joint >= 0 && (g.x != 0.0 || g.y != 0.0 || g.z != 0.0);
                }
            }
            apply(have, c, g, joint >= 0 ? M.chain[joint] : 0u);
            i += 4;
        }
    }

    // sphere pairs: frame pairs whose balls come near, then their rows
    for (int p0 = 0; p0 < M.n_pair_sets; p0 += 32) {
        unsigned near_sets = 0;
        for (int s0 = 0; s0 < 32 && p0 + s0 < M.n_pair_sets; s0 += 4) {
            const int s = p0 + s0 + l;
            bool near = false;
            if (run && s < M.n_pair_sets) {
                const ClrPairSet P = M.pair_sets[s];
                const float3 d = sub(place_hi(S.hi, P.ja, P.ball_a), place_hi(S.hi, P.jb, P.ball_b));
                const float rs = P.ball_a.w + P.ball_b.w + reach;
                near = dot(d, d) < rs * rs;
            }
            near_sets |= (__ballot_sync(FULL, near) >> base & 15u) << s0;
        }
        int row = 0, rows = 0, ja = -1, jb = -1;
        while (true) {
            if (row >= rows && near_sets) {
                const ClrPairSet P = M.pair_sets[p0 + __ffs(near_sets) - 1];
                near_sets &= near_sets - 1;
                row = P.first;
                rows = P.first + P.n;
                ja = P.ja;
                jb = P.jb;
            }
            if (!__any_sync(FULL, row < rows)) break;
            ClrPairRow R;
            float3 ca;
            int b = 0, nb = 0;
            if (row + l < rows) {
                R = M.pair_rows[row + l];
                ca = place_hi(S.hi, ja, R.a);
                const float3 d = sub(ca, place_hi(S.hi, jb, R.ball));
                const float rs = R.a.w + R.ball.w + reach;
                if (dot(d, d) < rs * rs) b = R.first, nb = R.first + R.n;
            }
            while (__any_sync(FULL, b < nb)) {
                bool have = false;
                double3 g = d3(0.0, 0.0, 0.0), pa = g, pb = g;
                if (b < nb) {
                    const float4 s = M.pair_spheres[b];
                    if (-sd_point_f(sub(ca, place_hi(S.hi, jb, s)), R.a.w + s.w) > keep) {
                        pa = place_dd(S, ja, R.a);
                        pb = place_dd(S, jb, s);
                        point_term(sub(pa, pb), (double)R.a.w + s.w, m, &cost, &g);
                        have = g.x != 0.0 || g.y != 0.0 || g.z != 0.0;
                    }
                    b++;
                }
                // joints that carry both spheres feel nothing
                const unsigned cha = ja >= 0 ? M.chain[ja] : 0u, chb = jb >= 0 ? M.chain[jb] : 0u;
                apply(have, pa, g, cha & ~chb);
                apply(have, pb, scale(-1.0, g), chb & ~cha);
            }
            row += 4;
        }
    }
    cost += __shfl_xor_sync(FULL, cost, 1);
    cost += __shfl_xor_sync(FULL, cost, 2);

    if (left) {
        *left = far;
    } else if (__any_sync(FULL, far)) {
        // table order, through the shared scratch
        if (far && l == 0) {
            float g[kClrMaxJoints];
            const float c = cost_grad(M, e, q, mf, 1.0f, g);
            for (int j = 0; j < NJ; j++) S.axes[j] = g[M.joints[j].q];
            S.axes[NJ] = c;
        }
        __syncwarp();
        if (far) {
#pragma unroll
            for (int t = 0; t < SLOTS; t++)
                if (l + 4 * t < NJ) gr[t] = S.axes[l + 4 * t];
            cost = S.axes[NJ];
        }
        __syncwarp();
    }
    return cost;
}

}  // namespace clr

// Every waypoint of every path, four lanes each; those out of the kinematics'
// range then by a thread each, next to one another.
template <class Gen>
__global__ void __launch_bounds__(64) k_path_cost_grad(ClrModel M, const ClrEnv *__restrict__ envs, int64_t rows,
                                                      int waypoints, const float *__restrict__ q, float margin,
                                                      float *__restrict__ cost, float *__restrict__ grad)
{
    constexpr int NJ = Gen::kFrames - 1, SLOTS = (Gen::kFrames + 2) / 4;
    __shared__ clr::EvalScratch<NJ> s_eval[16];
    __shared__ bool s_left[16];
    const int l = threadIdx.x & 3;
    const int64_t first = (int64_t)blockIdx.x * 16;
    int64_t row = first + (threadIdx.x >> 2);
    const bool active = row < rows;
    const ClrEnv e = envs[active ? row / waypoints : 0];
    double gr[SLOTS];
    bool left;
    const double c = clr::eval<Gen>(s_eval[threadIdx.x >> 2], M, e, q + (active ? row : 0) * M.dof, active, margin, gr, &left);
    if (active && !left) {
        if (l == 0) cost[row] = (float)c;
#pragma unroll
        for (int t = 0; t < SLOTS; t++)
            if (l + 4 * t < NJ) grad[row * M.dof + M.joints[l + 4 * t].q] = (float)gr[t];
    }
    if (!__syncthreads_or(left)) return;
    if (l == 0) s_left[threadIdx.x >> 2] = left;
    __syncthreads();
    if (threadIdx.x >= 16 || !s_left[threadIdx.x]) return;
    row = first + threadIdx.x;
    float g[kClrMaxJoints];
    cost[row] = clr::cost_grad(M, envs[row / waypoints], q + row * M.dof, margin, 1.0f, g);
    for (int d = 0; d < M.dof; d++) grad[row * M.dof + d] = g[d];
}

// The same with a thread per waypoint, blocks of 64 waypoints of one path and
// the path's obstacles in shared memory: for robots with fewer leaves than four
// lanes (the sphere robot's 256 paths among 32 obstacles 217 us a call, 257
// with four lanes).
template <class Gen>
__global__ void __launch_bounds__(64) k_path_cost_grad_one(ClrModel M, const ClrEnv *__restrict__ envs, int waypoints,
                                                          const float *__restrict__ q, float margin,
                                                          float *__restrict__ cost, float *__restrict__ grad)
{
    extern __shared__ float4 s_env[];
    __shared__ unsigned long long s_bar;
    const int path = blockIdx.y;
    const ClrEnv pe = envs[path];
    stage_env_bulk(s_env, pe.rec, pe.n.records(), &s_bar);
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= waypoints) return;
    const size_t row = (size_t)path * waypoints + w;
    float g[kClrMaxJoints];
    cost[row] = clr::cost_grad(M, ClrEnv{s_env, pe.n}, q + row * M.dof, margin, 1.0f, g);
    for (int d = 0; d < M.dof; d++) grad[row * M.dof + d] = g[d];
}

}  // namespace prrtc
