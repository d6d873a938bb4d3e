// The fast form of the table-driven checkers.
//
// Of the tests that the reference's checker makes on a configuration (about
// 370 sphere-obstacle and 270 sphere-pair tests on the Panda shelf scene)
// nearly all are far from contact.  The fast form finds those by bounds and
// makes only the others: straight-line code marks the steps of the schedule
// whose gate can be hit at all (a byte of the clearance grid per
// environment gate; one test per pair of frames, then per pair of gates,
// for self groups), and a walk tests the marked ones in the schedule's
// order, leaf spheres by the grid's lists and leaf pairs row by row.
//
// The marking code keeps everything in registers (frames die as the chain goes
// on); a lane with marked steps computes its frames again, into local memory,
// for the walk (near_resolve): most warps of an edge's points have none, and
// storing 7 frames and 11 centres for every point had cost more than that.
//
// It answers only where the answer is beyond rounding: a test within microns of
// contact (near_verdict), a configuration out of the range those bounds
// hold for or an environment without a grid is left to the exact form (about
// one configuration in a thousand).  So verdicts are the exact form's, bit
// for bit, and so are the work counts: a test that was skipped counts as the
// reference makes it.
#pragma once

#include "device_common.cuh"

namespace prrtc {

enum NearAnswer { kNearHit = 0, kNearFree = 1, kNearUnsure = 2 };

// Leaf pairs of one block (GenPairBlock).  row > 0: rows of `row` pairs with one
// sphere a each, every row against the same spheres b, all of which lie in
// the sphere `bound` of frame B.
struct alignas(16) NearPairBlock {
    int fa, fb, first, n;
    float4 bound;
    int row;
};

// Sine and cosine to 1.75 x 2^-24 (1.0e-7) for |x| <= 100: x minus a multiple of
// pi / 2 in three parts, the first two products exact (the reduction of W. J. Cody
// and W. Waite, "Software Manual for the Elementary Functions", 1980), then the
// Taylor series up to r^9 / r^10.  The exact form has the library's; the two
// forms' centres differ by at most 5.0e-7 m (near_verdict).
__device__ __forceinline__ void near_sincos(float x, float *s, float *c)
{
    const float k = rintf(x * 0.636619772f);
    const float r = fmaf(-k, 0x1.0b4612p-34f, fmaf(-k, 0x1.b544p-16f, fmaf(-k, 0x1.921ep+0f, x)));
    const float y = r * r;
    float u = fmaf(y, 1.0f / 362880.0f, -1.0f / 5040.0f), v = fmaf(y, -1.0f / 3628800.0f, 1.0f / 40320.0f);
    u = fmaf(y, u, 1.0f / 120.0f), v = fmaf(y, v, -1.0f / 720.0f);
    u = fmaf(y, u, -1.0f / 6.0f), v = fmaf(y, v, 1.0f / 24.0f);
    v = fmaf(y, v, -0.5f);
    u = fmaf(r * y, u, r), v = fmaf(y, v, 1.0f);
    const int n = (int)k;
    const float a = n & 1 ? v : u, b = n & 1 ? u : v;
    *s = n & 2 ? -a : a;
    *c = (n + 1) & 2 ? -b : b;
}

// The environment as the marking code reads it.
struct NearView {
    const EnvGrid *g;
    float pad;
    int pad_units;   // pad in grid units, rounded up
    bool wide;       // the pad is more than the leaf marks allow for (kNearPad): gates alone decide
};
constexpr float kNearPad = 1e-4f;

template <class Ctx>
__device__ __forceinline__ NearView near_view(const Ctx &ctx)
{
    return NearView{ctx.env.grid, ctx.pad, __float2int_ru(ctx.pad * kGridUnit), ctx.pad > kNearPad};
}

// Can sphere c (radius c.w, `units` in grid units rounded up) touch an obstacle?
__device__ __forceinline__ bool may_hit_env(const NearView &v, float4 c, int units)
{
    const int cell = grid_cell(*v.g, c.x, c.y, c.z);
    if (cell >= 0) return (int)__ldg(v.g->near_ + cell) < units + v.pad_units;
    return !(c.w + v.pad < v.g->out_r);
}

// The same for a sphere larger than the cells' margin around the obstacles:
// outside the cells by its distance to the box around them.
__device__ __forceinline__ bool may_hit_env_wide(const NearView &v, float4 c, int units)
{
    const int cell = grid_cell(*v.g, c.x, c.y, c.z);
    return cell >= 0 ? (int)__ldg(v.g->near_ + cell) < units + v.pad_units : !outside(*v.g, c.x, c.y, c.z, c.w + v.pad);
}

// Can the two spheres (gates, or spheres around several gates) overlap?
__device__ __forceinline__ bool may_hit_pair(const NearView &v, float4 a, float4 b)
{
    const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z, rs = (a.w + b.w) + 2.0f * v.pad + 1e-5f;
    return dx * dx + dy * dy + dz * dz < rs * rs;
}

// The gate pair's own test (near_verdict).
__device__ __forceinline__ int near_gate(const NearView &v, float4 a, float4 b)
{
    const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
    return near_verdict(dx * dx + dy * dy + dz * dz, (a.w + b.w) + 2.0f * v.pad);
}

// Leaf marks.  A self group whose gates overlap often without its leaves being
// near (two neighbouring links' gates always do) is marked by its leaves:
// balls around one link's leaves are brought into the other link's frame
// (local_point: coordinates and squared length), where that link's leaves are
// constants, and |a - p|^2 < s^2 is three multiply-adds with immediate operands
// and a comparison: (-2 a) . p + |p|^2 < s^2 - |a|^2.  A step that its leaves
// leave unmarked although its gates overlap is `passed`: the reference tests
// all its leaf pairs, and they count.
__device__ __forceinline__ float4 local_point(const Frame &T, float4 c)
{
    const float dx = c.x - T.m[3], dy = c.y - T.m[7], dz = c.z - T.m[11];
    const float x = T.m[0] * dx + T.m[4] * dy + T.m[8] * dz, y = T.m[1] * dx + T.m[5] * dy + T.m[9] * dz,
                z = T.m[2] * dx + T.m[6] * dy + T.m[10] * dz;
    return make_float4(x, y, z, x * x + y * y + z * z);
}
__device__ __forceinline__ bool near_leaf(float4 p, float ax, float ay, float az, float limit)
{
    return fmaf(p.x, ax, fmaf(p.y, ay, fmaf(p.z, az, p.w))) < limit;
}

// Sphere against every obstacle: kNearFree (cost: every test's FLOPs),
// kNearHit (cost: those up to the first hit) or kNearUnsure.
static __device__ __noinline__ int near_env_all(const EnvGrid *g, float x, float y, float z, float r, int *cost)
{
    for (int k = 0; k < g->counts.obstacles(); k++) {
        const int h = near_test(g->rec, g->counts, k, x, y, z, r);
        if (h == 2) return kNearUnsure;
        if (h == 1) {
            *cost = env_cost(g->counts, k + 1);
            return kNearHit;
        }
    }
    *cost = g->cost;
    return kNearFree;
}

__device__ __forceinline__ int near_env(const EnvGrid *g, float x, float y, float z, float r, int &cost)
{
    cost = g->cost;
    const int cell = grid_cell(*g, x, y, z);
    if (cell < 0 && outside(*g, x, y, z, r)) return kNearFree;
    const int t = __float2int_ru(r * kGridUnit);
    if (cell >= 0 && t <= 255) {
        if ((int)__ldg(g->near_ + cell) >= t) return kNearFree;
        unsigned m = listed_below(*g, cell, t);
        if (!(m >> kGridListed)) {
            const uint8_t *num = reinterpret_cast<const uint8_t *>(g->list + 2 * cell + 1);
            for (; m; m &= m - 1) {
                const int k = __ldg(num + __ffs(m) - 1);
                const int h = near_test(g->rec, g->counts, k, x, y, z, r);
                if (h == 2) return kNearUnsure;
                if (h == 1) {
                    cost = env_cost(g->counts, k + 1);
                    return kNearHit;
                }
            }
            return kNearFree;
        }
    }
    int c;
    const int h = near_env_all(g, x, y, z, r, &c);
    cost = c;
    return h;
}

// Leaf pairs of one block; cost as above.
__device__ __forceinline__ int near_pairs(const Frame &Tab, const LeafPair *__restrict__ pairs, const NearPairBlock &b,
                                          float pad2, int &cost)
{
    const int row = b.row ? b.row : b.n;
    unsigned rows = 1;
    if (b.row) {   // rows whose sphere a is clear of all spheres b cannot hit
        float x, y, z;
        xform(Tab, b.bound, x, y, z);
        rows = 0;
        for (int i = 0, k = b.first; k < b.first + b.n; i++, k += row) {
            const float4 a = pairs[k].a;
            const float dx = a.x - x, dy = a.y - y, dz = a.z - z, rs = a.w + b.bound.w + pad2 + 1e-5f;
            rows |= (dx * dx + dy * dy + dz * dz < rs * rs ? 1u : 0u) << i;
        }
    }
    for (; rows; rows &= rows - 1) {
        const int first = (__ffs(rows) - 1) * row;
        for (int i = first; i < first + row; i++) {
            const LeafPair p = pairs[b.first + i];
            float x, y, z;
            xform(Tab, p.b, x, y, z);
            const float dx = p.a.x - x, dy = p.a.y - y, dz = p.a.z - z;
            const int h = near_verdict(dx * dx + dy * dy + dz * dz, p.a.w + p.b.w + pad2);
            if (h == 2) return kNearUnsure;
            if (h == 1) {
                cost = kFlopPair * (i + 1);
                return kNearHit;
            }
        }
    }
    cost = kFlopPair * b.n;
    return kNearFree;
}

// A configuration by value.
template <int D>
struct NearCfg {
    float q[D];
};
// A frame in local memory, three 16-byte rows.
struct NearFrame {
    float4 r[3];
    __device__ __forceinline__ void set(const Frame &f)
    {
        r[0] = make_float4(f.m[0], f.m[1], f.m[2], f.m[3]);
        r[1] = make_float4(f.m[4], f.m[5], f.m[6], f.m[7]);
        r[2] = make_float4(f.m[8], f.m[9], f.m[10], f.m[11]);
    }
};
__device__ __forceinline__ Frame frame_at(const NearFrame *F, int i)   // i: joint's config index, -1 the world
{
    if (i < 0) return world_frame();
    const float4 a = F[i].r[0], b = F[i].r[1], c = F[i].r[2];
    return Frame{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w}};
}

// The marked steps, in the schedule's order.  The lanes of a warp take the
// union of their steps together, so that they read the same table entries
// and run the same code.  extra: FLOPs of the passed steps' leaf pairs.
// Returns NearAnswer + 4 * FLOPs: on a collision those of the whole check so
// far, else those beyond what all steps cost with nothing hit (negative where
// a gate was hit early and its leaves cost less).  T: the robot's tables.
template <class T>
__device__ __noinline__ unsigned near_resolve(const NearCfg<T::kDof> q, const StepMarks<T::kWords> m, int extra,
                                              const EnvGrid *g, float pad)
{
    NearFrame F[T::kFrames];
    float4 G[T::kGates];
    T::frames(q.q, F, G);
#pragma unroll 1
    for (int w = 0; w < T::kWords; w++) {
        // (the lanes that are together here, each with its own bits among `todo`:
        // verdicts do not depend on which lanes are, the speed does)
        const unsigned word = m.marked[w];
        unsigned todo = __reduce_or_sync(__activemask(), word);
#pragma unroll 1
        for (; todo; todo &= todo - 1) {
            const int s = __ffs(todo) - 1;
            if (!(word >> s & 1)) continue;
            const GenSched e = T::steps()[32 * w + s];
            int h = kNearFree, c;
            if (e.kind == 0) {
                const GenEnvGroup gr = T::env_groups()[e.index];
                bool go = true;
                if (gr.gate >= 0) {
                    const float4 p = G[gr.gate];
                    const int a = near_env(g, p.x, p.y, p.z, p.w + pad, c);
                    if (a == kNearUnsure) return kNearUnsure;
                    extra += c;
                    go = a == kNearHit;
                }
                if (go)
                    for (int k = gr.first_block; k < gr.first_block + gr.nblocks && h == kNearFree; k++) {
                        const GenLeafBlock b = T::leaf_blocks()[k];
                        const Frame A = frame_at(F, b.frame);
                        for (int i = b.first; i < b.first + b.n && h == kNearFree; i++) {
                            const float4 l = T::leaves()[i];
                            float x, y, z;
                            xform(A, l, x, y, z);
                            h = near_env(g, x, y, z, l.w + pad, c);
                            extra += c;
                        }
                    }
                extra -= g->cost * e.tests;
            } else {
                const GenSelfGroup gr = T::self_groups()[e.index];
                const float4 a = G[gr.ga], b = G[gr.gb];
                const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
                const int gate = near_verdict(dx * dx + dy * dy + dz * dz, (a.w + b.w) + 2.0f * pad);
                if (gate == 2) return kNearUnsure;
                if (gate == 1)
                    for (int k = gr.first_block; k < gr.first_block + gr.nblocks && h == kNearFree; k++) {
                        const NearPairBlock b = T::pair_blocks()[k];
                        h = near_pairs(relative_frame(frame_at(F, b.fa), frame_at(F, b.fb)), T::pairs(), b, 2.0f * pad, c);
                        extra += c;
                    }
            }
            if (h == kNearUnsure) return kNearUnsure;
            if (h == kNearHit) {   // the passed steps after this one were not reached
                unsigned after = m.passed[w] & ~0u << s;
                for (int v = w;;) {
                    for (; after; after &= after - 1) extra -= kFlopPair * T::steps()[32 * v + __ffs(after) - 1].tests;
                    if (++v >= T::kWords) break;
                    after = m.passed[v];
                }
                return kNearHit + 4u * (unsigned)(g->cost * e.env + kFlopPair * e.self + extra);
            }
        }
    }
    return kNearFree + 4u * (unsigned)extra;
}

}  // namespace prrtc
