// Clearance grids of environments (EnvGrid, device_common.cuh), built on the
// device.  No reference counterpart: pRRTC's checker tests every sphere
// against every obstacle (sphere_environment_in_collision, utils.cuh:211-242).
//
// One thread per cell walks the obstacles in their order, bounds the distance
// from the cell to each from below, and keeps the 16 nearest by a chain of
// min / max in registers.  What bounds the build of many is that arithmetic, ~60
// instructions per obstacle and cell; of one, its latency, so the records come
// to shared memory first and an upload's header is made on the host.
#include <algorithm>

#include "device_common.cuh"
#include "prrtc_internal.h"

namespace prrtc {

namespace {

constexpr int kThreads = 128;
constexpr float kInflate = 0.2f;    // the cells reach this far around the obstacles
constexpr float kRoom = 3.0f;       // and no further than this from the origin, where robots work
constexpr float kSlack = 2e-4f;     // taken off every bound: far above any rounding in it or in a checker's distance

struct Box {
    float lo[3], hi[3];
};

__device__ __forceinline__ float clamp01(float v) { return fmaxf(fminf(v, 1.0f), 0.0f); }

// the box around obstacle k, and whether every value of it is one the bounds
// hold for: at most kGridReach in size, axes no longer than 2, a capsule's
// rdv the inverse square of its length (or the length zero)
__host__ __device__ bool obstacle_box(const float4 *rec, const EnvCounts &n, int k, Box &b)
{
    auto small = [](float v, float most) { return fabsf(v) <= most; };   // false for NaN
    float c[3], e[3];
    bool ok;
    if (k < n.ns) {
        const float4 s = rec[k];
        ok = small(s.x, kGridReach) && small(s.y, kGridReach) && small(s.z, kGridReach) && small(s.w, kGridReach);
        c[0] = s.x, c[1] = s.y, c[2] = s.z;
        e[0] = e[1] = e[2] = fabsf(s.w);
    } else if (k < n.ns + n.nc + n.nzc) {
        const float4 *p = rec + n.ns + 2 * (k - n.ns);
        const float4 a = p[0];
        float4 v = p[1];
        ok = small(a.x, kGridReach) && small(a.y, kGridReach) && small(a.z, kGridReach) && small(a.w, kGridReach) &&
             small(v.x, kGridReach) && small(v.y, kGridReach) && small(v.z, kGridReach);
        if (k >= n.ns + n.nc) v.x = v.y = 0.0f;
        const float vv = v.x * v.x + v.y * v.y + v.z * v.z;
        ok = ok && (vv == 0.0f || small(v.w * vv - 1.0f, 0.01f));
        c[0] = a.x + 0.5f * v.x, c[1] = a.y + 0.5f * v.y, c[2] = a.z + 0.5f * v.z;
        e[0] = 0.5f * fabsf(v.x) + fabsf(a.w), e[1] = 0.5f * fabsf(v.y) + fabsf(a.w), e[2] = 0.5f * fabsf(v.z) + fabsf(a.w);
    } else {
        const bool upright = k >= n.ns + n.nc + n.nzc + n.ncb;
        const float4 *p = rec + n.ns + 2 * (n.nc + n.nzc) + 4 * (k - n.ns - n.nc - n.nzc);
        const float4 c0 = p[0];
        float4 a[3] = {p[1], p[2], p[3]};
        if (upright) {
            a[0].z = a[1].z = 0.0f;
            a[2] = make_float4(0.0f, 0.0f, 1.0f, 0.0f);
        }
        const float h[3] = {c0.w, p[1].w, p[2].w};
        ok = small(c0.x, kGridReach) && small(c0.y, kGridReach) && small(c0.z, kGridReach);
        c[0] = c0.x, c[1] = c0.y, c[2] = c0.z;
        e[0] = e[1] = e[2] = 0.0f;
        for (int i = 0; i < 3; i++) {
            ok = ok && small(a[i].x, 2.0f) && small(a[i].y, 2.0f) && small(a[i].z, 2.0f) && small(h[i], kGridReach);
            // a box: its axes are orthonormal (what the extents below rest on)
            const float4 o = a[(i + 1) % 3];
            ok = ok && small(a[i].x * a[i].x + a[i].y * a[i].y + a[i].z * a[i].z - 1.0f, 1e-3f) &&
                 small(a[i].x * o.x + a[i].y * o.y + a[i].z * o.z, 1e-3f);
            e[0] += fabsf(a[i].x * h[i]);
            e[1] += fabsf(a[i].y * h[i]);
            e[2] += fabsf(a[i].z * h[i]);
        }
        for (int i = 0; i < 3; i++) e[i] *= 1.01f;
    }
    for (int i = 0; i < 3; i++) {
        b.lo[i] = c[i] - e[i] - 1e-3f;
        b.hi[i] = c[i] + e[i] + 1e-3f;
    }
    return ok;
}

// A lower bound of what the reference's test of obstacle k compares a
// sphere's radius with, over the cell of centre c and half-extents h (half
// diagonal hd): the test hits a sphere of radius r only where r exceeds it.
//   sphere, capsule: the distance to the centre or segment minus |radius|
//     (the test's point lies on the segment whatever rounding its parameter
//     has).
//   box: the test's own terms max(0, |a_i . (p - c)| - h_i), each lowered by
//     the most that a_i . p changes over the cell.
__device__ __forceinline__ float gap(float dx, float dy, float dz, float hx, float hy, float hz)
{
    const float x = fmaxf(fabsf(dx) - hx, 0.0f), y = fmaxf(fabsf(dy) - hy, 0.0f), z = fmaxf(fabsf(dz) - hz, 0.0f);
    return sqrtf(x * x + y * y + z * z);
}

__device__ __forceinline__ unsigned bound_key(float d, int k)
{
    const float u = floorf((d - kSlack) * kGridUnit);
    return ((u >= 255.0f ? 255u : u > 0.0f ? (unsigned)u : 0u) << 8) | (unsigned)k;   // NaN: 0
}

__device__ __forceinline__ void insert(unsigned (&key)[16], unsigned v)
{
    if (v >= key[15] || v >= (255u << 8)) return;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const unsigned lo = min(key[i], v);
        v = max(key[i], v);
        key[i] = lo;
    }
}

// The header of a grid over the box b around usable obstacles (ok), and where
// it and what it points to lie.
__host__ __device__ void place(EnvGrid &g, const float4 *rec, const EnvGrid *where, int max_cells)
{
    g.rec = rec;
    g.near_ = reinterpret_cast<const uint8_t *>(where + 1);
    g.list = reinterpret_cast<const uint4 *>(g.near_ + max_cells);
}

__host__ __device__ EnvGrid make_header(const Box &b, bool ok, const EnvCounts &n, int max_cells)
{
    EnvGrid g{};
    g.out_r = -1.0f;
    float cells[3], from[3], ext[3];
    for (int i = 0; i < 3; i++) {
        g.lo[i] = ok ? b.lo[i] : 1.0f;
        g.hi[i] = ok ? b.hi[i] : -1.0f;
        from[i] = fmaxf(b.lo[i] - kInflate, -kRoom);
        ext[i] = fminf(b.hi[i] + kInflate, kRoom) - from[i];
    }
    g.cost = env_cost_all(n);
    g.counts = n;
    if (ok && ext[0] > 1e-3f && ext[1] > 1e-3f && ext[2] > 1e-3f) {
        // cubic cells, at most max_cells of them
        const float size = cbrtf(ext[0] * ext[1] * ext[2] / (float)max_cells);
        for (int i = 0; i < 3; i++) cells[i] = fmaxf(1.0f, fminf(128.0f, floorf(ext[i] / size)));
        g.out_r = 0.95f * kInflate;
        while (cells[0] * cells[1] * cells[2] > (float)max_cells) {
            const int i = cells[0] >= cells[1] && cells[0] >= cells[2] ? 0 : cells[1] >= cells[2] ? 1 : 2;
            cells[i] -= 1.0f;
        }
        for (int i = 0; i < 3; i++) {
            g.n[i] = (int)cells[i];
            g.inv[i] = cells[i] / ext[i];
            g.off[i] = -from[i] * g.inv[i] - 0.5f;
            if (b.lo[i] - kInflate < -kRoom || b.hi[i] + kInflate > kRoom) g.out_r = -1.0f;
        }
    }
    return g;
}

// Bounds and list of one cell; rec: the obstacles in shared memory.
__device__ __forceinline__ void build_cell(const EnvGrid &g, const float4 *rec, const EnvCounts &n, int cell)
{
    // the cell: centre and half-extents, a little larger than the cut (a
    // point's cell is rounded)
    const int ix = cell % g.n[0], iy = cell / g.n[0] % g.n[1], iz = cell / (g.n[0] * g.n[1]);
    const float cx = ((float)ix - g.off[0]) / g.inv[0], cy = ((float)iy - g.off[1]) / g.inv[1],
                cz = ((float)iz - g.off[2]) / g.inv[2];
    const float hx = 0.5005f / g.inv[0], hy = 0.5005f / g.inv[1], hz = 0.5005f / g.inv[2];
    const float hd = sqrtf(hx * hx + hy * hy + hz * hz);
    unsigned key[16];
#pragma unroll
    for (int i = 0; i < 16; i++) key[i] = 0xFFFFu;
    const float4 *p = rec;
    int k = 0;
    for (int i = 0; i < n.ns; i++, k++) {
        const float4 s = p[i];
        insert(key, bound_key(gap(cx - s.x, cy - s.y, cz - s.z, hx, hy, hz) - fabsf(s.w), k));
    }
    p += n.ns;
    for (int i = 0; i < n.nc + n.nzc; i++, k++) {
        const float4 a = p[2 * i];
        float4 v = p[2 * i + 1];
        if (i >= n.nc) v.x = v.y = 0.0f;
        const float dx = cx - a.x, dy = cy - a.y, dz = cz - a.z, vv = v.x * v.x + v.y * v.y + v.z * v.z;
        const float t = vv > 0.0f ? clamp01((dx * v.x + dy * v.y + dz * v.z) / vv) : 0.0f;
        const float ex = dx - t * v.x, ey = dy - t * v.y, ez = dz - t * v.z;
        insert(key, bound_key(sqrtf(ex * ex + ey * ey + ez * ez) - hd - fabsf(a.w), k));
    }
    p += 2 * (n.nc + n.nzc);
    for (int i = 0; i < n.ncb + n.nzb; i++, k++) {
        const float4 c0 = p[4 * i], c1 = p[4 * i + 1], c2 = p[4 * i + 2], c3 = p[4 * i + 3];
        const float dx = cx - c0.x, dy = cy - c0.y, dz = cz - c0.z;
        auto term = [&](float ax, float ay, float az, float h) {
            return fmaxf(fabsf(ax * dx + ay * dy + az * dz) - h - (fabsf(ax) * hx + fabsf(ay) * hy + fabsf(az) * hz), 0.0f);
        };
        const bool up = i >= n.ncb;
        const float t1 = term(c1.x, c1.y, up ? 0.0f : c1.z, c0.w), t2 = term(c2.x, c2.y, up ? 0.0f : c2.z, c1.w),
                    t3 = up ? term(0.0f, 0.0f, 1.0f, c2.w) : term(c3.x, c3.y, c3.z, c2.w);
        insert(key, bound_key(sqrtf(t1 * t1 + t2 * t2 + t3 * t3), k));
    }
    const unsigned next = key[15] >> 8;
    const_cast<uint8_t *>(g.near_)[cell] = (uint8_t)(key[0] >> 8);
    // the listed ones by obstacle number (a bitonic network; unused entries last)
    key[15] = 0xFFFFu;
#pragma unroll
    for (int i = 0; i < 16; i++) key[i] = ((key[i] & 255u) << 8) | (key[i] >> 8);
#pragma unroll
    for (int size = 2; size <= 16; size <<= 1)
#pragma unroll
        for (int step = size >> 1; step > 0; step >>= 1)
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const int j = i ^ step;
                if (j > i) {
                    const unsigned lo = min(key[i], key[j]), hi = max(key[i], key[j]);
                    key[i] = (i & size) ? hi : lo;
                    key[j] = (i & size) ? lo : hi;
                }
            }
    unsigned lb[4], num[4];
#pragma unroll
    for (int w = 0; w < 4; w++) {
        lb[w] = num[w] = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const unsigned v = 4 * w + i == 15 ? 0xFF00u | next : key[4 * w + i];
            lb[w] |= (v & 255u) << (8 * i);
            num[w] |= (v >> 8) << (8 * i);
        }
    }
    uint4 *L = const_cast<uint4 *>(g.list) + 2 * (size_t)cell;
    L[0] = make_uint4(lb[0], lb[1], lb[2], lb[3]);
    L[1] = make_uint4(num[0], num[1], num[2], num[3]);
}

// Scene blockIdx.y of `scenes`, its header from its records; without `scenes`
// the one grid of header `one`.
__global__ void __launch_bounds__(kThreads) k_env_grid(const BatchQueryDesc *__restrict__ scenes, EnvGrid one, int max_cells)
{
    __shared__ Box s_box[kThreads / 32];
    __shared__ EnvGrid s_g;
    __shared__ float4 s_rec[4 * kGridMaxObstacles];
    if (!scenes) {
        if (threadIdx.x == 0) s_g = one;
    } else {
        const BatchQueryDesc Q = scenes[blockIdx.y];
        // the box around the obstacles (every block for itself: at most 255 obstacles)
        Box b;
        for (int i = 0; i < 3; i++) {
            b.lo[i] = 1e30f;
            b.hi[i] = -1e30f;
        }
        const int no = Q.env_n.obstacles();
        bool ok = no >= 1 && no <= kGridMaxObstacles;
        if (ok)
            for (int k = threadIdx.x; k < no; k += kThreads) {
                Box o;
                ok = obstacle_box(Q.env, Q.env_n, k, o) && ok;
                for (int i = 0; i < 3; i++) {
                    b.lo[i] = fminf(b.lo[i], o.lo[i]);
                    b.hi[i] = fmaxf(b.hi[i], o.hi[i]);
                }
            }
        for (int i = 0; i < 3; i++)
            for (int off = 16; off > 0; off >>= 1) {
                b.lo[i] = fminf(b.lo[i], __shfl_xor_sync(0xffffffffu, b.lo[i], off));
                b.hi[i] = fmaxf(b.hi[i], __shfl_xor_sync(0xffffffffu, b.hi[i], off));
            }
        if ((threadIdx.x & 31) == 0) s_box[threadIdx.x >> 5] = b;
        ok = __syncthreads_and(ok);
        if (threadIdx.x == 0) {
            for (int w = 1; w < kThreads / 32; w++)
                for (int i = 0; i < 3; i++) {
                    b.lo[i] = fminf(b.lo[i], s_box[w].lo[i]);
                    b.hi[i] = fmaxf(b.hi[i], s_box[w].hi[i]);
                }
            s_g = make_header(b, ok, Q.env_n, max_cells);
            place(s_g, Q.env, Q.grid, max_cells);
        }
    }
    if (threadIdx.x == 0 && blockIdx.x == 0)   // the header lies in front of the bounds
        *(reinterpret_cast<EnvGrid *>(const_cast<uint8_t *>(s_g.near_)) - 1) = s_g;
    __syncthreads();
    const int cells = s_g.n[0] * s_g.n[1] * s_g.n[2];
    if (cells == 0) return;
    const EnvCounts n = s_g.counts;
    for (int i = threadIdx.x; i < n.records(); i += kThreads) s_rec[i] = __ldg(s_g.rec + i);
    __syncthreads();
    for (int cell = blockIdx.x * kThreads + threadIdx.x; cell < cells; cell += gridDim.x * kThreads) build_cell(s_g, s_rec, n, cell);
}
}  // namespace

// (the lists, 16-byte entries, follow the header and a multiple of 16 bytes)
static_assert(sizeof(EnvGrid) % 16 == 0, "the lists behind the header are 16-byte entries");
bool env_grid_header(const float4 *host_rec, const EnvCounts &n, int cells, EnvGrid *out)
{
    Box all{{1e30f, 1e30f, 1e30f}, {-1e30f, -1e30f, -1e30f}};
    if (n.obstacles() < 1 || n.obstacles() > kGridMaxObstacles) return false;
    for (int k = 0; k < n.obstacles(); k++) {
        Box b;
        if (!obstacle_box(host_rec, n, k, b)) return false;
        for (int i = 0; i < 3; i++) {
            all.lo[i] = std::min(all.lo[i], b.lo[i]);
            all.hi[i] = std::max(all.hi[i], b.hi[i]);
        }
    }
    *out = make_header(all, true, n, cells);
    return true;
}

size_t env_grid_bytes(int cells) { return sizeof(EnvGrid) + (size_t)cells * 33; }

cudaError_t launch_env_grid(EnvGrid header, const float4 *rec, const EnvGrid *where, int cells, cudaStream_t st)
{
    place(header, rec, where, cells);
    k_env_grid<<<(cells + kThreads - 1) / kThreads, kThreads, 0, st>>>(nullptr, header, cells);
    return cudaGetLastError();
}

cudaError_t launch_env_grids(const BatchQueryDesc *scenes, int n, int cells, cudaStream_t st)
{
    for (int first = 0; first < n; first += 65535) {
        // (many scenes: four cells a thread, for fewer headers and records read)
        const int per = n >= 64 ? 4 * kThreads : kThreads;
        const dim3 grid((cells + per - 1) / per, std::min(n - first, 65535));
        k_env_grid<<<grid, kThreads, 0, st>>>(scenes + first, EnvGrid{}, cells);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace prrtc
