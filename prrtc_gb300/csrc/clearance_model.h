// A robot's collision model rearranged for the clearance kernels (host
// side): the generated tables of robots/<robot>_model.h reindexed by table
// position, env leaf spheres and self-collision leaf pairs expanded.
#pragma once

#include <algorithm>
#include <cmath>
#include <map>
#include <utility>
#include <vector>

#include "clearance_device.cuh"
#include "prrtc/prrtc.h"
#include "robots/baxter_model.h"
#include "robots/fetch_model.h"
#include "robots/panda_model.h"
#include "robots/sphere_model.h"

namespace prrtc {

struct ClrHostModel {
    int dof = 0;
    std::vector<prrtc_joint_def> joints;
    std::vector<int> parent, leaf_joint;
    std::vector<float4> leaf, pa, pb;
    std::vector<int2> pair_joint;
    std::vector<unsigned> chain;
    std::vector<ClrLeafSet> leaf_sets;
    std::vector<float4> set_leaves, pair_spheres;
    std::vector<ClrPairSet> pair_sets;
    std::vector<ClrPairRow> pair_rows;

    // A ClrModel whose pointers are this object's own arrays (host memory).
    ClrModel host_view() const
    {
        return ClrModel{dof, (int)joints.size(), (int)leaf.size(), (int)pa.size(), joints.data(), parent.data(),
                        leaf.data(), leaf_joint.data(), pa.data(), pb.data(), pair_joint.data(),
                        (int)leaf_sets.size(), (int)pair_sets.size(), chain.data(), leaf_sets.data(), set_leaves.data(),
                        pair_sets.data(), pair_rows.data(), pair_spheres.data()};
    }
};

// A ball around spheres (radius rounded up): towards the farthest one in
// shrinking steps.
inline float4 clr_ball(const std::vector<float4> &s)
{
    double c[3] = {0.0, 0.0, 0.0};
    for (const float4 &p : s) c[0] += p.x / s.size(), c[1] += p.y / s.size(), c[2] += p.z / s.size();
    auto reach = [&](const float4 &p) { return std::hypot(p.x - c[0], p.y - c[1], p.z - c[2]) + std::fabs(p.w); };
    for (int k = 0; k < 500; k++) {
        const float4 *far = &s[0];
        for (const float4 &p : s)
            if (reach(p) > reach(*far)) far = &p;
        const double v[3] = {far->x - c[0], far->y - c[1], far->z - c[2]}, n = std::hypot(v[0], v[1], v[2]);
        if (n < 1e-9) break;
        const double step = std::min(n, reach(*far) * 0.5 / (k + 2)) / n;
        for (int d = 0; d < 3; d++) c[d] += step * v[d];
    }
    for (double &x : c) x = (float)x;
    double r = 0.0;
    for (const float4 &p : s) r = std::max(r, reach(p));
    return make_float4((float)c[0], (float)c[1], (float)c[2], (float)(r * 1.00001 + 1e-5));
}

// Spheres cut along their longest extent into parts of at most `most`.
inline std::vector<std::vector<float4>> clr_parts(std::vector<float4> s, int most)
{
    auto extent = [&](auto &&get) {
        float lo = 1e30f, hi = -1e30f;
        for (const float4 &p : s) lo = std::min(lo, get(p)), hi = std::max(hi, get(p));
        return hi - lo;
    };
    const float ex = extent([](const float4 &p) { return p.x; }), ey = extent([](const float4 &p) { return p.y; }),
                ez = extent([](const float4 &p) { return p.z; });
    std::stable_sort(s.begin(), s.end(), [&](const float4 &a, const float4 &b) {
        return ex >= ey && ex >= ez ? a.x < b.x : ey >= ez ? a.y < b.y : a.z < b.z;
    });
    const int n = (int)s.size(), parts = (n + most - 1) / most;
    std::vector<std::vector<float4>> out;
    for (int k = 0; k < parts; k++) out.emplace_back(s.begin() + n * k / parts, s.begin() + n * (k + 1) / parts);
    return out;
}

// The four-lane form's tables: each frame's leaves in sets of at most 8, and the
// pairs of every two frames in rows of one sphere against at most 6.
inline void clr_sets(ClrHostModel &h)
{
    h.chain.resize(h.joints.size());
    for (size_t j = 0; j < h.joints.size(); j++) h.chain[j] = 1u << j | (h.parent[j] >= 0 ? h.chain[h.parent[j]] : 0u);
    std::map<int, std::vector<float4>> frames;
    for (size_t i = 0; i < h.leaf.size(); i++) frames[h.leaf_joint[i]].push_back(h.leaf[i]);
    for (auto &[joint, leaves] : frames) {
        for (const std::vector<float4> &part : clr_parts(leaves, 8)) {
            h.leaf_sets.push_back(ClrLeafSet{clr_ball(part), joint, (int)h.set_leaves.size(), (int)part.size(), 0});
            h.set_leaves.insert(h.set_leaves.end(), part.begin(), part.end());
        }
    }
    // pairs by frames, in rows of one sphere a
    struct Row {
        float4 a;
        std::vector<float4> b;
    };
    std::map<std::pair<int, int>, std::vector<Row>> pairs;
    for (size_t i = 0; i < h.pa.size(); i++) {
        std::vector<Row> &rows = pairs[{h.pair_joint[i].x, h.pair_joint[i].y}];
        const float4 a = h.pa[i];
        auto same = [&](const Row &r) { return r.a.x == a.x && r.a.y == a.y && r.a.z == a.z && r.a.w == a.w; };
        auto it = std::find_if(rows.begin(), rows.end(), same);
        if (it == rows.end()) it = rows.insert(rows.end(), Row{a, {}});
        it->b.push_back(h.pb[i]);
    }
    for (auto &[frame, rows] : pairs) {
        std::vector<float4> as, bs;
        for (const Row &r : rows) {
            as.push_back(r.a);
            bs.insert(bs.end(), r.b.begin(), r.b.end());
        }
        h.pair_sets.push_back(ClrPairSet{clr_ball(as), clr_ball(bs), frame.first, frame.second, (int)h.pair_rows.size(), 0});
        ClrPairSet &set = h.pair_sets.back();
        for (const Row &r : rows)
            for (const std::vector<float4> &part : clr_parts(r.b, 6)) {   // tighter balls around fewer spheres
                h.pair_rows.push_back(ClrPairRow{r.a, clr_ball(part), (int)h.pair_spheres.size(), (int)part.size(), {0, 0}});
                h.pair_spheres.insert(h.pair_spheres.end(), part.begin(), part.end());
            }
        set.n = (int)h.pair_rows.size() - set.first;
    }
}

template <int NJ, int NS, int NL, int NP>
inline ClrHostModel make_clr_model(int dof, const prrtc_joint_def (&J)[NJ], const prrtc_sphere_def (&S)[NS],
                                   const short (&L)[NL], const short (&P)[NP][2], int num_pairs)
{
    ClrHostModel h;
    h.dof = dof;
    int pos_of_q[kClrMaxJoints] = {};
    for (int j = 0; j < NJ; j++) pos_of_q[J[j].q] = j;
    auto pos = [&](int q) { return q < 0 ? -1 : pos_of_q[q]; };
    for (int j = 0; j < NJ; j++) {
        h.joints.push_back(J[j]);
        h.parent.push_back(pos(J[j].parent));
    }
    for (int i = 0; i < NL; i++) {
        const prrtc_sphere_def &s = S[L[i]];
        h.leaf.push_back(make_float4(s.x, s.y, s.z, s.r));
        h.leaf_joint.push_back(pos(s.frame));
    }
    for (int i = 0; i < num_pairs; i++) {
        const prrtc_sphere_def &a = S[P[i][0]], &b = S[P[i][1]];
        h.pa.push_back(make_float4(a.x, a.y, a.z, a.r));
        h.pb.push_back(make_float4(b.x, b.y, b.z, b.r));
        h.pair_joint.push_back(make_int2(pos(a.frame), pos(b.frame)));
    }
    clr_sets(h);
    return h;
}

#define PRRTC_CLR_MODEL(R) \
    make_clr_model(k##R##Dof, k##R##Joints, k##R##Spheres, k##R##EnvLeaves, k##R##SelfPairs, k##R##NumSelfPairs)

inline const ClrHostModel &clr_host_model(prrtc_robot r)
{
    static const ClrHostModel m[4] = {PRRTC_CLR_MODEL(Sphere), PRRTC_CLR_MODEL(Panda), PRRTC_CLR_MODEL(Fetch),
                                      PRRTC_CLR_MODEL(Baxter)};
    return m[(int)r];
}

}  // namespace prrtc
