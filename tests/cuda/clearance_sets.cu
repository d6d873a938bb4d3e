// The clearance's four-lane evaluation (clearance_eval.cuh) on Panda's model
// with its leaves cut into sets of at most `most`, so that a model can have
// more sets than a word has bits.  Host arrays in and out, no grid.
#include <vector>

#include "clearance_model.h"
#include "device_common.cuh"
#include "robots/panda_fkcc.cuh"
#include "robot_kernels.cuh"

PRRTC_GEN_ADAPTER(GenPanda, gen_panda)

using namespace prrtc;

namespace {
struct Device {   // everything copied to the device for one call
    std::vector<void *> all;
    cudaError_t e = cudaSuccess;
    template <class T>
    T *put(const T *host, size_t n)
    {
        void *p = nullptr;
        if (e == cudaSuccess) e = cudaMalloc(&p, n * sizeof(T) + 16);
        if (e == cudaSuccess) all.push_back(p);
        if (e == cudaSuccess && host) e = cudaMemcpy(p, host, n * sizeof(T), cudaMemcpyHostToDevice);
        return static_cast<T *>(p);
    }
    template <class T>
    const T *put(const std::vector<T> &v) { return put(v.data(), v.size()); }
    ~Device()
    {
        for (void *p : all) cudaFree(p);
    }
};
}  // namespace

// number of leaf sets, or -1 with a CUDA error
extern "C" int clearance_with_sets(const float *rec, int ns, int nc, int nzc, int ncb, int nzb, const float *q, int rows,
                                   float margin, int most, float *cost, float *grad)
{
    ClrHostModel h = clr_host_model(PRRTC_ROBOT_PANDA);
    std::vector<ClrLeafSet> sets;
    for (const ClrLeafSet &s : h.leaf_sets)
        for (int i = 0; i < s.n; i += most) {
            const int n = std::min(most, s.n - i);
            const std::vector<float4> part(h.set_leaves.begin() + s.first + i, h.set_leaves.begin() + s.first + i + n);
            sets.push_back(ClrLeafSet{clr_ball(part), s.joint, s.first + i, n, 0});
        }
    Device D;
    ClrModel M{};
    M.dof = h.dof;
    M.nj = (int)h.joints.size();
    M.n_leaf = (int)h.leaf.size();
    M.n_pair = (int)h.pa.size();
    M.joints = D.put(h.joints);
    M.joint_parent = D.put(h.parent);
    M.leaf = D.put(h.leaf);
    M.leaf_joint = D.put(h.leaf_joint);
    M.pair_a = D.put(h.pa);
    M.pair_b = D.put(h.pb);
    M.pair_joint = D.put(h.pair_joint);
    M.n_leaf_sets = (int)sets.size();
    M.n_pair_sets = (int)h.pair_sets.size();
    M.chain = D.put(h.chain);
    M.leaf_sets = D.put(sets);
    M.set_leaves = D.put(h.set_leaves);
    M.pair_sets = D.put(h.pair_sets);
    M.pair_rows = D.put(h.pair_rows);
    M.pair_spheres = D.put(h.pair_spheres);
    const EnvCounts n{ns, nc, nzc, ncb, nzb};
    const ClrEnv env{D.put(reinterpret_cast<const float4 *>(rec), (size_t)n.records()), n, nullptr};
    const ClrEnv *envs = D.put(&env, 1);
    const float *dq = D.put(q, (size_t)rows * h.dof);
    float *dc = D.put<float>(nullptr, rows), *dg = D.put<float>(nullptr, (size_t)rows * h.dof);
    if (D.e != cudaSuccess) return -1;
    k_path_cost_grad<GenPanda><<<(rows + 15) / 16, 64>>>(M, envs, rows, rows, dq, margin, dc, dg);
    if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess ||
        cudaMemcpy(cost, dc, rows * sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(grad, dg, (size_t)rows * h.dof * sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess)
        return -1;
    return (int)sets.size();
}
