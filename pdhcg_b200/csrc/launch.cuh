// launch.cuh -- what the device units share on the host side: error checks,
// grid sizes, the cone blocks' launch classes, and the launchers of the heavy
// kernel templates, each of which is instantiated in one unit (steps.cu,
// residual.cu, inner.cu, project.cu) so that the units compile side by side.
#pragma once

#include <algorithm>
#include <mutex>
#include <stdexcept>
#include <string>
#include <type_traits>
#include <unordered_map>
#include <vector>

#include "bb.cuh"
#include "gridsum.cuh"
#include "internal.h"
#include "resident.cuh"
#include "residual.cuh"

namespace pdhcg {

struct CudaError : std::runtime_error {
    using std::runtime_error::runtime_error;
};

#define CK(call)                                                                                                       \
    do {                                                                                                               \
        cudaError_t e_ = (call);                                                                                       \
        if (e_ != cudaSuccess)                                                                                         \
            throw CudaError(std::string(#call) + ": " + cudaGetErrorString(e_) + " at " + __FILE__ + ":" +            \
                            std::to_string(__LINE__));                                                                 \
    } while (0)

inline int grid_for(long long work, int per_block, int cap = 148 * 16)
{
    long long g = (work + per_block - 1) / per_block;
    if (g < 1)
        g = 1;
    if (g > cap)
        g = cap;
    return (int)g;
}

// Lets `kernel` be launched with up to `bytes` of dynamic shared memory.  The
// limit is state of the kernel on the device, shared by every thread that
// solves: all callers pass one constant per kernel, the most that any of its
// launches takes, so that no caller lowers it under another's launch.
template <typename K>
void allow_shared(K kernel, size_t bytes)
{
    CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
}

// Blocks of `kernel` (TPB threads, static shared memory) resident at once
// on the current device; cached per kernel and device.
inline int resident_blocks(const void *kernel)
{
    static std::mutex mu;
    static std::unordered_map<const void *, int> cache[64];
    int dev = 0;
    CK(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    auto &c = cache[dev & 63];
    auto it = c.find(kernel);
    if (it != c.end())
        return it->second;
    int nsm = 0, per_sm = 0;
    CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, TPB, 0));
    const int r = std::max(1, nsm * std::max(per_sm, 1));
    c.emplace(kernel, r);
    return r;
}

// The primal step launches the SOC / RSOC blocks and the 3-slot blocks
// (exponential, power) separately: the 3-slot projections would otherwise
// sit in the wide kernels' register allocation.  A list pointer stays null
// when its launch covers every block (all of one kind).
struct ConeSplit {
    std::vector<int> wide, three, psd, sect;
    int *wide_d = nullptr, *three_d = nullptr, *psd_d = nullptr, *sect_d = nullptr;
    int n_wide = 0, n_three = 0, n_psd = 0, n_sect = 0;

    // fixed (may be empty): per block, does it hold slots fixed by
    // set_cone_fixed?  Those blocks take the section projectors.
    void build(const std::vector<int> &types, const std::vector<char> &fixed = {})
    {
        wide.clear();
        three.clear();
        psd.clear();
        sect.clear();
        for (int b = 0; b < (int)types.size(); ++b) {
            if (!fixed.empty() && fixed[b])
                sect.push_back(b);
            else if (types[b] == CONE_EXPONENTIAL || types[b] == CONE_POWER)
                three.push_back(b);
            else if (types[b] == CONE_PSD)
                psd.push_back(b);
            else
                wide.push_back(b);
        }
        n_wide = (int)wide.size();
        n_three = (int)three.size();
        n_psd = (int)psd.size();
        n_sect = (int)sect.size();
    }
    // more than one launch: every launch takes its index list
    bool mixed() const { return (n_wide > 0) + (n_three > 0) + (n_psd > 0) + (n_sect > 0) > 1; }
    // the lists back to back in one device array of n_wide + n_three + n_psd + n_sect ints
    void place(int *ids)
    {
        wide_d = ids;
        three_d = ids + n_wide;
        psd_d = ids + n_wide + n_three;
        sect_d = ids + n_wide + n_three + n_psd;
    }
    std::vector<int> joined() const
    {
        std::vector<int> all(wide);
        all.insert(all.end(), three.begin(), three.end());
        all.insert(all.end(), psd.begin(), psd.end());
        all.insert(all.end(), sect.begin(), sect.end());
        return all;
    }
};

template <typename F>
void dispatch_s(int S, F &&f)
{
    switch (S) {
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    default: f(std::integral_constant<int, 8>{}); break;
    }
}

template <typename F>
void dispatch_rg(int G, F &&f)
{
    switch (G) {
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    default: f(std::integral_constant<int, 32>{}); break;
    }
}

// steps.cu: the kernels of one step
template <typename T>
void launch_primal_free(const StepData<T> &D, const StepParams &P, bool hasq, bool box_free, int grid, cudaStream_t s);
// cone blocks of the primal step; returns the number of launches
template <typename T>
int launch_primal_cones(const StepData<T> &D, const StepParams &P, const ConeSplit &sp, int S, bool hasq, bool mixed,
                        cudaStream_t s);
// free variables, SOC / RSOC and 3-slot blocks in one launch; false: not for
// this problem
template <typename T>
bool launch_primal_mixed(const StepData<T> &D, const StepParams &P, const ConeSplit &sp, int S, bool hasq,
                         cudaStream_t s);
template <typename T>
void launch_dual_cones(const StepData<T> &D, const StepParams &P, int S, cudaStream_t s);
template <typename T>
void launch_dual_rows(const StepData<T> &D, const StepParams &P, bool eq_rows, bool has_g, int grid, cudaStream_t s);

// residual.cu
template <typename VT>
void launch_residual(const ResidualData<VT> &D, const ResidualParams &P, int S, bool fixed, int blocks,
                     cudaStream_t s);

// the variables' PSD blocks of the residual, a thread block each, partials
// from row `first` on; fits: whether a block of this order fits in one's shared
// memory
bool residual_psd_fits(int order);
template <typename VT>
void launch_residual_psd(const ResidualData<VT> &D, const ResidualParams &P, const int *ids, int nids, int max_order,
                         int first, int blocks, cudaStream_t s);

// inner.cu: the inner BB solve and the Q apply (G lanes per row of Q, S
// slots per lane of a cone block; one_per_sm: the form for a grid of one block
// per SM)
int bb_blocks_per_sm(int G, int S, bool fixed, bool one_per_sm); // resident blocks of both kernels
void launch_bb(int G, int S, bool fixed, bool one_per_sm, int grid, const BBData &D, const BBParams &P, cudaStream_t s);
void launch_q_apply(int G, int grid, const BBData &D, const double *v, double *qx, cudaStream_t s);

// inner_small.cu: sparse Q with short rows, no cones; blocks: 0 when Q does
// not fit the blocks' shared memory
struct SmallPlan {
    const void *kernel;
    int blocks, threads, cap; // cap: entries of Q that a block has room for
    bool cluster;
};
SmallPlan bb_small_plan(int n, long long nnz, const int *Q_rp, int sms, int *shares, cudaStream_t s);
void launch_bb_small(const SmallPlan &p, const BBData &D, const BBParams &P, const GridSlots &S, cudaStream_t s);

// inner_dense.cu: dense R, diagonal Q; blocks: 0 when the shape does not fit
int dense_tile_count(int width);
int dense_blocks(int k, int tiles, int S, int sms);
void dense_tiles(int k, int width, const int *rp, const double *v, int tiles, double *d, float *f, cudaStream_t s);
void dense_qdiag(int n, const int *rp, const int *ci, const double *v, double *qd, int *bad, cudaStream_t s);
void launch_bb_dense(int S, bool fp32, int blocks, const BBData &D, const BBParams &P, const DenseR &R,
                     const GridSlots &G, cudaStream_t s);

// resident.cu: persistent iterations of a problem without cones
struct ResidentPlan {
    int blocks; // 0: not for this shape
    int cap_a, cap_at, rows, vars; // per block: staged entries of A and A^T, rows, variables
    size_t smem;
};
ResidentPlan resident_plan(int n, int m, long long nnz, const int *A_rp, const int *At_rp, int sms, int *shares,
                           cudaStream_t s);
void launch_resident(const ResidentPlan &p, const ResidentData &D, const ResidentParams &P, const GridSlots &S,
                     cudaStream_t s);

// project.cu
struct ProjectArgs {
    int ncones;
    const int *start, *len, *type;
    const double *alpha;
    double *x;
    const double *d, *q;
    double tau;
    double *psd_work;
    const long long *psd_off;
    const unsigned char *fixed, *cone_fixed;
    double *warm;
};
void launch_project_cones(int S, const ProjectArgs &a, cudaStream_t s);
void launch_project_sections(int S, const ProjectArgs &a, cudaStream_t s); // every block a section block

} // namespace pdhcg
