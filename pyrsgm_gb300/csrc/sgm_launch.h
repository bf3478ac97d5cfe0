// sgm_launch.h -- host-side launch interface of the pyrsgm-gb300 kernels.
//
// Every stage is launched for a batch of independent level jobs (one stereo
// pair's level each); a single-pair call is a batch of one.  Job
// descriptors travel by value in the kernel parameter block, so a launch
// needs no host-to-device copy and can be captured in a CUDA graph.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "check.h"
#include "sgm_common.cuh"

namespace pg {

constexpr int kBatchJobs = 64;  // level jobs per batched launch
constexpr int kBatchPyr = 32;   // pyrDown images per batched launch

struct PyrDownDesc {
    const uint8_t* src;
    uint8_t* dst;
    int sstep, sw, sh, dstep, dw, dh;
};

template <int NB>
struct PyrDownBatch {
    PyrDownDesc d[NB];
    int n;
};

// Largest extents over the jobs of one launch (grid sizing).
struct LevelExtent {
    int max_w = 0, max_h = 0, max_D = 0;
    long long max_vox = 0;
    bool any_refine = false;
};

template <int NJ>
LevelExtent extent_of(const Jobs<NJ>& j)
{
    LevelExtent e;
    for (int i = 0; i < j.n; ++i) {
        const LevelDesc& d = j.d[i];
        e.max_w = std::max(e.max_w, d.w);
        e.max_h = std::max(e.max_h, d.h);
        e.max_D = std::max(e.max_D, d.D);
        e.max_vox = std::max(e.max_vox, (long long)d.w * d.h * d.D);
        e.any_refine = e.any_refine || d.refine;
    }
    return e;
}

// Sums over the jobs of a launch (algorithmic-byte accounting).
template <int NJ>
double jobs_px(const Jobs<NJ>& j)
{
    double s = 0;
    for (int i = 0; i < j.n; ++i) s += (double)j.d[i].w * j.d[i].h;
    return s;
}
template <int NJ>
double jobs_vox(const Jobs<NJ>& j)
{
    double s = 0;
    for (int i = 0; i < j.n; ++i) s += (double)j.d[i].w * j.d[i].h * j.d[i].D;
    return s;
}

// Kernel family of a label count: 10000 + D for 16, 32 and 64 labels, which
// keep a volume per path, else the labels a chain of the one-volume kernels
// holds (64, 128, 256, 512, 1024).  Jobs of one aggregation launch share it.
inline int path_variant(int D)
{
    if (uses_packed(D)) return 10000 + D;
    int cap = 64;
    while (cap < D) cap *= 2;
    return cap;
}

// Multiprocessor count of the current device (cached per device).
int sm_count();

// 0 (choose per launch), 8, or 2/4: the packed kernels' words per thread.
int packed_words_override();
// Warps per SM the wide shape must fill before a launch takes it by itself
// (INT_MAX: it is taken only when forced or measured faster).
int packed_min_warps_per_sm();
// 1: fused two-pass form of the 16-label pyramid levels (opt-in).
int fused_mode();
// T->B pass with the winner-take-all for those levels: 0 never, 1 when a
// launch fills the GPU (default), 2 always.
int tbw_mode();

// Measuring shape choice for the 16/32/64-label aggregation (opt-in,
// pyrsgm_gb300_set_autotune).  A launch is keyed by its label count, mode,
// total rows and widest level; while the calling thread is in a tuning
// scope (the batch engine's first, uncaptured run of a new batch) a key
// without an entry times both kernel shapes on the launch stream (twice
// each, host-synchronising; the outputs of either are identical) and keeps
// the faster.  Outside a tuning scope a recorded entry is used and an
// unknown key falls back to the rule of packed_nw().
struct TuneKey {
    int D, pyr, rows, w;
    bool operator<(const TuneKey& o) const
    {
        return D != o.D ? D < o.D : pyr != o.pyr ? pyr < o.pyr : rows != o.rows ? rows < o.rows : w < o.w;
    }
};
struct TuneEntry {
    int nw;              // chosen words per thread
    float ms_wide;       // NW = 8 shape, best of two
    float ms_spread;     // segmented shape, best of two
};
bool autotune_enabled();
bool tuning_thread();
// RAII: marks the calling thread as allowed to measure.
struct TuningScope {
    TuningScope();
    ~TuningScope();
    bool prev;
};
bool tune_lookup(const TuneKey& k, TuneEntry& out);
void tune_store(const TuneKey& k, const TuneEntry& e);

// Launch a kernel that begins with after_previous() (sgm_common.cuh): its
// blocks may become resident while the previous kernel of the stream
// finishes.  Every kernel waits for the whole one before it, so the order of
// the stream is kept.  Hides the launch and the start of the blocks, 1 to 2
// us a kernel (160x96 level, five kernels: 34 -> 28 us a call).  The launch
// error is left for cudaGetLastError().
template <class T>
struct LaunchArg {
    using type = T;
};
template <class... P>
void launch_after(void (*kernel)(P...), dim3 grid, int block, size_t smem, cudaStream_t st,
                  const typename LaunchArg<P>::type&... args)
{
    cudaLaunchAttribute a;
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &a;
    c.numAttrs = 1;
    void* p[] = {const_cast<void*>(static_cast<const void*>(&args))...};
    cudaLaunchKernelExC(&c, reinterpret_cast<const void*>(kernel), p);
}

// Dynamic shared memory of kernels whose launches need different amounts.
// The limit set here belongs to the kernel on the device, not to the thread
// or the launch: set to what each launch needs, a second thread could lower
// it between the set and the launch of the first.  So every launch sets the
// same, the most a block can have (such a kernel has no static shared
// memory); what a launch takes is its own argument still.
constexpr int kSmemPerBlock = 227 * 1024;
template <class... P>
cudaError_t allow_smem(void (*kernel)(P...))
{
    return cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                kSmemPerBlock);
}

// Count of kernel launches issued by this library (process-wide); a CUDA
// graph replay counts the kernels it contains.
void count_launch();
void count_launches(unsigned long long n);
unsigned long long launch_count();

template <int NB>
cudaError_t launch_pyrdown(const PyrDownBatch<NB>& b, int max_dw, int max_dh, cudaStream_t st);
cudaError_t launch_p2_table(int* lut, int P2, float alpha, float beta, float lower, float upper,
                            cudaStream_t st);
template <int NJ>
cudaError_t launch_prepare(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st);
template <int NJ>
cudaError_t launch_cost(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st);
// All jobs in one call share pyr (mode) and the path shape of their D.
template <int NJ>
cudaError_t launch_paths(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st);
// Paths, winner and LR check of one level with a penalty below zero
// (k_paths_signed.cu); the post pass is left without the check.
cudaError_t launch_paths_signed(const LevelDesc& d, cudaStream_t st);
template <int NJ>
cudaError_t launch_post(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st);

}  // namespace pg
