// k_paths.cuh -- choice and launch of the path-aggregation kernels of a
// level.
//
// Reference semantics (reference file:line):
//   single-scale  kernel_SGM_PathLR / PathTB / PathRL_WTA, src/sgm_kernels.cu:520-819
//   pyramid       kernel_SGM_PathLRPyramid / TBPyramid / RLPyramidWTA,
//                 src/sgm_kernels.cu:1191-1478
//
// The reference's clamped sums are order independent -- every term is
// non-negative and is clamped at one cap (SHRT_MAX single-scale; SHRT_MAX-1
// with a SHRT_MAX sentinel in the pyramid) -- so the totals equal its L->R,
// T->B, R->L accumulation in whatever order the paths are added.
//
// disp2 in the reference is written right to left and keeps the first
// strictly smaller cost, i.e. for every target column the minimum cost with
// ties going to the largest source column.  Here every candidate does
// atomicMin on (cost << 16 | (0xFFFF - x)), which selects the same winner
// independent of the visiting order; the LR check reads the keys in the post
// kernel.
#pragma once

#include <algorithm>
#include <climits>

#include "profiler.h"
#include "sgm_common.cuh"
#include "sgm_launch.h"
#include "k_paths_packed.cuh"
#include "k_paths_seg.cuh"
#include "k_wta_group.cuh"
#include "k_fused.cuh"

namespace pg {

// Winner-take-all of the packed levels: a thread per pixel with 16 and 32
// labels, four lanes with 64.
template <int D, bool PYR, int NJ>
cudaError_t launch_wta(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st)
{
    dim3 gw((e.max_w + 31) / 32, (e.max_h + 7) / 8, jobs.n);
    prof_begin(st);
    if constexpr (D <= 32) launch_after(k_wta<D, PYR, NJ>, gw, 256, 0, st, jobs);
    else launch_after(k_wta_group<D / 16, 1, 3, PYR, NJ>, gw, 256, 0, st, jobs);
    count_launch();
    prof_end(PK_WTA, jobs_vox(jobs) * 2 * (jobs.d[0].paths >= 3 ? 3 : jobs.d[0].paths) + jobs_px(jobs) * (2 + 6 + 4), st);
    return launched(st, "k_wta");
}

// The wide shape: one thread per 16 labels.
template <int T, bool PYR, int NJ>
cudaError_t launch_paths_wide(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st)
{
    constexpr int NW = 8;
    using G = pk::Grp<NW, T>;
    cudaError_t err;
    bool any_tb = false;
    for (int i = 0; i < jobs.n; ++i) any_tb = any_tb || jobs.d[i].paths >= 3;
    // T->B and the horizontal paths run one after the other: launches of
    // this shape fill the GPU, side by side they would only contend.
    // 16-label pyramid levels, wide shape, three paths everywhere, and
    // columns for at least kTbwMinWarpsPerSm warps per SM: the row pass
    // first, then T->B with the winner-take-all (k_gtbw).  Its serial chain
    // step carries the winner's work, so with few warps per SM it loses to
    // k_gtb + k_wta: per launch, 16 pairs of 1080p, 1165 against 1031 us
    // at 6.3 warps per SM and 467 against 308 us at 3.2; at 12.6 warps per
    // SM (32 pairs) it is about 15 % faster.
    bool tbw = false;
    if constexpr (PYR && T == 1) {
        long long cols = 0;
        tbw = tbw_mode() != 0;
        for (int i = 0; i < jobs.n; ++i) {
            tbw = tbw && jobs.d[i].paths >= 3;
            cols += jobs.d[i].w;
        }
        tbw = tbw && (tbw_mode() == 2 || cols >= 32LL * pk::kTbwMinWarpsPerSm * sm_count());
    }
    if (tbw) any_tb = false;
    if (any_tb) {
        Jobs<NJ> tbj = jobs;
        int n = 0;
        for (int i = 0; i < jobs.n; ++i)
            if (jobs.d[i].paths >= 3) tbj.d[n++] = jobs.d[i];
        tbj.n = n;
        constexpr size_t smem = pk::tb_smem<NW, T>();
        if ((err = cudaFuncSetAttribute(k_gtb<NW, T, PYR, NJ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)smem)) != cudaSuccess)
            return err;
        constexpr int kWarps = pk::kPackedWarps;
        const int cols = kWarps * G::CPW;
        dim3 g((e.max_w + cols - 1) / cols, n);
        prof_begin(st);
        launch_after(k_gtb<NW, T, PYR, NJ>, g, kWarps * 32, smem, st, tbj);
        count_launch();
        prof_end(PK_PATH_TB, jobs_vox(tbj) * 4 + jobs_px(tbj) * ((tbj.d[0].refine ? 2 : 0) + (tbj.d[0].adaptive ? 1 : 0)), st);
        if ((err = launched(st, "k_gtb")) != cudaSuccess) return err;
    }
    constexpr int kWarps = pk::kPackedWarps;
    const int rows = kWarps * G::CPW / 2;
    dim3 g((e.max_h + rows - 1) / rows, jobs.n);
    constexpr size_t smem = pk::row_smem<NW, T>();
    if ((err = cudaFuncSetAttribute(k_grow<NW, T, PYR, NJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) !=
        cudaSuccess)
        return err;
    prof_begin(st);
    launch_after(k_grow<NW, T, PYR, NJ>, g, kWarps * 32, smem, st, jobs);
    count_launch();
    if (prof_enabled()) {
        // algorithmic bytes: each horizontal path reads the cost volume and
        // writes its costs once
        double by = 0;
        for (int i = 0; i < jobs.n; ++i) {
            const LevelDesc& d = jobs.d[i];
            const double px = (double)d.w * d.h;
            by += px * d.D * 2 * (d.paths >= 2 ? 4 : 2) + px * 2 * ((d.refine ? 2 : 0) + (d.adaptive ? 1 : 0));
        }
        prof_end(PK_PATH_ROW, by, st);
    }
    if ((err = launched(st, "k_grow")) != cudaSuccess) return err;
    if constexpr (PYR && T == 1) {
        if (tbw) {
            constexpr size_t smem = pk::tbw_smem();
            if ((err = cudaFuncSetAttribute(k_gtbw<NJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) !=
                cudaSuccess)
                return err;
            dim3 gt((e.max_w + 127) / 128, jobs.n);
            prof_begin(st);
            launch_after(k_gtbw<NJ>, gt, 128, smem, st, jobs);
            count_launch();
            prof_end(PK_TBW, jobs_vox(jobs) * 6 + jobs_px(jobs) * ((jobs.d[0].refine ? 2 : 0) + (jobs.d[0].adaptive ? 1 : 0) + 10),
                     st);
            return launched(st, "k_gtbw");
        }
    }
    return launch_wta<G::D, PYR, NJ>(jobs, e, st);
}

// The segmented shape: every chain cut into segments that run at the same
// time, rows and columns in one launch.
template <int NW, int T, bool PYR, int NJ>
cudaError_t launch_paths_seg(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st)
{
    const cudaError_t err = launch_seg<NW, T, PYR, NJ>(jobs, true, st);
    return err != cudaSuccess ? err : launch_wta<2 * NW * T, PYR, NJ>(jobs, e, st);
}

// 16 labels: four threads a chain while the launch has at most three such
// groups of 8 chains per SM -- the step is shorter, and the lone walks that
// follow the first ones with it (us, two threads against four: 480x270 34
// and 24, 960x540 52 and 41, 1440x994 92 and 79) --, else two, which take
// fewer instructions (1080p 86 and 95, 2879x1987 213 and 250).
template <bool PYR, int NJ>
cudaError_t launch_paths_seg16(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st)
{
    long long chains = 0;
    for (int i = 0; i < jobs.n; ++i) chains += 2 * jobs.d[i].h + (jobs.d[i].paths >= 3 ? jobs.d[i].w : 0);
    return chains <= 3LL * 8 * sm_count() ? launch_paths_seg<2, 4, PYR, NJ>(jobs, e, st)
                                          : launch_paths_seg<4, 2, PYR, NJ>(jobs, e, st);
}

// Shape of the packed kernels for a launch: 2 (4 for 64 labels), the
// segmented shape, or 8, the wide one (one thread per 16 labels, whole
// chains).  With five segments a chain the segmented shape is the faster for
// every batch of textured pairs measured (us, wide against segmented, 1080p:
// 2 pairs 2310 and 771, 8 3298 and 2324, 32 9127 and 8345, 64 17177 and 16401;
// 64 VGA pairs of 64 labels 4042 and 3335), and without texture, where its
// batches walk whole chains too (k_seg), within 4 % of the wide one (32
// pairs: gradients 8690 and 8761, 8605 and 8716, one grey value 7164 and
// 7430).  So the wide one is taken only where packed_words_override() (set
// through pyrsgm_gb300_set_packed_words), the autotuner or
// PYRSGM_GB300_PACKED_WPS asks for it.
inline int packed_nw(int D, long long rows)
{
    const int force = packed_words_override();
    const int small = D == 64 ? 4 : 2;
    if (force == 8) return 8;
    if (force == 2 || force == 4) return small;
    const long long warps8 = rows * 2 * (D / 16) / 32;
    return warps8 >= (long long)packed_min_warps_per_sm() * sm_count() ? 8 : small;
}

// Words per thread for a packed launch: a forced setting, else a recorded
// measurement for its key, else (measuring it now when the thread is in a
// tuning scope) the rule of packed_nw().  `run(nw)` launches one shape.
template <class Run>
int packed_choice(const TuneKey& key, long long rows, cudaStream_t st, Run run, cudaError_t& err)
{
    err = cudaSuccess;
    if (packed_words_override() != 0 || !autotune_enabled()) return packed_nw(key.D, rows);
    TuneEntry te;
    if (tune_lookup(key, te)) return te.nw;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (!tuning_thread() || cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone)
        return packed_nw(key.D, rows);
    const int spread = key.D == 64 ? 4 : 2;
    float best[2] = {1e30f, 1e30f};
    cudaEvent_t a = nullptr, b = nullptr;
    if ((err = cudaEventCreate(&a)) != cudaSuccess || (err = cudaEventCreate(&b)) != cudaSuccess) {
        if (a) cudaEventDestroy(a);
        return packed_nw(key.D, rows);
    }
    for (int rep = 0; rep < 2 && err == cudaSuccess; ++rep) {
        for (int c = 0; c < 2 && err == cudaSuccess; ++c) {
            float ms = 0.0f;
            if ((err = cudaEventRecord(a, st)) != cudaSuccess || (err = run(c == 0 ? 8 : spread)) != cudaSuccess ||
                (err = cudaEventRecord(b, st)) != cudaSuccess || (err = cudaEventSynchronize(b)) != cudaSuccess ||
                (err = cudaEventElapsedTime(&ms, a, b)) != cudaSuccess)
                break;
            best[c] = std::min(best[c], ms);
        }
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    if (err != cudaSuccess) return packed_nw(key.D, rows);
    te.nw = best[0] <= best[1] ? 8 : spread;
    te.ms_wide = best[0];
    te.ms_spread = best[1];
    tune_store(key, te);
    return te.nw;
}

// k_paths_sum.cuh, compiled apart.
template <bool PYR, int NJ>
cudaError_t launch_paths_sum(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st);

template <bool PYR, int NJ>
cudaError_t launch_paths_mode(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st)
{
    long long rows = 0;
    for (int i = 0; i < jobs.n; ++i) rows += jobs.d[i].h;
    const int D = jobs.d[0].D;
    // 16-label pyramid levels with all three paths: the wide shape is the
    // fused T->B + L->R and R->L + WTA passes (k_fused.cuh)
    bool fused = false;
    if constexpr (PYR) fused = D == 16 && fused_mode() != 0 && fused_applicable(jobs);
    const TuneKey key{D, PYR ? (fused ? 2 : D == 16 && tbw_mode() ? 3 : 1) : 0, (int)std::min<long long>(rows, INT_MAX), e.max_w};
    cudaError_t err = cudaSuccess;
    switch (path_variant(D)) {
    case 10016: {
        auto run = [&](int nw) {
            if constexpr (PYR) {
                if (nw == 8 && fused) return launch_paths_fused16<NJ>(jobs, e, st);
            }
            return nw == 8 ? launch_paths_wide<1, PYR, NJ>(jobs, e, st)
                           : launch_paths_seg16<PYR, NJ>(jobs, e, st);
        };
        const int nw = packed_choice(key, rows, st, run, err);
        return err != cudaSuccess ? err : run(nw);
    }
    case 10032: {
        auto run = [&](int nw) {
            return nw == 8 ? launch_paths_wide<2, PYR, NJ>(jobs, e, st)
                           : launch_paths_seg<4, 4, PYR, NJ>(jobs, e, st);
        };
        const int nw = packed_choice(key, rows, st, run, err);
        return err != cudaSuccess ? err : run(nw);
    }
    case 10064: {
        auto run = [&](int nw) {
            return nw == 8 ? launch_paths_wide<4, PYR, NJ>(jobs, e, st)
                           : launch_paths_seg<4, 8, PYR, NJ>(jobs, e, st);
        };
        const int nw = packed_choice(key, rows, st, run, err);
        return err != cudaSuccess ? err : run(nw);
    }
    default: return launch_paths_sum<PYR, NJ>(jobs, e, st);   // one path volume
    }
}

}  // namespace pg
