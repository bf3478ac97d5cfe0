// k_paths_sum.cuh -- aggregation of the label counts that keep one path
// volume (every multiple of 16 but 16, 32 and 64, up to 1024): the columns
// write V (segmented, k_paths_seg.cuh), the rows of both directions add to
// it, and the winner is read from it.  One volume and the costs are all the
// memory such a level has; all of it moves 18 bytes per label (columns 4, rows
// 12, winner 2).
#pragma once

#include "k_paths_seg.cuh"
#include "k_wta_group.cuh"

namespace pg {

// Rows of both directions added to V, for the label counts that keep one
// path volume (every one but 16, 32 and 64): a warp a direction, a block the
// two of 32 / T rows.  Each direction comes first to half of the columns;
// after a barrier it adds to what the other one left in the rest.  12 bytes
// per label move (the costs, V in and out, for each direction).  Bound by
// the latency of a step (641x479 with 96 labels: 81 us, 148 ns a step; 89
// with both directions in one warp, 16 lanes each, which met in the middle
// and read V again there; 1316 on scalar chains with the winner inside) and,
// from 128 labels on, by memory (720p: 184 us, 193 and 2965).
template <int NW, int T, int MODE, int NJ>
__global__ void __launch_bounds__(64) k_rowadd(const __grid_constant__ Jobs<NJ> jobs)
{
    using namespace sg;
    using G = Geo<NW, T>;
    const LevelDesc& J = jobs.d[blockIdx.y];
    extern __shared__ __align__(16) uint32_t smem[];
    const int lane = threadIdx.x & 31, dir = threadIdx.x >> 5, row0 = blockIdx.x * G::CPW;
    if (row0 >= J.h) {
        after_previous();
        return;
    }
    const Extent<MODE> e(J);
    int* lut = reinterpret_cast<int*>(smem);
    uint32_t* mine = smem + 256 + dir * warp_words<NW, T, MODE>(2);
    for (int i = lane; i < warp_words<NW, T, MODE>(2); i += 32) mine[i] = kMax2;
    let_next_in();
    after_previous();
    const bool guard = __syncthreads_or(load_penalties(J, lut));
    const int k = lane % T;
    Ctx<NW, T, MODE> X{J, lut, mine, mine + 2 * kSC * G::SLOTW + lane / T + NW * k * G::WST, nullptr, lane, lane / T, k,
                       e, true, J.adaptive != 0, guard, 2 * row0 + dir, {}, J.V, pk::dup(imin(J.P1, 0x8000))};
    X.w = walk_of<MODE>(J, e, true, 2 * (row0 + X.c) + dir);
    // L->R comes first to the first `half` columns of its walk, R->L to the
    // others.  Both first parts end on whole chunks: R->L starts `pad` steps
    // early.
    const int half = imin(e.lr_n, e.rl_n / 2) / kCH * kCH;
    const int pad = dir ? (kCH - e.rl_n % kCH) % kCH : 0;
    const int n = dir ? e.rl_n : e.lr_n, mid = dir ? e.rl_n - half : half;
    const bool on = X.w.n > 0;
    State<NW, T> s;
    uint32_t spec[NW];
#pragma unroll
    for (int i = 0; i < NW; ++i) s.L[i] = spec[i] = kMax2;
    s.mp2 = kMax2;
#pragma unroll 1
    for (int part = 0; part < 2; ++part) {
        const int t0 = part ? mid : -pad;
        X.stop = part ? n : mid;
        X.sums = J.paths >= 3 || part;
        const int nch = (X.stop - t0 + kCH - 1) / kCH;
        seg_walk<NW, T, MODE, kAdd>(X, s, t0, imax(t0, 0), on ? X.stop : -(1 << 30), nch, 1, 0, 0, true, spec);
        __syncthreads();   // what the other direction has left
    }
}

template <int NW, int T, int MODE, int NJ>
cudaError_t launch_rowadd_mode(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st)
{
    using G = sg::Geo<NW, T>;
    constexpr size_t smem = sg::add_smem<NW, T, MODE>();
    const cudaError_t err =
        cudaFuncSetAttribute(k_rowadd<NW, T, MODE, NJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    prof_begin(st);
    launch_after(k_rowadd<NW, T, MODE, NJ>, dim3((e.max_h + G::CPW - 1) / G::CPW, jobs.n), 64, smem, st, jobs);
    count_launch();
    if (prof_enabled()) {
        // each direction reads the cost volume; V is read (T->B or the first
        // direction's sum) and written once per direction
        double by = 0;
        for (int i = 0; i < jobs.n; ++i) {
            const LevelDesc& d = jobs.d[i];
            const int dirs = d.paths >= 2 ? 2 : 1;
            by += (double)d.w * d.h * (d.D * (4.0 * dirs + 2.0 * (dirs - 1) + (d.paths >= 3 ? 2 : 0)) +
                                       dirs * ((d.refine ? 2 : 0) + (d.adaptive ? 1 : 0)));
        }
        prof_end(PK_PATH_ROW, by, st);
    }
    return launched(st, "k_rowadd");
}

// Columns into V, rows added to it, the winner from it.  On rows of fixed
// labels a chain takes twice the threads, of half the words, up to a whole
// warp (RNW, RT): their warps are few and wait for each step (720p Census,
// 4 words on 16 lanes against 2 on 32: 80 labels 397 and 324 us a call, 128
// labels 452 and 411).
template <int NW, int T, int G, int R, bool PYR, int NJ, int RNW = NW, int RT = T>
cudaError_t launch_sum(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st)
{
    cudaError_t err = launch_seg<NW, T, PYR, NJ>(jobs, false, st);
    if (err != cudaSuccess) return err;
    if constexpr (!PYR) {
        err = launch_rowadd_mode<RNW, RT, sg::kSingle, NJ>(jobs, e, st);
    } else {
        Jobs<NJ> part;
        for (int ref = 0; ref < 2 && err == cudaSuccess; ++ref) {
            part.n = 0;
            for (int i = 0; i < jobs.n; ++i)
                if ((jobs.d[i].refine != 0) == (ref != 0)) part.d[part.n++] = jobs.d[i];
            if (part.n == 0) continue;
            if constexpr (2 * NW * T <= kMaxRefineLabels) {
                err = ref ? launch_rowadd_mode<NW, T, sg::kRefine, NJ>(part, e, st)
                          : launch_rowadd_mode<RNW, RT, sg::kCoarse, NJ>(part, e, st);
            } else {
                err = ref ? cudaErrorInvalidValue : launch_rowadd_mode<RNW, RT, sg::kCoarse, NJ>(part, e, st);
            }
        }
    }
    if (err != cudaSuccess) return err;
    dim3 gw((e.max_w + 31) / 32, (e.max_h + 7) / 8, jobs.n);
    prof_begin(st);
    launch_after(k_wta_group<G, R, 1, PYR, NJ>, gw, 256, 0, st, jobs);
    count_launch();
    prof_end(PK_WTA, jobs_vox(jobs) * 2 + jobs_px(jobs) * (2 + 6 + 4), st);
    return launched(st, "k_wta_group");
}

template <bool PYR, int NJ>
cudaError_t launch_paths_sum(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st)
{
    switch (path_variant(jobs.d[0].D)) {
    case 64: return launch_sum<4, 8, 4, 1, PYR, NJ, 2, 16>(jobs, e, st);
    case 128: return launch_sum<4, 16, 8, 1, PYR, NJ, 2, 32>(jobs, e, st);
    case 256: return launch_sum<8, 16, 16, 1, PYR, NJ, 4, 32>(jobs, e, st);
    case 512: return launch_sum<16, 16, 32, 1, PYR, NJ>(jobs, e, st);
    case 1024: return launch_sum<32, 16, 32, 2, PYR, NJ>(jobs, e, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace pg
