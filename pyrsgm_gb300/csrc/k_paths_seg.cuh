// k_paths_seg.cuh -- path aggregation with every chain cut into segments
// that run at the same time.
//
// A path chain (a row in one direction, or a column) is a serial recurrence:
// with one warp walking it, a single pair leaves the GPU idle and a pass
// lasts (steps) x (latency of a step), 218 ns a step measured, 421 us for
// the rows of one 1080p level.  The recurrence forgets its start quickly:
// after subtracting the minimum the state lies in [0, P2], and two chains
// that see the same costs meet exactly after a median of 5-7 steps (99 %
// within about 60) on textured scenes.  So a block holds CPW chains and one
// warp per segment:
//   1. every warp walks its segment, from `warm` steps before it, starting
//      as a chain does that has no previous pixel;
//   2. a segment whose assumed state at its start differs from the path
//      costs its left neighbour ended with is walked again from those,
//      until the costs it computes equal the stored ones at the last pixel
//      of a chunk (from there on the stored ones are the continuation) or
//      its end is reached, which marks the next segment;
//   3. until no segment is marked.
// Each round makes at least the first marked segment of a chain final, so
// there are at most as many rounds as segments, and the result is that of
// the serial walk whatever the costs are.  Scenes without texture take longer:
// at worst every segment is walked once in each round up to its own, in the
// time of the serial walk after the parallel one on an idle GPU, in up to
// three times the work (five segments) on a full one (see k_seg for what
// batches do about it).  Waiting instead until the segment before is final
// was slower on those very scenes (32 pairs of a gradient 10350 us, 10607;
// blurred noise 10133, 10183 to 11953 with the first round cut short): a walk
// from an end that is not final mostly meets the final one soon.
//
// The rows of both directions and the columns share one launch.  Costs come
// through a ring of 4-step chunks per warp: the warp copies the 16-byte
// pieces of all its chains together (cp.async), 4 pixels x 32 bytes of a
// row being a whole line.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "k_paths_packed.cuh"
#include "profiler.h"
#include "sgm_common.cuh"
#include "sgm_launch.h"

namespace pg {

namespace sg {

using pk::kMax2;
using pk::kOne2;

// Level semantics of a walk.
enum { kSingle = 0, kCoarse = 1, kRefine = 2 };
// What a walk does with the path costs: store them; store them until they
// equal the stored ones; add them to the sum in V.
enum { kStore = 0, kAgain = 1, kAdd = 2 };

constexpr int kCH = 4;       // steps per chunk
constexpr int kSC = 3;       // chunk slots per warp
constexpr int kAhead = 3;    // chunks of look-ahead of the per-pixel inputs
constexpr int kForgetful = 4;   // chains for each segment walked again to its end (k_seg)
constexpr int kMaxSeg = 16;  // segments (warps) per block at most
// ... for NW words a thread: shared memory for the rings, and registers.
template <int NW>
__host__ __device__ constexpr int max_seg() { return NW >= 32 ? 4 : NW >= 16 ? 8 : kMaxSeg; }

template <int NW, int T>
struct Geo {
    static_assert(T >= 2, "a chain is held by several lanes");
    static constexpr int D = 2 * NW * T;     // labels a chain can hold
    static constexpr int CPW = 32 / T;       // chains per warp
    static constexpr int PPX = D / 8;        // 16-byte pieces per pixel
    static constexpr int PPC = kCH * PPX;    // pieces per chain and chunk
    static constexpr int NCOP = CPW * PPC / 32;
    // words of one chain's chunk: padded so that the reads of a step (T
    // lanes x NW words per chain) hit distinct banks
    static constexpr int CSTR = kCH * D / 2 + (NW == 8 ? 4 : D == 16 ? 8 : D == 32 ? 16 : 0);
    static constexpr int SLOTW = CPW * CSTR;
    static constexpr int PADW = D / 2 + 1;   // guard words before label 0
    static constexpr int LENW = PADW + D + 2;
    // Word w of chain c lies at w * WST + c: the stride makes the windows of
    // a chain's lanes (NW words apart) fall into distinct banks.
    static constexpr int WST = T >= 16 ? CPW : NW == 2 || T == 2 ? 20 : T == 4 ? 10 : 9;
    static constexpr int BUFW = (LENW * WST + 3) / 4 * 4;   // (the rings between the windows stay 16-byte aligned)
    static constexpr int QL = kCH > T ? kCH / T : 1;   // pixels of a chunk a lane prepares
};

template <int NW, int T, int MODE>
__host__ __device__ constexpr int warp_words(int rings = 1)
{
    using G = Geo<NW, T>;
    static_assert(G::CSTR % 4 == 0 && G::BUFW % 4 == 0, "cp.async writes 16-byte pieces");
    return rings * kSC * G::SLOTW + (MODE == kRefine ? 2 * G::BUFW : 0);
}
template <int NW, int T, int MODE>
constexpr size_t add_smem()
{
    return 4 * (256 + 2 * (size_t)warp_words<NW, T, MODE>(2));   // a warp a direction
}
template <int NW, int T, int MODE>
constexpr size_t seg_smem(int segs)
{
    return 4 * (256 + (size_t)(kMaxSeg + 1) * 32 +
                (size_t)segs * (warp_words<NW, T, MODE>() + (segs > 1 ? 32 * NW : 0)));
}

// Labels of a level on chains that hold D: 16 and 32 exactly, else any
// multiple of 16 up to D (the other slots stay SHRT_MAX).
template <int D>
__device__ __forceinline__ int labels_of(const LevelDesc& J)
{
    return D <= 32 ? D : J.D;
}

// The lane's stored path costs of a pixel (labels d0 on; those past Dr stay).
template <int NW>
__device__ __forceinline__ void load_words(const int16_t* p, int d0, int Dr, uint32_t (&v)[NW])
{
    if constexpr (NW == 2) {
        const uint2 a = __ldcg(reinterpret_cast<const uint2*>(p));
        v[0] = a.x; v[1] = a.y;
    } else {
#pragma unroll
        for (int i = 0; i < NW / 4; ++i) {
            if (d0 + 8 * i >= Dr) break;
            const uint4 a = __ldcg(reinterpret_cast<const uint4*>(p) + i);
            v[4 * i] = a.x; v[4 * i + 1] = a.y; v[4 * i + 2] = a.z; v[4 * i + 3] = a.w;
        }
    }
}

template <int NW, bool FULL>   // FULL: the level has every label of the chain
__device__ __forceinline__ void store_words(int16_t* p, int d0, int Dr, const uint32_t (&v)[NW])
{
    if constexpr (NW == 2) {
        if (FULL || d0 < Dr) *reinterpret_cast<uint2*>(p) = make_uint2(v[0], v[1]);
    } else {
#pragma unroll
        for (int i = 0; i < NW / 4; ++i) {
            if (d0 + 8 * i >= Dr) break;
            reinterpret_cast<uint4*>(p)[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        }
    }
}

__device__ __forceinline__ void cp16s(uint32_t dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// Where a chain runs: step t is at pixel p0 + dp * t (image byte l0 + dl * t,
// column xs + dx * t), 0 <= t < n.
struct Walk {
    long long p0, l0;
    int dp, dl, n, xs, dx;
};

// Path extents of a level (single-scale: kernel_AggregateLR/RL ranges).
template <int MODE>
struct Extent {
    int lr_x0, lr_n, rl_n, xlo, ncol;
    __device__ __forceinline__ explicit Extent(const LevelDesc& J)
    {
        if (MODE == kSingle) {
            const int minX1 = imax(J.minD + J.D, 0), maxX1 = J.w + imin(J.minD, 0);
            lr_x0 = xlo = minX1;
            lr_n = J.paths >= 2 ? imax(0, maxX1 - minX1) : 0;
            rl_n = imax(0, J.w - minX1);
            ncol = imax(0, maxX1 - minX1);
        } else {
            lr_x0 = xlo = 0;
            lr_n = J.paths >= 2 ? J.w : 0;
            rl_n = ncol = J.w;
        }
        if (J.paths < 3) ncol = 0;
    }
};

template <int MODE>
__device__ __forceinline__ Walk walk_of(const LevelDesc& J, const Extent<MODE>& e, bool rows, int g)
{
    Walk w;
    if (rows) {
        const int y = g >> 1, dir = g & 1;
        const bool ok = y < J.h;
        w.n = !ok ? 0 : dir ? e.rl_n : e.lr_n;
        w.xs = dir ? J.w - 1 : e.lr_x0;
        w.dx = w.dp = w.dl = dir ? -1 : 1;
        const long long yy = ok ? y : 0;
        w.p0 = yy * J.w + w.xs;
        w.l0 = yy * J.lstep + w.xs;
    } else {
        const bool ok = g < e.ncol;
        w.n = ok ? J.h : 0;
        w.xs = e.xlo + (ok ? g : 0);
        w.dx = 0;
        w.dp = J.w;
        w.dl = J.lstep;
        w.p0 = w.l0 = w.xs;
    }
    return w;
}

template <int NW, int T>
struct State {
    uint32_t L[NW];
    uint32_t mp2;   // minimum over the chain's labels, in both halves
};

template <int NW, int T, bool LONE = false>
__device__ __forceinline__ uint32_t chain_min_dup(const uint32_t (&L)[NW])
{
    uint32_t m = L[0];
    if constexpr (NW == 2) {
        m = __vminu2(L[0], L[1]);
    } else {
#pragma unroll
        for (int i = 1; i + 1 < NW; i += 2) m = __vimin3_u16x2(m, L[i], L[i + 1]);
        m = __vminu2(m, L[NW - 1]);
    }
    m = __vminu2(m, __funnelshift_l(m, m, 16));
    // Across lanes: a shuffle a level of the tree or a warp reduction a chain.
    // Two reductions are shorter than four dependent shuffles (641x479 with 96
    // labels 209 us a call, 182), as is one than five; four against three only
    // where a lone warp waits for each step (LONE; 720p with 48 labels 311,
    // 285; the segments of 64 labels 217, 222).
    if constexpr (T >= 16 || (LONE && T == 8)) {
        const unsigned g = (threadIdx.x & 31) / T;
        uint32_t r = m;
#pragma unroll
        for (unsigned i = 0; i < 32 / T; ++i) {
            const uint32_t a = __reduce_min_sync(0xffffffffu, g == i ? m : 0xffffffffu);
            if (g == i) r = a;
        }
        return r;
    } else {
#pragma unroll
        for (int o = 1; o < T; o <<= 1) m = __vminu2(m, __shfl_xor_sync(0xffffffffu, m, o));
        return m;
    }
}

// Window position of a label shift: byte offset of the word holding label
// -1 of the shifted window, its half in bit 0.
template <int NW, int T>
__device__ __forceinline__ uint32_t window_at(int delta)
{
    using G = Geo<NW, T>;
    const int i0 = 2 * G::PADW + iclamp(delta, -(G::D + 1), G::D + 1) - 1;
    return (uint32_t)((i0 >> 1) * G::WST * 4) | (uint32_t)(i0 & 1);
}

// One step: c = the lane's costs, at = window_at(label shift) in the low
// half (refine), p22 = the penalty in both halves, win = the lane's word 0
// in the chain's window buffer of this parity.  pk::gstep's recurrence with
// the jump taken out of the chain,
//   min(c + min(best, minPrev + P2) - minPrev, MAX) =
//   min(c + best - minPrev, min(c + P2, MAX)),
// so that only the neighbours' minimum and minPrev are on it.  `guard`: an
// active chain's best may reach SHRT_MAX (see k_seg), which then stays.
template <int NW, int T, int MODE, bool LONE>
__device__ __forceinline__ void seg_step(State<NW, T>& s, const uint32_t (&c)[NW], uint32_t at, uint32_t p22,
                                         uint32_t p12, uint32_t* win, int k, bool guard)
{
    using G = Geo<NW, T>;
    uint32_t w[NW + 1], n0[NW];   // (L[s - 1], L[s]) of label pair m, and (L[s], L[s + 1])
    if constexpr (MODE == kRefine) {
#pragma unroll
        for (int i = 0; i < NW; ++i) win[(G::PADW + i) * G::WST] = s.L[i];
        __syncwarp();
        const uint32_t* wp = reinterpret_cast<const uint32_t*>(reinterpret_cast<const char*>(win) + (at & 0xfffcu));
        const uint32_t sh = at << 4;   // the funnel takes it modulo 32
        uint32_t w0[NW + 2];
#pragma unroll
        for (int j = 0; j < NW + 2; ++j) w0[j] = wp[j * G::WST];
#pragma unroll
        for (int j = 0; j < NW + 1; ++j) w[j] = __funnelshift_r(w0[j], w0[j + 1], sh);
#pragma unroll
        for (int m = 0; m < NW; ++m) n0[m] = __funnelshift_r(w[m], w[m + 1], 16);
    } else {
        uint32_t wl = __shfl_up_sync(0xffffffffu, s.L[NW - 1], 1, T);
        uint32_t wr = __shfl_down_sync(0xffffffffu, s.L[0], 1, T);
        if (k == 0) wl = kMax2;
        if (k == T - 1) wr = kMax2;
        w[0] = __funnelshift_r(wl, s.L[0], 16);
#pragma unroll
        for (int m = 1; m < NW; ++m) w[m] = __funnelshift_r(s.L[m - 1], s.L[m], 16);
        w[NW] = __funnelshift_r(s.L[NW - 1], wr, 16);
#pragma unroll
        for (int m = 0; m < NW; ++m) n0[m] = s.L[m];
    }
    uint32_t best[NW];
#pragma unroll
    for (int m = 0; m < NW; ++m) best[m] = __vimin3_u16x2(n0[m], w[m] + p12, w[m + 1] + p12);
#pragma unroll
    for (int m = 0; m < NW; ++m)
        s.L[m] = __viaddmin_u16x2(c[m], best[m] - s.mp2, __viaddmin_u16x2(c[m], p22, kMax2));
    if (MODE != kSingle && guard && s.mp2 != kMax2) {
        const uint32_t lj2 = __viaddmin_u16x2(s.mp2, p22, kMax2);
#pragma unroll
        for (int m = 0; m < NW; ++m) s.L[m] |= pk::sign_mask2(__vminu2(best[m], lj2) + kOne2) & kMax2;
    }
    s.mp2 = chain_min_dup<NW, T, LONE>(s.L);
}

// The block's adaptive-P2 table; returns whether an active chain's best may
// reach SHRT_MAX.  It does only where minPrev + P2 does; path costs are at
// most cost + P2, so with costs of at most cmax that takes cmax + 2 P2 >=
// SHRT_MAX.
__device__ __forceinline__ bool load_penalties(const LevelDesc& J, int* lut)
{
    const int side = imin(J.bs | 1, 127);
    const int cmax = J.cost == COST_CENSUS ? 24 : imin(kMax, 255 * side * side);
    bool high = cmax + 2 * imin(J.P2, kMax) >= kMax;
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
        lut[i] = J.adaptive ? J.p2lut[i] : 0;
        high = high || cmax + 2 * imin(lut[i], kMax) >= kMax;
    }
    return high;
}

// SHRT_MAX at the lane's labels (from d0 on) that label_range rules out for
// pixel x of a coarse level.
template <int NW>
__device__ __forceinline__ void invalid_labels(int x, int minD, int maxD, int wLast, int d0, uint32_t (&mask)[NW])
{
    const int lo = imax(0, x - wLast - minD) - d0, hi = imin(maxD, x) - minD - d0;   // relative to d0
#pragma unroll
    for (int i = 0; i < NW; ++i)
        mask[i] = (2 * i < lo || 2 * i > hi ? 0x7fffu : 0u) | (2 * i + 1 < lo || 2 * i + 1 > hi ? 0x7fff0000u : 0u);
}

// What a walk needs beside its state.
template <int NW, int T, int MODE>
struct Ctx {
    const LevelDesc& J;
    const int* lut;
    uint32_t* ring;      // [kSC][SLOTW]
    uint32_t* win;       // [2][BUFW] (refine): this lane's word 0
    uint32_t* edge;      // [segment][lane][NW]: path costs at each segment's last step
    int lane, c, k;
    Extent<MODE> e;
    bool rows, adaptive, guard;
    int g0;              // first chain of the warp
    Walk w;              // this lane's chain
    int16_t* out;        // its path-cost volume
    uint32_t p12;
    int stop = 0;        // kAdd: the walk's end
    bool sums = false;   // kAdd: V holds other paths' costs, which are added to
};

// Walk the steps [t0, t0 + 4 * nch) of the warp's chains that lie below each
// chain's te (a per-lane bound; `segs` and `b` give the same bound for the
// chains a lane copies for).  Steps before ts are not stored.  FIX: only the
// chains with `act` set are walked, the state of step t0 - 1 is in `s`, a
// chain stops at the first step whose costs equal the stored ones; returns
// whether it reached te without one.  ADD: chains of one direction (every
// second one from g0 on); t0 may be up to three steps before the chain's
// start, where the ring's SHRT_MAX keeps the state empty.
template <int NW, int T, int MODE, int KIND>
__device__ __forceinline__ bool seg_walk(const Ctx<NW, T, MODE>& X, State<NW, T>& s, int t0, int ts, int te, int nch,
                                         int segs, int b, int wch, bool act, uint32_t (&spec)[NW])
{
    using G = Geo<NW, T>;
    constexpr int D = G::D;
    constexpr bool FIX = KIND == kAgain, ADD = KIND == kAdd;
    const LevelDesc& J = X.J;
    const int lane = X.lane, k = X.k;
    const int Dr = labels_of<D>(J);
    // the descriptor's fields that the loop reads, in registers
    const int minD = J.minD, maxD = J.maxD, wLast = J.w - 1, P2 = J.P2;
    const int16_t* const Bg = J.base;
    const uint8_t* const Lg = J.left;
    int16_t* const Vg = J.V;
    const int16_t* const Cg = J.C;
    // Copies of a chunk: piece i = lane + 32 j of the warp's CPW * PPC.
    // Below 64 labels a lane copies one piece each of NCOP chains a fixed
    // number apart (of the same direction); from 64 on the chain of copy j
    // is a constant and its pieces lie a fixed number of pixels apart.
    constexpr bool kApart = G::PPC < 32;
    static_assert(!ADD || !kApart, "the chains of a warp are two apart");
    constexpr int kChains = kApart ? 1 : G::CPW;            // start pointers a lane keeps
    constexpr int kStep = kApart ? 32 / G::PPC : 1;         // chains between two copies
    constexpr int kPer = kApart ? 1 : G::PPC / 32;          // copies per chain
    const int r0 = lane % G::PPC;
    const int q0 = G::PPX <= 32 ? r0 / G::PPX : 0, off0 = G::PPX <= 32 ? (r0 % G::PPX) * 8 : lane * 8;
    const int16_t* src[kChains];
    int lim[kChains], advD[kChains];                        // chunk ci is copied while 4 * ci < lim
    int jmax = G::NCOP;
    long long apart = 0;
#pragma unroll
    for (int i = 0; i < kChains; ++i) {
        const int cc = kApart ? lane / G::PPC : i;
        const Walk w = walk_of<MODE>(J, X.e, X.rows, X.g0 + cc * (ADD ? 2 : 1));
        const int len = ((w.n + segs - 1) / segs + kCH - 1) / kCH * kCH;
        const int first = b * len, tb = ADD ? t0 : first - wch * kCH;
        lim[i] = w.n > 0 && off0 < Dr ? (ADD ? X.stop : imin(w.n, first + len)) - tb - q0 : -(1 << 30);
        advD[i] = w.dp * Dr;
        src[i] = J.C + (w.p0 + (long long)w.dp * (tb + q0)) * Dr + off0;
        if (kApart) {
            apart = X.rows ? (long long)(kStep / 2) * J.w * Dr : (long long)kStep * Dr;
            jmax = X.rows ? (J.h - ((X.g0 + cc) >> 1) + kStep / 2 - 1) / (kStep / 2 > 0 ? kStep / 2 : 1)
                          : (X.e.ncol - (X.g0 + cc) + kStep - 1) / kStep;
        }
    }
    const uint32_t dst0 =
        pk::smem_addr(X.ring + (kApart ? (lane / G::PPC) * G::CSTR : 0) + q0 * (D / 2) + off0 / 2);
    const int early = -t0 - q0;   // ADD: pixels of the first chunk before the chain's start
    int ci_issue = 0;
    auto issue = [&](int slot) {
#pragma unroll
        for (int j = 0; j < G::NCOP; ++j) {
            constexpr int kQ = G::PPX <= 32 ? 32 / G::PPX : 1;   // pixels between two copies of a chain
            const int i = kApart ? 0 : j / kPer, jj = kApart ? 0 : j % kPer;
            const int dq = kApart ? 0 : G::PPX <= 32 ? jj * kQ : jj / (G::PPX > 32 ? G::PPX / 32 : 1);
            const int doff = G::PPX <= 32 ? 0 : 256 * (jj % (G::PPX > 32 ? G::PPX / 32 : 1));
            const bool in = kCH * ci_issue + dq < lim[i] && (!ADD || ci_issue > 0 || dq >= early) &&
                            (kApart ? j < jmax : off0 + doff < Dr);
            const int16_t* p = src[i] + (kApart ? j * apart : (long long)dq * advD[i] + doff);
            const uint32_t dst =
                dst0 + 4 * (slot * G::SLOTW + (kApart ? j * kStep : i) * G::CSTR + dq * (D / 2) + doff / 2);
            if (in && PG_IN(p - J.C, 8, (size_t)J.w * J.h * Dr, 5)) {
                cp16s(dst, p);
                if (ADD) cp16s(dst + 4 * kSC * G::SLOTW, Vg + (p - Cg));
            }
        }
#pragma unroll
        for (int i = 0; i < kChains; ++i) src[i] += (long long)kCH * advD[i];
        pk::cp_commit();
        ++ci_issue;
    };
    // label bases and intensities of the pixels this lane prepares (q = k +
    // T * i of a chunk), loaded kAhead chunks before their use: a load that
    // misses L2 takes several chunks of steps, and nothing may touch the
    // loaded values before
    const bool need = MODE == kRefine || X.adaptive;
    const uint32_t p2const = pk::dup(imin(P2, 0x7fff));
    const unsigned span = te > ts ? te - ts : 0;
    struct Pixel {
        uint32_t base, img;
    };
    auto load_pixel = [&](int t, Pixel& v) {
        if (MODE == kRefine) v.base = (uint32_t)(uint16_t)Bg[X.w.p0 + (long long)X.w.dp * t];
        if (X.adaptive) v.img = Lg[X.w.l0 + (long long)X.w.dl * t];
    };
    auto load_chunk = [&](int t, Pixel (&v)[G::QL]) {
#pragma unroll
        for (int i = 0; i < G::QL; ++i) {
            const int tq = t + k + T * i;
            v[i] = {0u, 0u};
            if (need && k < kCH && tq < te && (!ADD || tq >= 0)) load_pixel(tq, v[i]);
        }
    };
    Pixel pix[kAhead + 1][G::QL], first{0u, 0u};
    if (need && t0 > 0 && t0 - 1 < te) load_pixel(t0 - 1, first);
    uint32_t last = first.base << 16 | first.img;   // of the previous chunk's last pixel
    int16_t* op = X.out + (X.w.p0 + (long long)X.w.dp * t0) * Dr + 2 * NW * k;
    const long long ostep = (long long)X.w.dp * Dr;
    // stored path costs of the last step of this chunk and the next ones (FIX)
    uint32_t old[FIX ? kAhead + 1 : 1][NW];
    auto load_old = [&](int t, const int16_t* p, uint32_t (&v)[NW]) {
        if (FIX && act && t + kCH <= te) load_words<NW>(p + (kCH - 1) * ostep, 2 * NW * k, Dr, v);
    };
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
        load_chunk(t0 + kCH * i, pix[i]);
        if constexpr (FIX) load_old(t0 + kCH * i, op + kCH * i * ostep, old[i]);
    }
#pragma unroll
    for (int j = 0; j < kSC - 1; ++j) issue(j);
    int slot = 0, islot = kSC - 1;
    uint32_t mask[NW];   // coarse: SHRT_MAX at the pixel's invalid labels (a column's are those of every pixel)
#pragma unroll
    for (int i = 0; i < NW; ++i) mask[i] = 0;
    for (int ci = 0; ci < nch; ++ci) {
        if (FIX && !__any_sync(0xffffffffu, act)) break;
        const int t = t0 + kCH * ci;
        load_chunk(t + kCH * kAhead, pix[kAhead]);
        if constexpr (FIX) load_old(t + kCH * kAhead, op + kCH * kAhead * ostep, old[kAhead]);
        __syncwarp();   // every lane has read the slot that is filled next
        issue(islot);
        islot = islot + 1 == kSC ? 0 : islot + 1;
        uint32_t cur[G::QL];
#pragma unroll
        for (int i = 0; i < G::QL; ++i) cur[i] = pix[0][i].base << 16 | pix[0][i].img;
        // window position (low half) and penalty (high half) towards the previous pixel
        uint32_t info[G::QL];
        if (need) {
            uint32_t prev[G::QL];
            if constexpr (T == 2) {
                const uint32_t a = __shfl_xor_sync(0xffffffffu, cur[0], 1), z = __shfl_xor_sync(0xffffffffu, cur[1], 1);
                prev[0] = k ? a : last;
                prev[1] = k ? z : a;
                last = k ? cur[1] : z;
            } else {
                const uint32_t a = __shfl_up_sync(0xffffffffu, cur[0], 1, T);
                prev[0] = k ? a : last;
                last = __shfl_sync(0xffffffffu, cur[0], kCH - 1, T);
            }
#pragma unroll
            for (int i = 0; i < G::QL; ++i) {
                int p2 = P2;
                if (X.adaptive) p2 = X.lut[abs((int)(cur[i] & 255u) - (int)(prev[i] & 255u))];
                info[i] = (uint32_t)imin(p2, 0x7fff) << 16;
                if (MODE == kRefine)
                    info[i] |= window_at<NW, T>((int)(int16_t)(cur[i] >> 16) - (int)(int16_t)(prev[i] >> 16));
            }
        }
        pk::cp_wait<kSC - 1>();
        __syncwarp();
        if constexpr (KIND == kStore) {
            if (ci == wch) {
#pragma unroll
                for (int i = 0; i < NW; ++i) spec[i] = s.L[i];
            }
        }
        // coarse levels: does a pixel of the chunk have an invalid label?
        bool border = false;
        if (MODE == kCoarse) {
            const int xa = X.w.xs + X.w.dx * t, xb = xa + X.w.dx * (kCH - 1);
            border = __any_sync(0xffffffffu, imin(maxD, imin(xa, xb)) - minD < Dr - 1 || imax(xa, xb) - wLast > minD);
            if (border && (X.rows || ci == 0)) invalid_labels<NW>(xa, minD, maxD, wLast, 2 * NW * k, mask);
        }
        const uint32_t* cin = X.ring + slot * G::SLOTW + X.c * G::CSTR + k * NW;
        slot = slot + 1 == kSC ? 0 : slot + 1;
        // ADD: a lone warp waits for every load, so a chunk's costs and sums
        // are read ahead of its steps (641x479 with 96 labels 182 us a call, 179)
        constexpr bool kEarly = ADD && NW <= 8;
        uint32_t ce[kEarly ? kCH : 1][NW], ve[kEarly ? kCH : 1][NW];
        if constexpr (kEarly) {
#pragma unroll
            for (int q = 0; q < kCH; ++q) {
                pk::ldw<NW>(cin + q * (D / 2), ce[q]);
                pk::ldw<NW>(cin + kSC * G::SLOTW + q * (D / 2), ve[q]);
            }
        }
#pragma unroll
        for (int q = 0; q < kCH; ++q) {
            uint32_t cc[NW];
            if constexpr (kEarly) {
#pragma unroll
                for (int i = 0; i < NW; ++i) cc[i] = ce[q][i];
            } else {
                pk::ldw<NW>(cin + q * (D / 2), cc);
            }
            uint32_t at = 0, p22 = p2const;
            if (need) {
                at = __shfl_sync(0xffffffffu, info[T < kCH ? q / T : 0], T < kCH ? q % T : q, T);
                p22 = __byte_perm(at, 0, 0x3232);
            }
            if (MODE == kCoarse && border) {
                if (X.rows && q > 0) invalid_labels<NW>(X.w.xs + X.w.dx * (t + q), minD, maxD, wLast, 2 * NW * k, mask);
#pragma unroll
                for (int i = 0; i < NW; ++i) cc[i] |= mask[i];
            }
            seg_step<NW, T, MODE, ADD>(s, cc, at, p22, X.p12, X.win + (q & 1) * G::BUFW, k, X.guard);
            bool put = (unsigned)(t + q - ts) < span;
            if constexpr (FIX) put = put && act;
            uint32_t res[NW];
#pragma unroll
            for (int i = 0; i < NW; ++i) res[i] = s.L[i];
            if constexpr (ADD) {
                if (X.sums) {
                    uint32_t v[NW];
                    if constexpr (kEarly) {
#pragma unroll
                        for (int i = 0; i < NW; ++i) v[i] = ve[q][i];
                    } else {
                        pk::ldw<NW>(cin + kSC * G::SLOTW + q * (D / 2), v);
                    }
#pragma unroll
                    for (int i = 0; i < NW; ++i) res[i] = pk::gcombine<MODE != kSingle>(v[i], res[i]);
                }
            }
            if (put && PG_IN(op - X.out, imin(2 * NW, Dr - 2 * NW * k), (size_t)J.w * J.h * Dr, 6))
                store_words<NW, D <= 32>(op, 2 * NW * k, Dr, res);
            op += ostep;
        }
        if constexpr (FIX) {
            uint32_t diff = 0;
#pragma unroll
            for (int i = 0; i < NW; ++i)
                if (2 * NW * k + 2 * i < Dr) diff |= s.L[i] ^ old[0][i];
            const unsigned ne = __ballot_sync(0xffffffffu, diff != 0);
            const unsigned mine = T == 32 ? ne : (ne >> (X.c * T)) & ((1u << (T & 31)) - 1u);
            if (t + kCH <= te && mine == 0) act = false;
        }
        // segments followed by another hold whole chunks
        if (!ADD && segs > 1 && t + kCH == te && (!FIX || act)) {
#pragma unroll
            for (int i = 0; i < NW; ++i) X.edge[(b * 32 + lane) * NW + i] = s.L[i];
        }
#pragma unroll
        for (int a = 0; a < kAhead; ++a) {
#pragma unroll
            for (int i = 0; i < G::QL; ++i) pix[a][i] = pix[a + 1][i];
            if constexpr (FIX) {
#pragma unroll
                for (int i = 0; i < NW; ++i) old[a][i] = old[a + 1][i];
            }
        }
    }
    pk::cp_wait<0>();
    __syncwarp();
    return act;
}

}  // namespace sg

// The chains of a level: groups [0, row groups) hold rows (both directions),
// the following ones columns, a block a group; `rows_too` 0 launches the
// columns alone (their path costs are all that is written, into V).
//
// Batches: images without texture (gradients, wide flat parts, sparse
// detail) have chains that do not forget, whose segments are walked again
// and again, up to three times the work.  A refinement level counts the
// segments that it walks again to their ends (in launches as large as its
// child's has to be for the rule below), and where its parent counted
// more than one for every `kForgetful` chains, a block's warps take whole
// chains instead, a group each: one walk, at the occupancy of the segments'.
// Textured pairs count 0.05 a chain at most, the others 0.25 to 9.  32 pairs
// of 1080p (us; segments, whole chains there, and before there were
// segments): gradient 10337, 8763, 9789; diagonal one 11829, 8707, 9581;
// sparse dots 11104, 8720, 9658; flat but for a sixteenth of the width 10777,
// 8175, 8895; texture 7928, 7911, 9983.  A whole chain takes its n steps
// however few there are beside it, segments a time that grows with their
// number: whole chains pay from n / kWholePace groups per SM on (`may_whole`;
// 12 pairs of 1080p: at 20 a level of 1920 steps 4666 and 3708, 8 pairs, at
// 13, 2722 and 2955).
template <int NW, int T, int MODE, int NJ>
__global__ void __launch_bounds__(sg::max_seg<NW>() * 32) k_seg(const __grid_constant__ Jobs<NJ> jobs, int rows_too, int warm,
                                                                       int may_whole)
{
    using namespace sg;
    using G = Geo<NW, T>;
    const LevelDesc& J = jobs.d[blockIdx.y];
    extern __shared__ __align__(16) uint32_t smem[];
    const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const Extent<MODE> e(J);
    const int Dr = labels_of<G::D>(J);
    const int rgroups = rows_too ? (2 * J.h + G::CPW - 1) / G::CPW : 0;
    if ((int)blockIdx.x >= rgroups && ((int)blockIdx.x - rgroups) * G::CPW >= e.ncol) {   // the block is past the level
        after_previous();
        return;
    }
    int* lut = reinterpret_cast<int*>(smem);
    int* marked = reinterpret_cast<int*>(smem + 256);   // [segment][chain]: walk it (again)
    uint32_t* mine = smem + 256 + (kMaxSeg + 1) * 32 + warp * warp_words<NW, T, MODE>();
    uint32_t* edge = smem + 256 + (kMaxSeg + 1) * 32 + warps * warp_words<NW, T, MODE>();
    for (int i = lane; i < warp_words<NW, T, MODE>(); i += 32) mine[i] = kMax2;
    if (rows_too) let_next_in();   // (columns alone: k_rowadd is next)
    after_previous();
    // whole chains, a group a warp, or segments of one group's?
    bool whole = false;
    if constexpr (NJ > 1 && MODE == kRefine)
        whole = may_whole && J.parent_rewalked && *J.parent_rewalked > (2 * J.ph + J.pw) / kForgetful;
    const int segs = whole ? 1 : warps, b = whole ? 0 : warp;
    const int group = whole ? (int)blockIdx.x * warps + warp : (int)blockIdx.x;
    const bool rows = group < rgroups;
    const int g0 = (rows ? group : group - rgroups) * G::CPW;
    const bool high = load_penalties(J, lut);
    const bool guard = __syncthreads_or(high);
    if (whole) {
        if (blockIdx.x == 0 && threadIdx.x == 0) *J.rewalked = INT_MAX;   // the child's chains too
        if (!rows && g0 >= e.ncol) return;
    }

    const int k = lane % T;
    Ctx<NW, T, MODE> X{J, lut, mine, mine + kSC * G::SLOTW + lane / T + NW * k * G::WST, edge, lane, lane / T, k, e,
                       rows, J.adaptive != 0, guard, g0, {}, nullptr, pk::dup(imin(J.P1, 0x8000))};
    const int g = g0 + X.c;
    X.w = walk_of<MODE>(J, e, rows, g);
    X.out = rows ? ((g & 1) ? J.Vr : J.Vl) : J.V;
    const int n = X.w.n;
    const int len = ((n + segs - 1) / segs + kCH - 1) / kCH * kCH;
    const int ts = b * len, te = n > 0 ? imin(n, ts + len) : -(1 << 30);
    const int nmax = rows ? imax(e.lr_n, e.rl_n) : J.h;
    const int nch = ((nmax + segs - 1) / segs + kCH - 1) / kCH;
    const int nmin = rows && e.lr_n > 0 ? imin(e.lr_n, e.rl_n) : nmax;
    const int wch = b == 0 ? 0 : imin(warm, (nmin + segs - 1) / segs) / kCH;

    State<NW, T> s;
    uint32_t spec[NW];
#pragma unroll
    for (int i = 0; i < NW; ++i) s.L[i] = spec[i] = kMax2;
    s.mp2 = kMax2;
    seg_walk<NW, T, MODE, kStore>(X, s, ts - wch * kCH, ts, te, wch + nch, segs, b, wch, true, spec);
    if (segs == 1) return;

    const bool has = b > 0 && ts < te;
    auto start_state = [&]() {   // the path costs of the pixel before the segment
#pragma unroll
        for (int i = 0; i < NW; ++i) s.L[i] = has ? edge[((b - 1) * 32 + lane) * NW + i] : kMax2;
        s.mp2 = chain_min_dup<NW, T>(s.L);
    };
    __syncthreads();
    start_state();
    bool go;
    {
        uint32_t diff = 0;
#pragma unroll
        for (int i = 0; i < NW; ++i) diff |= s.L[i] ^ spec[i];
        const unsigned ne = __ballot_sync(0xffffffffu, diff != 0);
        const unsigned m = T == 32 ? ne : (ne >> (X.c * T)) & ((1u << (T & 31)) - 1u);
        go = has && m != 0;
    }
    [[maybe_unused]] int again = 0;   // segments walked again to their ends
    for (int round = 0; round < segs; ++round) {
        // a warp reads and clears its own row of marks; the warp before it
        // sets them between this barrier and the next
        __syncwarp();
        marked[b * 32 + lane] = 0;
        if (!__syncthreads_or(go)) break;   // also: every start state has been read
        if (__any_sync(0xffffffffu, go)) {
            const bool past = seg_walk<NW, T, MODE, kAgain>(X, s, ts, ts, te, nch, segs, b, 0, go, spec);
            if (past && X.k == 0) marked[(b + 1) * 32 + X.c] = 1;
            if (NJ > 1 && MODE == kRefine && may_whole) again += __popc(__ballot_sync(0xffffffffu, past && X.k == 0));
        }
        __syncthreads();
        go = has && marked[b * 32 + X.c] != 0;
        start_state();
    }
    if (NJ > 1 && MODE == kRefine && lane == 0 && again > 0 && J.rewalked) atomicAdd(J.rewalked, again);
}

// Segments for a launch of `blocks` chain groups whose longest walk has n
// steps.
// Refinement levels: as many as fill the SMs where there are one or two
// groups per SM (960x540 42 us with 8, 1080p 90 with 7), else five, four for
// short walks: a block then holds a few rows over a stretch that L2 keeps
// between its two directions, and three blocks of five warps are as many as
// shared memory and L1 serve well.  1080p rows of 16 pairs: 1543 us with one
// segment, 1275 with 4, 1099 with 5, 1091 with 6, 1110 with 7, 1220 with 8,
// 1220 with 12, 1354 with 16.
// Coarse and single-scale levels forget their start over 100 to 200 steps
// and walk more segments again and again (mixed batch, 64 labels: 204 us with
// 1, 134 with 2, 137 with 4, 175 with 8, 276 with 16); columns alone
// (k_rowadd does the rows) take what keeps every group resident (641x479, 96
// labels: 37 us with 8, 46 with 4).
// A segment holds at least 64 steps (2879x1987 pyramid: 1247 us a call with
// 64, 1262 with 40, 1270 with 130), 40 for the first four segments of small
// levels (160x96: 42 us a call, 46 at 64).
constexpr int kMinSeg = 64, kMinSegSmall = 40;
constexpr int kMaxRefineLabels = 256;   // pyrsgm_compute_level takes no more on a refinement level
constexpr int kWholePace = 100;  // steps of a whole chain for each group per SM (k_seg)
constexpr int kWarmSteps = 16;   // 0 to 32 measured within 5 % of each other, 64 10 % slower

template <int MODE>
int segments_for(long long blocks, int n, bool rows_too, int most)
{
    const long long per_sm = std::max<long long>(1, (blocks + sm_count() - 1) / sm_count());
    long long want;
    if (MODE == sg::kRefine) want = per_sm == 1 ? 16 : per_sm == 2 ? 7 : n >= 480 ? 5 : 4;
    else want = std::max<long long>(2, std::min<long long>(16 / per_sm, rows_too ? 4 : 16));
    const long long fit = std::max(n / kMinSeg, std::min(4, n / kMinSegSmall));
    return (int)std::max<long long>(1, std::min<long long>(std::min<long long>(want, most), fit));
}

template <int NW, int T, int MODE, int NJ>
cudaError_t launch_seg_mode(const Jobs<NJ>& jobs, bool rows_too, cudaStream_t st)
{
    using G = sg::Geo<NW, T>;
    long long blocks = 0;
    int grid = 0, n = 0;
    for (int i = 0; i < jobs.n; ++i) {
        const LevelDesc& d = jobs.d[i];
        const int rg = rows_too ? (2 * d.h + G::CPW - 1) / G::CPW : 0;
        const int cg = d.paths >= 3 ? (d.w + G::CPW - 1) / G::CPW : 0;
        grid = std::max(grid, rg + cg);
        blocks += rg + cg;
        n = std::max(n, rows_too ? std::max(d.w, d.h) : d.h);
    }
    if (grid == 0) return cudaSuccess;
    int segs = segments_for<MODE>(blocks, n, rows_too, sg::max_seg<NW>());
    while (segs > 1 && sg::seg_smem<NW, T, MODE>(segs) > kSmemPerBlock) --segs;
    const size_t smem = sg::seg_smem<NW, T, MODE>(segs);
    const cudaError_t err = allow_smem(k_seg<NW, T, MODE, NJ>);
    if (err != cudaSuccess) return err;
    prof_begin(st);
    launch_after(k_seg<NW, T, MODE, NJ>, dim3(grid, jobs.n), segs * 32, smem, st, jobs, rows_too ? 1 : 0, kWarmSteps,
                 blocks * kWholePace >= (long long)n * sm_count() ? 1 : 0);
    count_launch();
    if (prof_enabled()) {
        // each path reads the cost volume and writes its costs once
        double by = 0;
        for (int i = 0; i < jobs.n; ++i) {
            const LevelDesc& d = jobs.d[i];
            const int paths = rows_too ? d.paths : d.paths >= 3 ? 1 : 0;
            by += (double)d.w * d.h * paths * (d.D * 4 + (d.refine ? 2 : 0) + (d.adaptive ? 1 : 0));
        }
        prof_end(PK_PATH_ROW, by, st);
    }
    return launched(st, "k_seg");
}

// Path costs of every chain (rows_too 0: the columns only).  Coarse and
// refinement levels of one batch take a launch each.
template <int NW, int T, bool PYR, int NJ>
cudaError_t launch_seg(const Jobs<NJ>& jobs, bool rows_too, cudaStream_t st)
{
    if constexpr (!PYR) {
        return launch_seg_mode<NW, T, sg::kSingle, NJ>(jobs, rows_too, st);
    } else {
        int nref = 0;
        for (int i = 0; i < jobs.n; ++i) nref += jobs.d[i].refine != 0;
        if (nref == 0) return launch_seg_mode<NW, T, sg::kCoarse, NJ>(jobs, rows_too, st);
        if constexpr (2 * NW * T <= kMaxRefineLabels) {
            if (nref == jobs.n) return launch_seg_mode<NW, T, sg::kRefine, NJ>(jobs, rows_too, st);
            Jobs<NJ> part;
            for (int ref = 0; ref < 2; ++ref) {
                part.n = 0;
                for (int i = 0; i < jobs.n; ++i)
                    if ((jobs.d[i].refine != 0) == (ref != 0)) part.d[part.n++] = jobs.d[i];
                const cudaError_t err = ref ? launch_seg_mode<NW, T, sg::kRefine, NJ>(part, rows_too, st)
                                            : launch_seg_mode<NW, T, sg::kCoarse, NJ>(part, rows_too, st);
                if (err != cudaSuccess) return err;
            }
            return cudaSuccess;
        }
        return cudaErrorInvalidValue;
    }
}

}  // namespace pg
