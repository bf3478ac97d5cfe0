// k_post.cu -- 3x3 median, median-changed confidence reset and the output
// conversion of one level, fused into one pass; plus the path-kernel
// dispatch.  Reference: kernel_MedianFilter3x3, kernel_ClearChangedMedian-
// Confidence (src/sgm_kernels.cu:891-931), convertDispAndConfKernel
// (src/sgm_kernels.cu:1530-1551) and the output copies of
// pyrsgm_compute_level / pyrsgm_compute_single_scale
// (src/sgm_kernels.cu:1837-1858, 2053-2069).
#include "profiler.h"
#include "sgm_common.cuh"
#include "sgm_launch.h"

namespace pg {

template <bool PYR, int NJ>
cudaError_t launch_paths_mode(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st);

template <int NJ>
cudaError_t launch_paths(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st)
{
    return jobs.d[0].pyr ? launch_paths_mode<true, NJ>(jobs, e, st) : launch_paths_mode<false, NJ>(jobs, e, st);
}

// 3x3 median of the interior by column sorts: each column of three is
// sorted once and shared by the three windows it belongs to; the median of
// the nine is the median of (largest column minimum, median of the column
// medians, smallest column maximum) -- the structure of the opt_med9
// network of Paeth / Devillard ("Fast median search: an ANSI C
// implementation") --, two pixels at a time in 16-bit halves.
__device__ __forceinline__ uint32_t med3(uint32_t a, uint32_t b, uint32_t c)
{
    return __vmaxs2(__vmins2(a, b), __vmins2(__vmaxs2(a, b), c));
}

struct Col3 {
    uint32_t lo, mid, hi;
};
__device__ __forceinline__ Col3 sort3(uint32_t a, uint32_t b, uint32_t c)
{
    const uint32_t l = __vmins2(a, b), h = __vmaxs2(a, b);
    return {__vmins2(l, c), __vmaxs2(l, __vmins2(h, c)), __vmaxs2(h, c)};
}
// The columns one to the left of the second pair: the high half of a, the low half of b.
__device__ __forceinline__ Col3 between(const Col3& a, const Col3& b)
{
    return {__funnelshift_r(a.lo, b.lo, 16), __funnelshift_r(a.mid, b.mid, 16), __funnelshift_r(a.hi, b.hi, 16)};
}
__device__ __forceinline__ uint32_t median9(const Col3& a, const Col3& b, const Col3& c)
{
    return med3(__vimax3_s16x2(a.lo, b.lo, c.lo), med3(a.mid, b.mid, c.mid), __vimin3_s16x2(a.hi, b.hi, c.hi));
}

// One block: 128 x 8 pixels.  The (LR-checked) disparities of the tile and a
// halo of one row and four columns are computed once into shared memory, a
// thread per 4 adjacent pixels: 340 of the block's 352 threads (256 threads in
// two rounds spent the second one on a third of them).  Loads come first, in
// three rounds so that they overlap: confidences and raw disparities, the
// disp2 keys they point at, decisions.  Then 8 warps take a row each, 4
// pixels a thread; the median takes the in-image neighbours only (sorted,
// middle element) at the image border.  Bound by the latency of the dependent
// loads and by instruction issue (32 levels of 1080p: 496 -> 433 us).
constexpr int kPoX = 128, kPoY = 8;
constexpr int kPoG = kPoX / 4 + 2;   // groups of 4 pixels per staged row: columns x0 - 4 .. x0 + 131
constexpr int kPoN = (kPoY + 2) * kPoG, kPoThreads = (kPoN + 31) / 32 * 32;

template <int NJ>
__global__ void __launch_bounds__(kPoThreads) k_post(const __grid_constant__ Jobs<NJ> jobs)
{
    let_next_in();
    after_previous();
    const LevelDesc& J = jobs.d[blockIdx.z];
    const int x0 = blockIdx.x * kPoX, y0 = blockIdx.y * kPoY;
    if (x0 >= J.w || y0 >= J.h) return;
    const int W = J.w, H = J.h;
    const int inv = (int)(int16_t)((J.minD - 1) * 16);
    // The LR check (kernel_StrictPyramidLRCheck / kernel_PseudoLRCheck,
    // src/sgm_kernels.cu:825-889).
    const bool check = (J.post & POST_LRCHECK) != 0;
    const bool med = (J.post & POST_MEDIAN) != 0;
    const bool quad = (W & 3) == 0;   // rows of raw disparities and confidences start on 4-pixel boundaries
    const int tx = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int xb = x0 + 4 * tx, y = y0 + warp;
    const int np = warp < kPoY && y < H ? imin(4, W - xb) : 0;
    __shared__ __align__(16) uint2 td[kPoY + 2][kPoG];   // row r, group g: pixels x0 - 4 + 4 g .. of row y0 - 1 + r
    float cin[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (np > 0) {
        const float* c = J.conf_raw + (size_t)y * W + xb;
        if (quad) {
            const float4 v = *reinterpret_cast<const float4*>(c);
            cin[0] = v.x; cin[1] = v.y; cin[2] = v.z; cin[3] = v.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j < np) cin[j] = c[j];
        }
    }
    if (threadIdx.x < kPoN) {
        const int r = threadIdx.x / kPoG, g = threadIdx.x - r * kPoG;
        const int yy = y0 - 1 + r, xg = x0 - 4 + 4 * g;
        const bool in = yy >= 0 && yy < H && xg >= 0 && xg < W;
        const uint32_t inv2 = (uint32_t)(uint16_t)inv * 0x10001u;
        uint2 a = make_uint2(inv2, inv2);   // the four disparities
        if (in) {
            const int16_t* p = J.disp_raw + (size_t)yy * W + xg;
            if (quad) {
                a = *reinterpret_cast<const uint2*>(p);
            } else {
                uint32_t v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = xg + j < W ? (uint32_t)(uint16_t)p[j] : (uint32_t)(uint16_t)inv;
                a = make_uint2(v[0] | (v[1] << 16), v[2] | (v[3] << 16));
            }
        }
        if (check && in) {
            // The key of right pixel rx holds the cost and 0xffff - x' of its
            // winner x' (all ones: none); the winner's disparity there is x' - rx, and
            // rx + d0 = x, so that disp2 - d0 = x' - x.  A right pixel
            // without a winner has disparity `inv` in the reference, which
            // counts where it is not below minD (minD > 1).
            const unsigned* row = J.keys + (size_t)yy * W;
            const int maxdiff = J.maxdiff;
            unsigned k0[4], k1[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int d = (int)(int16_t)(j < 2 ? a.x >> (16 * j) : a.y >> (16 * (j - 2)));
                const int r0 = xg + j - (d >> 4), r1 = xg + j - ((d + 15) >> 4);
                k0[j] = k1[j] = 0xffffffffu;
                if ((unsigned)r0 < (unsigned)W) k0[j] = row[r0];
                if ((unsigned)r1 < (unsigned)W) k1[j] = row[r1];
            }
            bool bad[4];
            if (inv < J.minD && maxdiff >= 0 && maxdiff <= 65536) {
                // |x' - x| <= maxdiff as one unsigned comparison; the top bit
                // (a cost never has it) keeps no winner far from any x
                const unsigned span = 2u * (unsigned)maxdiff;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const unsigned c = (unsigned)(0xffff + maxdiff - xg - j);
                    const bool far0 = c - (k0[j] & 0x8000ffffu) > span, far1 = c - (k1[j] & 0x8000ffffu) > span;
                    bad[j] = far0 && far1 && (J.pyr || (k0[j] != 0xffffffffu && k1[j] != 0xffffffffu));
                }
            } else {
                const bool none_counts = inv >= J.minD;
#pragma unroll 1
                for (int j = 0; j < 4; ++j) {
                    const int d = (int)(int16_t)(j < 2 ? a.x >> (16 * j) : a.y >> (16 * (j - 2)));
                    const int x = xg + j, d0 = d >> 4, d1 = (d + 15) >> 4;
                    const unsigned q0 = k0[0], q1 = k1[0];
                    bool on0 = q0 != 0xffffffffu, on1 = q1 != 0xffffffffu;
                    int e0 = abs((int)(~q0 & 0xffffu) - x), e1 = abs((int)(~q1 & 0xffffu) - x);
                    if (none_counts) {
                        if (!on0) e0 = abs(inv - d0);
                        if (!on1) e1 = abs(inv - d1);
                        on0 = (unsigned)(x - d0) < (unsigned)W;
                        on1 = (unsigned)(x - d1) < (unsigned)W;
                    }
                    const bool b = J.pyr ? !((on0 && e0 <= maxdiff) || (on1 && e1 <= maxdiff))
                                         : (on0 && e0 > maxdiff) && (on1 && e1 > maxdiff);
#pragma unroll
                    for (int i = 0; i < 3; ++i) { k0[i] = k0[i + 1]; k1[i] = k1[i + 1]; bad[i] = bad[i + 1]; }
                    bad[3] = b;
                }
            }
            // (an invalid disparity stays what it is)
            if (bad[0]) a.x = __byte_perm(a.x, inv2, 0x3254);
            if (bad[1]) a.x = __byte_perm(a.x, inv2, 0x5410);
            if (bad[2]) a.y = __byte_perm(a.y, inv2, 0x3254);
            if (bad[3]) a.y = __byte_perm(a.y, inv2, 0x5410);
        }
        (&td[0][0])[threadIdx.x] = a;
    }
    __syncthreads();
    if (np <= 0) return;
    uint2 d = td[warp + 1][tx + 1], m = d;   // checked disparities, median
    if (med) {
        if (xb > 0 && xb + 4 < W && y > 0 && y + 1 < H) {
            // column pairs (xb - 2, xb - 1) .. (xb + 4, xb + 5)
            Col3 c[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t v[3];
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    const uint2* row = &td[warp + r][tx];
                    v[r] = i == 0 ? row[0].y : i == 1 ? row[1].x : i == 2 ? row[1].y : row[2].x;
                }
                c[i] = sort3(v[0], v[1], v[2]);
            }
            const Col3 mid = between(c[1], c[2]);
            m.x = median9(between(c[0], c[1]), c[1], mid);
            m.y = median9(mid, c[2], between(c[2], c[3]));
        } else {
            int16_t o[4] = {0, 0, 0, 0};
            for (int j = 0; j < np; ++j) {
                const int x = xb + j;
                int v[9];
                int n = 0;
                for (int dy = -1; dy <= 1; ++dy) {
                    if (y + dy < 0 || y + dy >= H) continue;
                    const int16_t* row = reinterpret_cast<const int16_t*>(td[warp + 1 + dy]);
                    for (int dx = -1; dx <= 1; ++dx) {
                        if (x + dx < 0 || x + dx >= W) continue;
                        v[n++] = row[4 * tx + 4 + j + dx];
                    }
                }
                for (int i = 1; i < n; ++i) {
                    const int key = v[i];
                    int q = i - 1;
                    while (q >= 0 && v[q] > key) { v[q + 1] = v[q]; --q; }
                    v[q + 1] = key;
                }
                o[j] = (int16_t)v[n / 2];
            }
            m = make_uint2((uint32_t)(uint16_t)o[0] | ((uint32_t)(uint16_t)o[1] << 16),
                           (uint32_t)(uint16_t)o[2] | ((uint32_t)(uint16_t)o[3] << 16));
        }
    }
    const bool vec = np == 4;
    if (J.out16 && PG_IN((size_t)y * J.out16_pitch + xb, np, (size_t)J.out16_pitch * H, 8)) {
        int16_t* o = J.out16 + (size_t)y * J.out16_pitch + xb;
        if (vec && ((reinterpret_cast<uintptr_t>(o) & 7) == 0)) {
            *reinterpret_cast<uint2*>(o) = m;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j < np) o[j] = (int16_t)(j < 2 ? m.x >> (16 * j) : m.y >> (16 * (j - 2)));
        }
    }
    const bool conv = J.out32 && J.outc;
    if (!conv && !(J.outc && J.conf_only_copy)) return;
    // the confidence stays where neither the check (which leaves `inv`) nor
    // the median changed the disparity; invalid pixels have 0
    float f32[4], fc[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int dn = (int)(int16_t)(j < 2 ? m.x >> (16 * j) : m.y >> (16 * (j - 2)));
        const int dc = (int)(int16_t)(j < 2 ? d.x >> (16 * j) : d.y >> (16 * (j - 2)));
        const bool ok = dn != inv && dn > 0;
        f32[j] = ok ? dn / 16.0f : 0.0f;
        fc[j] = dn == dc && dc != inv && (ok || !conv) ? cin[j] : 0.0f;
    }
    auto store4 = [&](float* o, const float (&v)[4]) {
        if (vec && ((reinterpret_cast<uintptr_t>(o) & 15) == 0)) {
            *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j < np) o[j] = v[j];
        }
    };
    if (conv) store4(J.out32 + (size_t)y * J.out32_pitch + xb, f32);
    store4(J.outc + (size_t)y * J.outc_pitch + xb, fc);
}

template <int NJ>
cudaError_t launch_post(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st)
{
    dim3 g((e.max_w + kPoX - 1) / kPoX, (e.max_h + kPoY - 1) / kPoY, jobs.n);
    prof_begin(st);
    launch_after(k_post<NJ>, g, kPoThreads, 0, st, jobs);
    count_launch();
    if (prof_enabled()) {
        double by = 0;
        for (int i = 0; i < jobs.n; ++i) {
            const LevelDesc& d = jobs.d[i];
            const double outb = (d.out16 ? 2 : 0) + (d.out32 ? 4 : 0) + (d.outc ? 4 : 0);
            by += (double)d.w * d.h * (6 + outb);
        }
        prof_end(PK_POST, by, st);
    }
    return launched(st, "k_post");
}

template cudaError_t launch_paths<1>(const Jobs<1>&, const LevelExtent&, cudaStream_t);
template cudaError_t launch_paths<kBatchJobs>(const Jobs<kBatchJobs>&, const LevelExtent&, cudaStream_t);
template cudaError_t launch_post<1>(const Jobs<1>&, const LevelExtent&, cudaStream_t);
template cudaError_t launch_post<kBatchJobs>(const Jobs<kBatchJobs>&, const LevelExtent&, cudaStream_t);

}  // namespace pg
