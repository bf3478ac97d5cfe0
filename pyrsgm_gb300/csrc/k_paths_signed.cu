// k_paths_signed.cu -- aggregation and winner of a level whose penalties may
// be below zero.
//
// StereoMatcher and the batch engine refuse such penalties, but
// pyrsgm_compute_level and pyrsgm_compute_single_scale take any, as the
// reference does.  With them a path cost falls below the previous pixel's
// minimum and below zero, which the packed kernels (unsigned 16-bit halves)
// cannot hold.  Here everything is signed, in the reference's order: L->R,
// T->B and R->L each add to V, then the winner and the LR check of a row
// (src/sgm_kernels.cu:520-889, 1191-1478).
//
// A warp walks a chain, lane l holding labels l, l + 32, ...; the next
// pixel's costs are loaded before the current one is finished.  Bound by the
// latency of a step; a call with sensible penalties never comes here.
#include <type_traits>

#include "profiler.h"
#include "sgm_common.cuh"
#include "sgm_launch.h"

namespace pg {

enum { kLR = 0, kTB = 1, kRL = 2 };

template <int K, bool PYR>
__global__ void __launch_bounds__(32) k_path_signed(const __grid_constant__ LevelDesc J, int dir, int add)
{
    const int W = J.w, H = J.h, D = J.D, lane = threadIdx.x, chain = blockIdx.x;
    int xlo = 0, xhi = W;
    if (!PYR) {
        xlo = imax(J.minD + D, 0);
        xhi = dir == kRL ? W : W + imin(J.minD, 0);
    }
    const bool rows = dir != kTB;
    const int n = rows ? xhi - xlo : H;
    if (n <= 0 || (!rows && chain >= xhi - xlo)) return;
    int x = rows ? (dir == kRL ? xhi - 1 : xlo) : xlo + chain;
    const int dx = dir == kRL ? -1 : dir == kLR ? 1 : 0;
    const long long dp = rows ? dx : W, dl = rows ? dx : J.lstep;
    long long p = rows ? (long long)chain * W + x : x;
    const uint8_t* img = J.left + (rows ? (long long)chain * J.lstep + x : x);

    __shared__ int lut[256], prev[2][32 * K];
    if (J.adaptive)
        for (int i = lane; i < 256; i += 32) lut[i] = J.p2lut[i];
    __syncwarp();
    int next[K], nextBase = 0, nextImg = 0;
    auto load = [&](long long q, const uint8_t* im) {
#pragma unroll
        for (int k = 0; k < K; ++k) next[k] = lane + 32 * k < D ? (int)J.C[q * D + lane + 32 * k] : kMax;
        nextBase = PYR && J.refine ? (int)J.base[q] : J.minD;
        nextImg = J.adaptive ? (int)*im : 0;
    };
    load(p, img);
    int minPrev = kMax, prevBase = J.minD, prevImg = 0, par = 0;
    bool active = false;   // the previous pixel had a finite path cost
    for (int t = 0; t < n; ++t) {
        int c[K];
#pragma unroll
        for (int k = 0; k < K; ++k) c[k] = next[k];
        const int base = nextBase, im = nextImg;
        if (t + 1 < n) load(p + dp, img + dl);
        int lo = 0, hi = D - 1;
        if (PYR) label_range(J, x, base, lo, hi);
        const int p2 = J.adaptive ? lut[abs(im - prevImg)] : J.P2;
        const int jump = imin(kMax, minPrev + p2), shift = base - prevBase;
        const int* L = prev[par];
        int m = kMax;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int d = lane + 32 * k;
            if (d >= D) break;
            const bool valid = !PYR || (d >= lo && d <= hi && c[k] < kMax);
            int v = kMax;
            if (valid && !active) {
                v = c[k];
            } else if (valid) {
                const int s = d + shift;
                const bool below = s > 0 && s <= D, above = s >= -1 && s + 1 < D;
                int same = s >= 0 && s < D ? L[s] : kMax, lm = below ? L[s - 1] : kMax, lp = above ? L[s + 1] : kMax;
                // (an invalid neighbour of a pyramid level takes no penalty)
                if (below && (!PYR || lm < kMax)) lm += J.P1;
                if (above && (!PYR || lp < kMax)) lp += J.P1;
                const int best = imin(imin(same, jump), imin(lm, lp));
                v = PYR && best >= kMax ? kMax : sat16(c[k] + best - minPrev);
            }
            prev[par ^ 1][d] = v;
            m = imin(m, v);
            if (PG_IN(p * D + d, 1, (long long)W * H * D, 12)) {
                int16_t* o = J.V + p * D + d;
                const int old = add ? (int)*o : 0;
                if (PYR) *o = (int16_t)(old < kMax && v < kMax ? imin(kMax - 1, old + v) : kMax);
                else *o = (int16_t)imin(kMax, old + v);
            }
        }
        minPrev = __reduce_min_sync(0xffffffffu, m);
        __syncwarp();
        active = !PYR || (hi >= lo && minPrev < kMax);
        prevBase = base;
        prevImg = im;
        par ^= 1;
        p += dp;
        img += dl;
        x += dx;
    }
}

// Winner of every pixel of a row, then its LR check (the post pass has none
// to do): a block per row.  Costs order as the reference's keys do, the label
// of the smallest unsigned 16-bit cost; the right image's candidates by their
// signed cost, hence the bias.
template <bool PYR>
__global__ void __launch_bounds__(256) k_wta_signed(const __grid_constant__ LevelDesc J)
{
    const int W = J.w, D = J.D, y = blockIdx.x;
    const int16_t inv = (int16_t)((J.minD - 1) * 16);
    unsigned* keys = J.keys + (size_t)y * W;
    int xlo = 0, xhi = W;
    if (!PYR) {
        xlo = imax(J.minD + D, 0);
        xhi = imin(W + imin(J.minD, 0), W - 1);   // the last column has no winner
    }
    for (int x = threadIdx.x; x < W; x += 256) {
        const size_t p = (size_t)y * W + x;
        int16_t disp = inv;
        float conf = 0.0f;
        if (x >= xlo && x < xhi) {
            const int16_t* v = J.V + p * D;
            unsigned key = 0xffffffffu;
            for (int d = 0; d < D; ++d) key = min(key, ((unsigned)(uint16_t)v[d] << 16) | (unsigned)d);
            const int minCost = (int)(int16_t)(key >> 16), bd = (int)(key & 0xffffu);
            int alt = kMax;
            for (int d = 0; d < D; ++d)
                if (abs(d - bd) > 1) alt = imin(alt, v[d]);
            const int base = PYR && J.refine ? (int)J.base[p] : J.minD, real = base + bd;
            bool ok;
            if (PYR) {
                int lo, hi;
                label_range(J, x, base, lo, hi);
                ok = hi - lo >= 2 && minCost < kMax && alt < kMax;
                if (J.uniq > 0 && alt * (100 - J.uniq) < minCost * 100) ok = false;
                if ((bd == 0 && base > J.minD) || (bd == D - 1 && base + D - 1 < imin(J.maxD, x))) ok = false;
            } else {
                ok = minCost < kMax / 2 && !(J.uniq > 0 && alt * (100 - J.uniq) < minCost * 100);
            }
            const float c = fminf(fmaxf(((float)alt - (float)minCost) / fmaxf((float)minCost, 1.0f), 0.0f), 1.0f);
            if (PYR && c < J.minConf) ok = false;
            if (ok) {
                int d16 = real * 16;
                if (bd > 0 && bd + 1 < D) {
                    const int c0 = v[bd - 1], c1 = v[bd], c2 = v[bd + 1];
                    const int den = imax(c0 + c2 - 2 * c1, 1);
                    if (!PYR || (c0 < kMax && c1 < kMax && c2 < kMax)) d16 += ((c0 - c2) * 16 + den) / (den * 2);
                }
                disp = (int16_t)d16;
                conf = c;
                const int x2 = x - real;
                if (x2 >= 0 && x2 < W)
                    atomicMin(&keys[x2], ((unsigned)(minCost - SHRT_MIN) << 16) | (unsigned)(0xffff - x));
            }
        }
        J.disp_raw[p] = disp;
        J.conf_raw[p] = conf;
    }
    if (!(J.post & POST_LRCHECK)) return;
    __syncthreads();
    for (int x = threadIdx.x; x < W; x += 256) {
        const size_t p = (size_t)y * W + x;
        const int d16 = J.disp_raw[p];
        if (d16 == inv) continue;
        auto far = [&](int d, bool& seen) {   // the right image's disparity at x - d, if it has one, is not d
            const int rx = x - d;
            seen = rx >= 0 && rx < W;
            if (!seen) return false;
            const unsigned k = __ldcg(&keys[rx]);
            const int v = k == 0xffffffffu ? (int)inv : (int)(0xffffu - (k & 0xffffu)) - rx;
            seen = v >= J.minD;
            return seen && abs(v - d) > J.maxdiff;
        };
        bool on0, on1;
        const bool far0 = far(d16 >> 4, on0), far1 = far((d16 + 15) >> 4, on1);
        if (PYR ? !((on0 && !far0) || (on1 && !far1)) : far0 && far1) {
            J.disp_raw[p] = inv;
            J.conf_raw[p] = 0.0f;
        }
    }
}

template <int K, bool PYR>
static cudaError_t launch_signed(const LevelDesc& d, cudaStream_t st)
{
    cudaError_t err = cudaSuccess;
    for (int dir = d.paths >= 2 ? kLR : kRL; dir <= kRL && err == cudaSuccess; ++dir) {
        if (dir == kTB && d.paths < 3) continue;
        prof_begin(st);
        k_path_signed<K, PYR><<<dir == kTB ? d.w : d.h, 32, 0, st>>>(d, dir, dir != kLR && d.paths >= 2);
        count_launch();
        prof_end(dir == kTB ? PK_PATH_TB : PK_PATH_ROW, (double)d.w * d.h * d.D * (dir == kLR ? 4 : 6), st);
        err = launched(st, "k_path_signed");
    }
    if (err != cudaSuccess) return err;
    prof_begin(st);
    k_wta_signed<PYR><<<d.h, 256, 0, st>>>(d);
    count_launch();
    prof_end(PK_WTA, (double)d.w * d.h * (d.D * 2 + 12), st);
    return launched(st, "k_wta_signed");
}

cudaError_t launch_paths_signed(const LevelDesc& d, cudaStream_t st)
{
    auto run = [&](auto k) {
        constexpr int K = decltype(k)::value;
        return d.pyr ? launch_signed<K, true>(d, st) : launch_signed<K, false>(d, st);
    };
    if (d.D <= 32) return run(std::integral_constant<int, 1>());
    if (d.D <= 128) return run(std::integral_constant<int, 4>());
    if (d.D <= 512) return run(std::integral_constant<int, 16>());
    return run(std::integral_constant<int, 32>());
}

}  // namespace pg
