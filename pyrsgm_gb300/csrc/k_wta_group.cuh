// k_wta_group.cuh -- winner-take-all with several lanes a pixel
// (kernel_WTA_Subpixel, src/sgm_kernels.cu:573-640; pyramid
// kernel_PyramidWTA, src/sgm_kernels.cu:1290-1370).
//
// G lanes read a pixel's labels, 16 R each, and reduce; after G pixels every
// lane has one winner of its own, and the rules and outputs run on full
// warps.  VOLS 1: the total is in V (label counts that keep one path
// volume).  VOLS 3: it is the capped sum of V, Vl and Vr (64 labels; with 16
// and 32 the thread per pixel of k_wta is as fast or faster: 1080p with a
// 32-label coarse level 470 us a call against 473).  With 64 a thread per
// pixel read 16 bytes of 32 lines a load: 640x480 117 us a call, now 109.
// Bound by memory and, over one volume, by the integer pipe.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "k_paths_packed.cuh"
#include "sgm_common.cuh"
#include "sgm_launch.h"

namespace pg {

__device__ __forceinline__ void load16(const int16_t* p, uint32_t (&v)[8])
{
    const uint4 *q = reinterpret_cast<const uint4*>(p), a = q[0], b = q[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

template <int G, int R, int VOLS, bool PYR, int NJ>
__global__ void __launch_bounds__(256) k_wta_group(const __grid_constant__ Jobs<NJ> jobs)
{
    if (NJ == 1) let_next_in();   // (in a batch the next label count's chains may follow)
    after_previous();
    const LevelDesc& J = jobs.d[blockIdx.z];
    const int W = J.w, D = J.D, lane = threadIdx.x & 31, gl = lane % G;
    const int y = blockIdx.y * 8 + (threadIdx.x >> 5), x0 = blockIdx.x * 32;
    if (x0 >= W || y >= J.h) return;
    int xlo = 0, xhi = W;
    if (!PYR) {
        xlo = imax(J.minD + D, 0);
        xhi = imin(W + imin(J.minD, 0), W - 1);   // the last column has no winner
    }
    const size_t row0 = (size_t)y * W * D;
    const int16_t* row = J.V + row0;
    [[maybe_unused]] const int paths = J.paths, accEnd = PYR ? W : paths >= 2 ? W + imin(J.minD, 0) : W;
    unsigned myBest = 0;
    int myAlt = 0, c0 = 0, c2 = 0;
#pragma unroll 2
    for (int i = 0; i < G; ++i) {
        const int x = imin(x0 + lane - gl + i, W - 1);
        uint32_t t[8 * R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int d0 = 16 * (gl + G * r);
            uint32_t v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = pk::kMax2;
            if (d0 < D && PG_IN(row0 + (size_t)x * D + d0, 16, (size_t)W * J.h * D, 14)) {
                const size_t at = (size_t)x * D + d0;
                load16((VOLS == 1 ? row : J.Vr + row0) + at, v);
                if constexpr (VOLS == 3) {
                    uint32_t u[8], z[8];
                    if (paths >= 2) load16(J.Vl + row0 + at, u);
                    if (paths >= 3) load16(row + at, z);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        if (paths >= 2) v[j] = pk::gcombine<PYR>(u[j], v[j]);
                        if (paths >= 3) v[j] = pk::gcombine<PYR>(z[j], v[j]);
                    }
                    if (J.debug_acc && x0 + lane - gl + i < W && x >= xlo && x < accEnd) {
                        uint4* o = reinterpret_cast<uint4*>(J.V + row0 + at);
                        o[0] = make_uint4(v[0], v[1], v[2], v[3]);
                        o[1] = make_uint4(v[4], v[5], v[6], v[7]);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) t[8 * r + j] = v[j];
        }
        // cost in the high half, label in the low one (the shift as a product: the other pipe)
        unsigned best = 0xffffffffu;
#pragma unroll
        for (int j = 0; j < 8 * R; ++j) {
            const unsigned d = 16u * (gl + G * (j / 8)) + 2 * (j % 8);
            best = __vimin3_u32(best, t[j] * 65536u + d, (t[j] & 0xffff0000u) | (d + 1));
        }
#pragma unroll
        for (int o = 1; o < G; o <<= 1) best = umin(best, __shfl_xor_sync(0xffffffffu, best, o));
        const int bd = (int)(best & 0xffffu);
        [[maybe_unused]] int before = 0, after = 0;   // the costs next to the best
        if constexpr (VOLS == 3) {
            static_assert(VOLS == 1 || R == 1, "one lane holds each label's total");
            const uint32_t v[8] = {t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7]};
            before = __shfl_sync(0xffffffffu, pk::half_of(v, (bd - 1) & 15), ((bd - 1) >> 4) & (G - 1), G);
            after = __shfl_sync(0xffffffffu, pk::half_of(v, (bd + 1) & 15), ((bd + 1) >> 4) & (G - 1), G);
        }
        // minimum over the labels further than one from the best, two at a
        // time: d - bd + 1 is 0, 1 or 2 at the others, which become SHRT_MAX
        // (from 3 on the addition sets the sign)
        uint32_t far2 = pk::kMax2;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t first = pk::dup(16 * (gl + G * r) + 1 - bd) + 0x00010000u;   // of labels 0 and 1
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t far3 = __viaddmin_u16x2(first, 0x00020002u * j, 0x00030003u) + 0x7ffd7ffdu;
                t[8 * r + j] |= ~pk::sign_mask2(far3) & pk::kMax2;
            }
#pragma unroll
            for (int j = 0; j < 8; j += 2) far2 = __vimin3_u16x2(far2, t[8 * r + j], t[8 * r + j + 1]);
        }
        unsigned far = umin(far2 & 0xffffu, far2 >> 16);
#pragma unroll
        for (int o = 1; o < G; o <<= 1) far = umin(far, __shfl_xor_sync(0xffffffffu, far, o));
        if (gl == i) {
            myBest = best;
            myAlt = (int)far;
            if constexpr (VOLS == 3) {
                c0 = bd > 0 ? before : 0;
                c2 = bd + 1 < D ? after : 0;
            }
        }
    }
    const int x = x0 + lane;
    if (x >= W) return;
    const size_t p = (size_t)y * W + x;
    if (x < xlo || x >= xhi) {
        J.disp_raw[p] = (int16_t)((J.minD - 1) * 16);
        J.conf_raw[p] = 0.0f;
        return;
    }
    const int minCost = (int)(myBest >> 16), bd = (int)(myBest & 0xffffu);
    if constexpr (VOLS == 1) {
        c0 = bd > 0 ? (int)row[(size_t)x * D + bd - 1] : 0;
        c2 = bd + 1 < D ? (int)row[(size_t)x * D + bd + 1] : 0;
    }
    const int base = (PYR && J.refine) ? (int)J.base[p] : J.minD;
    pk::wta_out<PYR>(J, D, y, x, base, minCost, bd, myAlt, c0, minCost, c2);
}

}  // namespace pg
