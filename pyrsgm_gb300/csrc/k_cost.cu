// k_cost.cu -- per-pixel stages of one level: pyrDown, census / BT features,
// refine-label preparation, the adaptive-P2 table and the matching-cost
// volume.  Integer arithmetic, clamps and sentinels follow the reference
// kernels cited at each function (reference file:line).
#include <type_traits>

#include "profiler.h"
#include "sgm_common.cuh"
#include "sgm_launch.h"

namespace pg {

// ---------------------------------------------------------------------------
// pyrDown: 5x5 [1 4 6 4 1]^2 / 256, BORDER_REFLECT_101, (sum+128)>>8.
// Reference: src/pyrdown.cu:16-52.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int reflect101(int i, int n)
{
    if (i < 0) i = -i;
    if (i >= n) i = 2 * n - 2 - i;
    return i < 0 ? 0 : i;
}

// Bytes c .. c + 3 of an image row as a word: one load where the row is word
// aligned there, two otherwise, single bytes at the indices that `map` gives
// where the four leave [0, w) or the words the image [first, end).
template <typename Map>
__device__ __forceinline__ uint32_t load4(const uint8_t* row, int c, int w, const uint8_t* first, const uint8_t* end,
                                          Map map)
{
    if (c >= 0 && c + 4 <= w) {
        const unsigned s = (unsigned)(reinterpret_cast<uintptr_t>(row + c) & 3u);
        const uint8_t* a = row + c - s;
        if (s == 0) return *reinterpret_cast<const uint32_t*>(a);
        if (a >= first && a + 8 <= end) {
            const uint32_t* q = reinterpret_cast<const uint32_t*>(a);
            return __funnelshift_r(*q, q[1], 8 * s);
        }
    }
    uint32_t v = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) v |= (uint32_t)row[map(c + j)] << (8 * j);
    return v;
}

// One block: 128 x 16 output pixels, a thread per 4 adjacent outputs of two
// rows.  The source tile (rows 2*y0 - 2 .. 2*y0 + 32, columns 2*x0 - 4 ..
// 2*x0 + 259) is staged as words, a warp per row with all its loads in
// flight; of a border tile (80 of the 272 of 960x540 outputs) only the words
// with reflected columns come byte by byte.  Rows that are not word aligned
// take two loads a word.  Vertical sums are at most 16 * 255 and the sums of
// both directions 256 * 255 + 128, so two columns share a register
// throughout: even and odd source columns apart, the taps of two outputs
// come out as one product each.  Bound by instruction issue: 32 images of
// 1080p 75 us with bytes and one column a register, 26 now.
constexpr int kPdX = 128, kPdY = 16;
constexpr int kPdSWB = 2 * kPdX + 8;    // staged source bytes per row
constexpr int kPdSWW = kPdSWB / 4;
constexpr int kPdSH = 2 * kPdY + 3;     // staged source rows

template <int NB>
__global__ void __launch_bounds__(256) k_pyrdown(const __grid_constant__ PyrDownBatch<NB> b)
{
    let_next_in();
    after_previous();
    const PyrDownDesc& P = b.d[blockIdx.z];
    const int x0 = blockIdx.x * kPdX, y0 = blockIdx.y * kPdY;
    if (x0 >= P.dw || y0 >= P.dh) return;
    __shared__ __align__(8) uint32_t tw[kPdSH][kPdSWW];   // byte c of row r: source (reflect(2*y0 - 2 + r), reflect(2*x0 - 4 + c))
    const int sx0 = 2 * x0 - 4, sy0 = 2 * y0 - 2, sw = P.sw, sh = P.sh;
    const uint8_t* const first = P.src;
    const uint8_t* const end = first + (size_t)(sh - 1) * P.sstep + sw;
    const int tx = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // a warp per row
    if (((reinterpret_cast<uintptr_t>(first) | (uintptr_t)P.sstep) & 3u) == 0) {
        const bool in0 = sx0 + 4 * tx >= 0 && sx0 + 4 * tx + 4 <= sw, in1 = sx0 + 4 * tx + 132 <= sw,
                   in2 = tx < kPdSWW - 64 && sx0 + 4 * tx + 260 <= sw;
#pragma unroll
        for (int r = warp; r < kPdSH; r += 8) {
            const uint32_t* q =
                reinterpret_cast<const uint32_t*>(first + (size_t)reflect101(sy0 + r, sh) * P.sstep + sx0) + tx;
            if (in0) tw[r][tx] = *q;
            if (in1) tw[r][tx + 32] = q[32];
            if (in2) tw[r][tx + 64] = q[64];
        }
        // the words with columns outside that an output needs: the first one, and from `from` on
        const int left = sx0 < 0 ? 1 : 0, from = imax((sw - sx0) >> 2, left);
        const int last = (2 * imin(x0 + kPdX - 1, P.dw - 1) + 2 - sx0) >> 2;
        const int edge = left + imax(0, imin(last + 1, kPdSWW) - from);
        for (int i = threadIdx.x; i < kPdSH * edge; i += 256) {
            const int r = i / edge, m = i - r * edge, k = m < left ? 0 : from + m - left;
            const uint8_t* row = first + (size_t)reflect101(sy0 + r, sh) * P.sstep;
            uint32_t v = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) v |= (uint32_t)row[reflect101(sx0 + 4 * k + j, sw)] << (8 * j);
            tw[r][k] = v;
        }
    } else {
        for (int r = warp; r < kPdSH; r += 8) {
            const uint8_t* row = first + (size_t)reflect101(sy0 + r, sh) * P.sstep;
#pragma unroll
            for (int k = tx; k < kPdSWW; k += 32)
                tw[r][k] = load4(row, sx0 + 4 * k, sw, first, end, [&](int c) { return reflect101(c, sw); });
        }
    }
    __syncthreads();
    const int xb = x0 + 4 * tx, yb = y0 + 2 * warp;
    if (xb >= P.dw || yb >= P.dh) return;
    const int np = imin(4, P.dw - xb);
    // tile bytes 8 * tx + 2 .. 8 * tx + 12 are the source columns of the four
    // outputs: even ones 0 | 2, 4 | 6, 8 | 10, 12 | 14, odd ones 1 | 3, ...
    uint32_t ev[2][4], od[2][3];
#pragma unroll
    for (int o = 0; o < 2; ++o) {
#pragma unroll
        for (int k = 0; k < 4; ++k) ev[o][k] = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) od[o][k] = 0;
    }
#pragma unroll
    for (int r = 0; r < 7; ++r) {
        const uint2* row = reinterpret_cast<const uint2*>(tw[4 * warp + r]) + tx;
        const uint2 a = row[0], z = row[1];
        const uint32_t q[4] = {a.x, a.y, z.x, z.y};
        constexpr uint32_t w5[5] = {1, 4, 6, 4, 1};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t e = __byte_perm(q[k], 0, 0x4240), u = __byte_perm(q[k], 0, 0x4341);
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                const int ky = r - 2 * o;
                if (ky < 0 || ky > 4) continue;
                ev[o][k] += w5[ky] * e;
                if (k < 3) od[o][k] += w5[ky] * u;
            }
        }
    }
#pragma unroll
    for (int o = 0; o < 2; ++o) {
        const int y = yb + o;
        if (y >= P.dh) break;
        const uint32_t(&e)[4] = ev[o];
        const uint32_t(&u)[3] = od[o];
        // outputs 0 | 1 (centres 4 | 6) and 2 | 3 (centres 8 | 10)
        const uint32_t e01 = __funnelshift_r(e[0], e[1], 16), e12 = __funnelshift_r(e[1], e[2], 16),
                       e23 = __funnelshift_r(e[2], e[3], 16);
        const uint32_t u01 = __funnelshift_r(u[0], u[1], 16), u12 = __funnelshift_r(u[1], u[2], 16);
        const uint32_t s0 = e01 + e12 + 6 * e[1] + 4 * (u01 + u[1]) + 0x00800080u;
        const uint32_t s1 = e12 + e23 + 6 * e[2] + 4 * (u12 + u[2]) + 0x00800080u;
        const uint32_t out = __byte_perm(s0, s1, 0x7531);
        uint8_t* dst = P.dst + (size_t)y * P.dstep + xb;
        if (np == 4 && (reinterpret_cast<uintptr_t>(dst) & 3u) == 0) {
            *reinterpret_cast<uint32_t*>(dst) = out;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j < np) dst[j] = (uint8_t)(out >> (8 * j));
        }
    }
}

// ---------------------------------------------------------------------------
// Features.  Census: 5x5, replicate borders, MSB first, dy-major, bit =
// neighbour < centre (src/sgm_kernels.cu:251-298).  BT: the Sobel-like
// x-gradient clipped to +-ftzero and offset by ftzero, as a byte
// (src/sgm_kernels.cu:94-118), plus for both the gradient and intensity
// channels the half-sample interval [lo, hi] of dev_bt_channel_cost
// (src/sgm_kernels.cu:1002-1028) with clamped neighbours.  Census pixels
// store their 25-bit descriptor as one word per pixel; BT pixels store four
// words of signed 16-bit pairs (gradient low half, intensity high half):
// value, -value, lo, -hi -- the operands of bt_pixel().
//
// The view-0 blocks also start the level: every pixel's disp2 key is
// cleared, and on refine levels the label base is derived from the parent
// level (kernel_PrepareRefineLabels, src/sgm_kernels.cu:955-1000; a
// rejected parent -- invalid disparity or confidence below the minimum --
// becomes kNoParent: every label of the pixel is invalid).
//
// One block: 128 x 8 pixels of one view, a warp per row.  The image tile
// with its 2-pixel border (4 columns on each side, so rows stay word
// aligned) is staged as words, byte by byte only those with replicated
// columns.  Census: a thread
// per 4 adjacent pixels, 16-byte stores.  BT: gradients of 4 adjacent pixels
// per thread on 16-bit pairs, laid down with the intensities as one word per
// pixel; then a thread per pixel, 32 apart, makes the intervals of both
// channels at once from three words and stores 16 bytes beside its
// neighbour's (a thread storing the features of 4 adjacent pixels kept L1
// busy with quarter-line requests: 26 us for the two views of a 1080p level).
// The parent's values are loaded before the tile is waited for.
// ---------------------------------------------------------------------------
constexpr int kFtX = 128, kFtY = 8;
constexpr int kFtSWB = kFtX + 8;        // staged bytes per row: image columns x0 - 4 .. x0 + 131
constexpr int kFtSWW = kFtSWB / 4;      // ... as words
constexpr int kFtSH = kFtY + 4;         // staged rows: y0 - 2 .. y0 + 9
constexpr int kFtGW = kFtX + 8;         // gradient words per row: columns x0 - 4 ..

__device__ __forceinline__ uint32_t byte_of(uint32_t w, int k) { return (w >> (8 * k)) & 0xffu; }

// Label base of pixel x from its parent (the body of
// kernel_PrepareRefineLabels).
__device__ __forceinline__ int16_t refine_base(const LevelDesc& J, int x, int raw, float conf)
{
    const int16_t pinv = (int16_t)((J.minD - 1) * 16);
    if (raw == pinv || conf < J.minConf) return kNoParent;
    const int pred16 = raw * 2;
    const int center = (pred16 + 8) >> 4;
    const int resid = pred16 - center * 16;
    int base = center + (resid < 0 ? -(J.D / 2) : -(J.D / 2) + 1);
    const int physMax = imin(J.maxD, x);
    const int largest = physMax - J.D + 1;
    base = largest >= J.minD ? imin(imax(base, J.minD), largest) : J.minD;
    return (int16_t)base;
}

template <int NJ>
__global__ void __launch_bounds__(256) k_features(const __grid_constant__ Jobs<NJ> jobs)
{
    // (the strips of a BT level of fixed disparities are a few even waves)
    if (jobs.d[0].refine || jobs.d[0].cost == COST_CENSUS) let_next_in();
    after_previous();
    const LevelDesc& J = jobs.d[blockIdx.z >> 1];
    const int view = blockIdx.z & 1;
    const int x0 = blockIdx.x * kFtX, y0 = blockIdx.y * kFtY;
    if (x0 >= J.w || y0 >= J.h) return;
    const uint8_t* img = view ? J.right : J.left;
    const int step = view ? J.rstep : J.lstep;
    uint4* feat = view ? J.featR : J.featL;
    const int W = J.w, H = J.h;

    __shared__ uint32_t tw[kFtSH][kFtSWW];   // byte c of row r: image pixel (y0 - 2 + r, x0 - 4 + c), clamped
    __shared__ __align__(16) uint32_t gi[kFtY][kFtGW];   // BT: gradient | intensity << 16 of column x0 - 4 + c
    if (NJ > 1 && blockIdx.x + blockIdx.y + view + threadIdx.x == 0 && J.rewalked) *J.rewalked = 0;
    const int tx = threadIdx.x & 31, rr = threadIdx.x >> 5;
    const int xb = x0 + 4 * tx, y = y0 + rr;
    const int np = y < H ? imin(4, W - xb) : 0;     // pixels of this thread inside the image
    const bool vec = np == 4 && (W & 3) == 0;       // 16-byte stores of 4 words / 8-byte of 4 int16
    // the parent's values of this thread's pixels
    int praw[4];
    float pcf[4];
    if (view == 0 && J.refine && np > 0) {
        const int py = imin(y >> 1, J.ph - 1);
        const int16_t* prow = J.pdisp + (size_t)py * J.pd_pitch;
        const float* crow = J.pconf + (size_t)py * J.pc_pitch;
#pragma unroll
        for (int j = 0; j < 2; ++j) {   // xb is even: pixels 2 j and 2 j + 1 have one parent
            const int px = imin((xb >> 1) + j, J.pw - 1);
            praw[2 * j] = praw[2 * j + 1] = prow[px];
            pcf[2 * j] = pcf[2 * j + 1] = crow[px];
        }
    }
    if (((reinterpret_cast<uintptr_t>(img) | (uintptr_t)step) & 3u) == 0) {
        const int c = x0 - 4 + 4 * tx;
        const bool in0 = c >= 0 && c + 4 <= W, in1 = tx < kFtSWW - 32 && c + 132 <= W;
#pragma unroll
        for (int r = rr; r < kFtSH; r += 8) {
            const uint32_t* q =
                reinterpret_cast<const uint32_t*>(img + (size_t)iclamp(y0 - 2 + r, 0, H - 1) * step + x0 - 4) + tx;
            if (in0) tw[r][tx] = *q;
            if (in1) tw[r][tx + 32] = q[32];
        }
        // the words with columns outside that a pixel needs: the first one, and from `from` on
        const int left = x0 == 0 ? 1 : 0, from = imax((W - x0 + 4) >> 2, left);
        const int last = (imin(x0 + kFtX, W) + 5 - x0) >> 2;   // (two columns past the last pixel)
        const int edge = left + imax(0, imin(last + 1, kFtSWW) - from);
        for (int i = threadIdx.x; i < kFtSH * edge; i += 256) {
            const int r = i / edge, m = i - r * edge, k = m < left ? 0 : from + m - left;
            const uint8_t* row = img + (size_t)iclamp(y0 - 2 + r, 0, H - 1) * step;
            uint32_t v = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) v |= (uint32_t)row[iclamp(x0 - 4 + 4 * k + j, 0, W - 1)] << (8 * j);
            tw[r][k] = v;
        }
    } else {
        const uint8_t* const end = img + (size_t)(H - 1) * step + W;
        for (int r = rr; r < kFtSH; r += 8) {
            const uint8_t* row = img + (size_t)iclamp(y0 - 2 + r, 0, H - 1) * step;
#pragma unroll
            for (int k = tx; k < kFtSWW; k += 32)
                tw[r][k] = load4(row, x0 - 4 + 4 * k, W, img, end, [&](int c) { return iclamp(c, 0, W - 1); });
        }
    }
    __syncthreads();
    if (y >= H) return;
    // The gradient (at most 1020) is a byte in the reference: with a cap from
    // 128 on, gradient + cap wraps.
    const int ftzero = imax(J.pfc, 15) | 1, clip = imin(ftzero, 1020), offset = ftzero & 255;
    {
        const size_t p = (size_t)y * W + xb;
        if (!PG_IN((size_t)y * W + x0, imin(kFtX, W - x0), (size_t)W * H, 9)) return;
        if (J.cost == COST_CENSUS) {
            // bit (dy, dx) of the 4 pixels at once: bytes 2 + dx .. 5 + dx of
            // the 12-byte row window, compared with the 4 centre bytes
            const uint32_t ctr = tw[rr + 2][tx + 1];
            const uint32_t ctr7 = ctr & 0x7f7f7f7fu;
            uint32_t acc[4] = {0u, 0u, 0u, 0u};   // 8 bits per byte lane, first bit highest
            int pos = 0;
#pragma unroll
            for (int dy = 0; dy < 5; ++dy) {
                const uint32_t w0 = tw[rr + dy][tx], w1 = tw[rr + dy][tx + 1], w2 = tw[rr + dy][tx + 2];
                const uint32_t n[5] = {__funnelshift_r(w0, w1, 16), __funnelshift_r(w0, w1, 24), w1,
                                       __funnelshift_r(w1, w2, 8), __funnelshift_r(w1, w2, 16)};
#pragma unroll
                for (int dx = 0; dx < 5; ++dx, ++pos) {
                    // unsigned a < b per byte (SWAR): the low seven bits by a
                    // subtraction that cannot borrow across bytes, then the top bits
                    const uint32_t a = n[dx];
                    const uint32_t d = (a | 0x80808080u) - ctr7;
                    const uint32_t lt = ((~a & ctr) | (~(a ^ ctr) & ~d)) & 0x80808080u;
                    acc[pos >> 3] = (acc[pos >> 3] << 1) | (lt >> 7);
                }
            }
            uint32_t cv[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                cv[j] = (byte_of(acc[0], j) << 17) | (byte_of(acc[1], j) << 9) | (byte_of(acc[2], j) << 1) |
                        byte_of(acc[3], j);
            uint32_t* out = reinterpret_cast<uint32_t*>(feat) + p;
            if (np <= 0) return;
            if (vec) {
                *reinterpret_cast<uint4*>(out) = make_uint4(cv[0], cv[1], cv[2], cv[3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (j < np) out[j] = cv[j];
            }
        } else {
            // columns xb - 1 .. xb + 4 of the three rows as 16-bit pairs
            // (xb - 1, xb), (xb + 1, xb + 2), (xb + 3, xb + 4)
            const uint32_t lim = (uint32_t)clip * 0x10001u, off2 = (uint32_t)offset * 0x10001u;
            uint32_t v[3] = {0u, 0u, 0u}, mid[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const uint32_t a = tw[rr + 1 + k][tx], m = tw[rr + 1 + k][tx + 1], z = tw[rr + 1 + k][tx + 2];
                const uint32_t q[3] = {__byte_perm(__byte_perm(a, m, 0x0043), 0, 0x4140), __byte_perm(m, 0, 0x4241),
                                       __byte_perm(__byte_perm(m, z, 0x0043), 0, 0x4140)};
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    v[i] += k == 1 ? 2 * q[i] : q[i];
                    if (k == 1) mid[i] = q[i];
                }
            }
            // gradient of column c: v(c + 1) - v(c - 1), clipped and offset
            uint32_t g[2];
#pragma unroll
            for (int i = 0; i < 2; ++i)
                g[i] = __vadd2(__vmaxs2(__vmins2(__vsub2(v[i + 1], v[i]), lim), __vsub2(0u, lim)), off2) & 0x00ff00ffu;
            // intensities (xb, xb + 1), (xb + 2, xb + 3)
            const uint32_t in0 = __byte_perm(mid[0], mid[1], 0x5432), in1 = __byte_perm(mid[1], mid[2], 0x5432);
            *reinterpret_cast<uint4*>(&gi[rr][4 + 4 * tx]) =
                make_uint4(__byte_perm(g[0], in0, 0x5410), __byte_perm(g[0], in0, 0x7632), __byte_perm(g[1], in1, 0x5410),
                           __byte_perm(g[1], in1, 0x7632));
            if (tx == 0 || tx == 31) {   // the columns beside the tile
                const uint8_t* tb = reinterpret_cast<const uint8_t*>(&tw[0][0]);
                const int c = tx == 0 ? 3 : kFtX + 4;   // staged column
                int d = 0;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const uint8_t* r = tb + (rr + 1 + k) * kFtSWB + c;
                    d += (k == 1 ? 2 : 1) * ((int)r[1] - (int)r[-1]);
                }
                gi[rr][c] = (uint32_t)((iclamp(d, -clip, clip) + offset) & 255) | (uint32_t)tb[(rr + 2) * kFtSWB + c] << 16;
            }
            __syncwarp();
            uint4* out = feat + (size_t)y * W;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                // the neighbour columns are clamped first (x - 1 -> 0 at the left border)
                const int x = x0 + tx + 32 * j, c = 4 + tx + 32 * j;
                if (x < W) {
                    const uint32_t u = gi[rr][c], l = gi[rr][x > 0 ? c - 1 : c], r = gi[rr][x + 1 < W ? c + 1 : c];
                    const uint32_t ul = ((u + l) >> 1) & 0x7fff7fffu, ur = ((u + r) >> 1) & 0x7fff7fffu;
                    const uint32_t lo = __vimin3_u16x2(ul, ur, u), hi = __vimax3_u16x2(ul, ur, u);
                    out[x] = make_uint4(u, __vsub2(0u, u), lo, __vsub2(0u, hi));
                }
            }
            if (np <= 0) return;
        }
        if (view == 0) {
            if (vec) {
                *reinterpret_cast<uint4*>(J.keys + p) = make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (j < np) J.keys[p + j] = 0xffffffffu;   // no disp2 candidate yet
            }
            if (J.refine) {
                int16_t b[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = refine_base(J, xb + j, praw[j], pcf[j]);
                int16_t* bo = J.base + p;
                if (vec) {
                    *reinterpret_cast<uint2*>(bo) =
                        make_uint2((uint32_t)(uint16_t)b[0] | ((uint32_t)(uint16_t)b[1] << 16),
                                   (uint32_t)(uint16_t)b[2] | ((uint32_t)(uint16_t)b[3] << 16));
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (j < np) bo[j] = b[j];
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Adaptive P2 table.  dev_adaptive_p2 (src/sgm_kernels.cu:63-74) depends on
// the pixels only through |I(p) - I(p-r)| in [0, 255]; the table holds its
// value for every difference, computed on the device with the same
// expression and the same intrinsic (__expf) so that each entry equals the
// reference's per-voxel value.
// ---------------------------------------------------------------------------
__device__ __noinline__ int adaptive_p2_value(int P2, int cur, int prev, float alpha, float beta,
                                              float lowerMult, float upperMult)
{
    const float diff = fabsf((float)(cur - prev));
    const float ratio = lowerMult + (1.0f + alpha - lowerMult) * __expf(-diff / beta);
    float adaptive = (float)P2 * ratio;
    const float lower = fmaxf(1.0f, (float)P2 * lowerMult);
    const float upper = (float)P2 * upperMult;
    adaptive = fminf(upper, fmaxf(lower, adaptive));
    return (int)(adaptive + 0.5f);
}

__global__ void k_p2_table(int* lut, int P2, float alpha, float beta, float lower, float upper)
{
    let_next_in();
    after_previous();
    const int i = threadIdx.x;
    if (i < 256) lut[i] = adaptive_p2_value(P2, i, 0, alpha, beta, lower, upper);
}

// ---------------------------------------------------------------------------
// Census cost volume.  Coarse / single-scale: kernel_CensusCost
// (src/sgm_kernels.cu:303-327), 24 when x - d - minD is outside the image.
// Refine: kernel_CensusCostLocal (src/sgm_kernels.cu:1112-1133), kMax for a
// geometry-invalid label.  A thread per pixel and eight labels, so that a
// warp stores whole lines whatever D is (a thread per pixel, its labels D * 2
// bytes from the next one's, took 42 us for 641x479 with 96 labels, 19 for
// 1080p with 16), of kCnRows rows, whose loads overlap.  The right
// descriptors of neighbouring threads overlap and come from L1.
// ---------------------------------------------------------------------------
constexpr int kCnRows = 4;

template <int NJ>
__global__ void __launch_bounds__(256) k_cost_census(const __grid_constant__ Jobs<NJ> jobs)
{
    after_previous();
    const LevelDesc& J = jobs.d[blockIdx.z];
    const int W = J.w, D = J.D, y0 = blockIdx.y * kCnRows;
    const int i = blockIdx.x * 256 + threadIdx.x;
    const int x = D == 16 ? i >> 1 : i / (D / 8);
    if (x >= W || y0 >= J.h) return;
    const int d0 = (i - x * (D / 8)) * 8;
    const int rows = imin(kCnRows, J.h - y0);
    const size_t p0 = (size_t)y0 * W + x;
    const uint32_t* const fl = reinterpret_cast<const uint32_t*>(J.featL);
    const uint32_t* const fr = reinterpret_cast<const uint32_t*>(J.featR);
    uint32_t cl[kCnRows];
    int off[kCnRows];
#pragma unroll
    for (int r = 0; r < kCnRows; ++r) {
        const size_t p = p0 + (size_t)(r < rows ? r : 0) * W;
        cl[r] = fl[p];
        off[r] = J.refine ? (int)J.base[p] : J.minD;
    }
#pragma unroll
    for (int r = 0; r < kCnRows; ++r) {
        if (r >= rows) break;
        const size_t p = p0 + (size_t)r * W;
        // label d reads right pixel x - off - d when lo <= d <= hi, else `fill`
        int lo, hi, fill;
        if (J.refine) {
            label_range(J, x, off[r], lo, hi);
            fill = kMax;
        } else {
            lo = imax(0, x - off[r] - (W - 1));
            hi = imin(D - 1, x - off[r]);
            fill = 24;
        }
        uint32_t c[8];
        const uint32_t* q = fr + (p - x) + (x - off[r] - d0);
        if (lo <= d0 && hi >= d0 + 7) {
#pragma unroll
            for (int k = 0; k < 8; ++k) c[k] = (uint32_t)__popc(cl[r] ^ q[-k]);
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k)
                c[k] = d0 + k >= lo && d0 + k <= hi ? (uint32_t)__popc(cl[r] ^ q[-k]) : (uint32_t)fill;
        }
        if (!PG_IN(p * D + d0, 8, (size_t)W * J.h * D, 10)) continue;
        *reinterpret_cast<uint4*>(J.C + p * D + d0) =
            make_uint4(c[0] | (c[1] << 16), c[2] | (c[3] << 16), c[4] | (c[5] << 16), c[6] | (c[7] << 16));
    }
}

// BT cost of one (left pixel, right pixel) pair: dev_bt_pixel_cost,
// src/sgm_kernels.cu:1030-1043, i.e. min(255, bt(gradient) + bt(intensity)
// >> 2) with bt(u, v) = min(max(0, u - v.hi, v.lo - u), max(0, v - u.hi,
// u.lo - v)), on both channels at once as 16-bit pairs: the features hold
// the negated operands, so each difference and maximum is one instruction.
// Seven in all.
__device__ __forceinline__ uint32_t bt_pixel(const uint4 l, const uint4 r)
{
    const uint32_t c0 = __viaddmax_s16x2(l.x, r.w, __viaddmax_s16x2(r.z, l.y, 0u));
    const uint32_t c1 = __viaddmax_s16x2(r.x, l.w, __viaddmax_s16x2(l.z, r.y, 0u));
    const uint32_t m = __vminu2(c0, c1);
    return __viaddmin_u16x2(m, m >> 18, 255u);   // the high half comes out 0
}

// A right feature whose cost against any left one is 255: right pixels
// outside the image.
__device__ __forceinline__ uint4 bt_outside() { return make_uint4(0x30003000u, 0u, 0x30003000u, 0u); }

__device__ __forceinline__ void tile_cp16(void* dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void tile_commit_wait()
{
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// ---------------------------------------------------------------------------
// BT coarse / single-scale cost: kernel_BTCost followed by kernel_BoxFilterH
// and kernel_BoxFilterV (src/sgm_kernels.cu:139-239, 354-416), fused.  The
// separable sums keep the reference's two saturation points:
//   C = min(MAX, sum_dy min(MAX, sum_dx bt(clamp(y+dy), clamp(x+dx), d))).
// One block: 32 x 8 output pixels x 16 labels.  bt values are staged in
// shared memory for the (8+2h) x (32+2h) window of clamped pixels.
// ---------------------------------------------------------------------------
constexpr int kBxX = 32, kBxY = 8, kBxD = 16;

template <int NJ>
__global__ void __launch_bounds__(256) k_cost_bt_box(const __grid_constant__ Jobs<NJ> jobs, int maxHalf, int nxt)
{
    after_previous();
    const LevelDesc& J = jobs.d[blockIdx.z];
    const int x0 = (blockIdx.x % nxt) * kBxX;
    const int d0 = (blockIdx.x / nxt) * kBxD;
    const int y0 = blockIdx.y * kBxY;
    if (x0 >= J.w || y0 >= J.h || d0 >= J.D) return;
    const int h = J.bs / 2;
    const int SW = kBxX + 2 * maxHalf, SH = kBxY + 2 * maxHalf;
    extern __shared__ unsigned char sm[];
    uint8_t* bt = sm;                                               // [SH][SW][kBxD]
    uint16_t* hs = reinterpret_cast<uint16_t*>(sm + ((SH * SW * kBxD + 15) & ~15));  // [SH][kBxX][kBxD]
    const int W = J.w, H = J.h;
    const int sw = kBxX + 2 * h, sh = kBxY + 2 * h;
    for (int i = threadIdx.x; i < sh * sw * kBxD; i += blockDim.x) {
        const int dd = i % kBxD;
        const int j = (i / kBxD) % sw;
        const int r = i / (kBxD * sw);
        const int gy = iclamp(y0 - h + r, 0, H - 1), gx = iclamp(x0 - h + j, 0, W - 1);
        const int x2 = gx - (d0 + dd + J.minD);
        int v = 255;
        if (x2 >= 0 && x2 < W) v = (int)bt_pixel(J.featL[(size_t)gy * W + gx], J.featR[(size_t)gy * W + x2]);
        bt[(r * SW + j) * kBxD + dd] = (uint8_t)v;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < sh * kBxX * kBxD; i += blockDim.x) {
        const int dd = i % kBxD;
        const int j = (i / kBxD) % kBxX;
        const int r = i / (kBxD * kBxX);
        int s = 0;
        for (int k = 0; k <= 2 * h; ++k) s += bt[(r * SW + j + k) * kBxD + dd];
        hs[(r * kBxX + j) * kBxD + dd] = (uint16_t)imin(kMax, s);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kBxY * kBxX * (kBxD / 2); i += blockDim.x) {
        const int dp = i % (kBxD / 2);
        const int j = (i / (kBxD / 2)) % kBxX;
        const int r = i / ((kBxD / 2) * kBxX);
        const int x = x0 + j, y = y0 + r;
        if (x >= W || y >= H) continue;
        int s0 = 0, s1 = 0;
        for (int k = 0; k <= 2 * h; ++k) {
            s0 += hs[((r + k) * kBxX + j) * kBxD + 2 * dp];
            s1 += hs[((r + k) * kBxX + j) * kBxD + 2 * dp + 1];
        }
        const uint32_t v = (uint32_t)imin(kMax, s0) | ((uint32_t)imin(kMax, s1) << 16);
        reinterpret_cast<uint32_t*>(J.C + ((size_t)y * W + x) * J.D + d0)[dp] = v;
    }
}

// ---------------------------------------------------------------------------
// The same for windows of 3 to 7 pixels, whose sums cannot reach either
// saturation point (49 * 255 < SHRT_MAX), so that they may be taken in any
// grouping.  A block owns 64 (label, 32-column segment) units of 4 labels x
// 8 window rows: db labels (16, 32, 48 or 64) by 32 * nseg columns, and walks
// down a strip of rows, 8 window rows at a time:
//   staging: the features of the 8 rows (cp.async); right pixel p of a row
//            lies at [p & 3][p >> 2], so that the threads of a row, four
//            pixels apart, read adjacent 16-byte words;
//   phase 1: a thread per (row, 4 labels, segment) walks the 32 + 2 HW
//            window columns; label d + 1 needs at a column the right feature
//            that d needed one column before, so one left and one right
//            feature are loaded per column for four costs; running sums of
//            the last 2 HW + 1 costs, two labels per word, go to shared
//            memory;
//   phase 2: a thread per (4 columns, 4 labels) keeps the running column
//            sums and the last 2 HW rows of its sums in registers across the
//            strip: adds a row, stores the costs, takes off the row 2 HW
//            before.  The next rows' features are copied meanwhile.
// The ALU pipe bounds it (half of its instructions): 133 us for 720p with
// 128 labels and 5x5 windows (884 in k_cost_bt_box); four blocks per SM at
// 128 registers were slower than three at 168 (153 us), and so were the old
// rows' sums read back from shared memory (162 us).
// ---------------------------------------------------------------------------
constexpr int kBsThreads = 128, kBsRows = 8, kBsSeg = 32;
__host__ __device__ constexpr int bs_segments(int db) { return db <= 16 ? 4 : db <= 32 ? 2 : 1; }
// staged features of one row: left, right (a multiple of 4)
template <int HW>
__host__ __device__ constexpr int bs_left(int db) { return kBsSeg * bs_segments(db) + 2 * HW; }
template <int HW>
__host__ __device__ constexpr int bs_right(int db) { return (bs_left<HW>(db) + db - 1 + 3) / 4 * 4; }
template <int HW>
__host__ __device__ constexpr size_t bs_smem(int db)
{
    return (size_t)kBsRows * kBsSeg * bs_segments(db) * db * 2 +
           (size_t)kBsRows * (bs_left<HW>(db) + bs_right<HW>(db)) * 16 + 256;   // (a turn reads past the window)
}

template <int HW, int NJ>
__global__ void __launch_bounds__(kBsThreads) k_cost_bt_strip(const __grid_constant__ Jobs<NJ> jobs, int strip)
{
    after_previous();
    constexpr int SW = kBsSeg + 2 * HW;
    constexpr int U = HW == 3 ? 12 : 4;   // columns per turn: a multiple of 4 right features and 2 HW costs kept
    const LevelDesc& J = jobs.d[blockIdx.z];
    const int W = J.w, H = J.h, D = J.D;
    const int nblk = (D + 63) / 64, db = ((D + nblk - 1) / nblk + 15) / 16 * 16;
    const int nseg = bs_segments(db), TX = kBsSeg * nseg, ntx = (W + TX - 1) / TX;
    const int bd = blockIdx.x / ntx, x0 = (blockIdx.x - bd * ntx) * TX, y0 = blockIdx.y * strip;
    const int d0 = bd * db;
    if (d0 >= D || y0 >= H) return;
    const int nd = imin(db, D - d0), DQ = nd / 4;   // labels and label quads of this block
    extern __shared__ __align__(16) unsigned char smb[];
    uint16_t* sums = reinterpret_cast<uint16_t*>(smb);                   // [rows][TX][db]
    uint4* sl = reinterpret_cast<uint4*>(smb + (size_t)kBsRows * TX * db * 2);   // [rows][nsl]
    const int nsl = TX + 2 * HW, nsr = nsl + nd - 1, srs = (nsr + 3) / 4;
    uint4* sr = sl + kBsRows * nsl;                                      // [rows][4][srs]
    const int xrs = x0 - HW - (d0 + J.minD + nd - 1);                    // image column of right pixel 0
    // no window column is clamped
    const bool interior = x0 - HW >= 0 && x0 + TX - 1 + HW < W;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    // phase 1 unit
    const int q = t % DQ, rs = t / DQ, r1 = rs % kBsRows, seg = rs / kBsRows;
    const bool unit = seg < nseg;
    // phase 2 items: columns xq + step * i, label quad q
    const int step = kBsThreads / DQ, xq = rs;
    constexpr int kItems = kBsSeg * 16 / kBsThreads;   // columns per thread at 16 quads per segment
    const int items = t < step * DQ ? (TX - xq + step - 1) / step : 0;
    uint2 run[kItems], before[kItems][2 * HW];
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        run[i] = make_uint2(0u, 0u);
#pragma unroll
        for (int k = 0; k < 2 * HW; ++k) before[i][k] = make_uint2(0u, 0u);
    }
    const int y1 = imin(y0 + strip, H);
    const int nrow = y1 - y0 + 2 * HW;                 // window rows of the strip; whole turns of 8 are walked
    auto stage = [&](int w0) {                         // a warp per row
        for (int r = warp; r < kBsRows; r += kBsThreads / 32) {
            const size_t grow = (size_t)iclamp(y0 - HW + w0 + r, 0, H - 1) * W;
            for (int j = lane; j < nsl; j += 32)
                tile_cp16(sl + r * nsl + j, J.featL + grow + iclamp(x0 - HW + j, 0, W - 1));
            uint4* o = sr + (size_t)r * 4 * srs + (lane & 3) * srs + (lane >> 2);
            for (int p = lane; p < nsr; p += 32, o += 8) {
                const int xx = xrs + p;
                if (xx >= 0 && xx < W) tile_cp16(o, J.featR + grow + xx);
                else *o = bt_outside();
            }
        }
    };
    int16_t* orow = J.C + ((long long)(y0 - 2 * HW) * W + x0 + xq) * D + d0 + 4 * q;   // of window row w0
    stage(0);
    for (int w0 = 0; w0 < nrow; w0 += kBsRows) {
        tile_commit_wait();
        __syncthreads();
        if (unit) {
            const uint4* lrow = sl + r1 * nsl + seg * kBsSeg;
            const uint4* rrow = sr + r1 * 4 * srs;
            uint16_t* out = sums + (r1 * TX + seg * kBsSeg) * db + 4 * q;
            uint32_t h0[2 * HW], h1[2 * HW], s0 = 0, s1 = 0;
#pragma unroll
            for (int i = 0; i < 2 * HW; ++i) h0[i] = h1[i] = 0;
            // add the four labels' costs of column j (u: its place in the turn)
            auto column = [&](int j, int u, const uint32_t (&e)[4]) {
                const uint32_t p0 = e[0] | (e[1] << 16), p1 = e[2] | (e[3] << 16);
                s0 += p0;
                s1 += p1;
                if (j >= 2 * HW && j < SW)
                    *reinterpret_cast<uint2*>(out + (size_t)(j - 2 * HW) * db) = make_uint2(s0, s1);
                s0 -= h0[u % (2 * HW)];
                s1 -= h1[u % (2 * HW)];
                h0[u % (2 * HW)] = p0;
                h1[u % (2 * HW)] = p1;
            };
            if (interior) {
                // label d0 + 4 q + i needs right pixel top + j - i at window
                // column j; top is 3 modulo 4
                const int top = seg * kBsSeg + nd - 1 - 4 * q;
                const uint4* rp = rrow + (top >> 2);
                uint4 win[4];   // right pixel p at p & 3
#pragma unroll
                for (int i = 1; i < 4; ++i) win[(3 - i) & 3] = rp[((3 - i) & 3) * srs];
#pragma unroll 1
                for (int j0 = 0; j0 < SW; j0 += U) {
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const uint4 l = lrow[j0 + u];
                        win[(3 + u) & 3] = rp[((3 + u) & 3) * srs + ((3 + u) >> 2)];
                        uint32_t e[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) e[i] = bt_pixel(l, win[(3 + u - i) & 3]);
                        column(j0 + u, u, e);
                    }
                    rp += U / 4;
                }
            } else {
#pragma unroll 1
                for (int j0 = 0; j0 < SW; j0 += 2 * HW) {
#pragma unroll
                    for (int u = 0; u < 2 * HW; ++u) {
                        const int gx = iclamp(x0 - HW + seg * kBsSeg + j0 + u, 0, W - 1);
                        const int p = gx - (d0 + J.minD + 4 * q) - xrs;
                        const uint4 l = lrow[j0 + u];
                        uint32_t e[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) e[i] = bt_pixel(l, rrow[((p - i) & 3) * srs + ((p - i) >> 2)]);
                        column(j0 + u, u, e);
                    }
                }
            }
        }
        __syncthreads();
        if (w0 + kBsRows < nrow) stage(w0 + kBsRows);   // its copies run beside phase 2
        const uint16_t* add = sums + xq * db + 4 * q;
#pragma unroll
        for (int r = 0; r < kBsRows; ++r) {
            const int wr = w0 + r;
            const bool put = wr >= 2 * HW && wr < nrow;
#pragma unroll
            for (int i = 0; i < kItems; ++i) {
                if (i < items) {
                    const uint2 a = *reinterpret_cast<const uint2*>(add + (r * TX + step * i) * db);
                    run[i].x += a.x;
                    run[i].y += a.y;
                    if (put && x0 + xq + step * i < W && PG_IN(orow - J.C + (long long)step * i * D, 4, (size_t)W * H * D, 13))
                        *reinterpret_cast<uint2*>(orow + (size_t)(step * i) * D) = run[i];
                    run[i].x -= before[i][0].x;
                    run[i].y -= before[i][0].y;
#pragma unroll
                    for (int k = 0; k + 1 < 2 * HW; ++k) before[i][k] = before[i][k + 1];
                    before[i][2 * HW - 1] = a;
                }
            }
            orow += (size_t)W * D;
        }
    }
}

// ---------------------------------------------------------------------------
// BT refine cost: kernel_BTWindowCostLocal, src/sgm_kernels.cu:1075-1110.
// For label d of pixel p the reference sums, over the blockSize^2 window of
// clamped pixels q, the BT cost of q at the real disparity base_p + d (255
// when q - (base_p + d) leaves the image), clamps the sum to kMax - 1, and
// writes kMax for a geometry-invalid label.  The sum depends on p only
// through the window and the real disparity, so one 32x16 tile evaluates
// each (window pixel, real disparity) pair once, 16 labels at a time and one
// pass per cluster of bases: the pixels whose real disparities span at most
// kTiRn.  Most tiles are one cluster.  A pass:
//   staging: the features of the window rows of the cluster (left: one per
//            window column, clamped; right: the ones its disparities reach)
//            are copied once into shared memory with cp.async, a warp per
//            row; right pixels outside the image get a feature of cost 255;
//   phase 1: a lane takes four adjacent real disparities of a window row and
//            half of the tile's columns, walks the window columns left to
//            right and keeps the running sums of the last blockSize costs
//            (sums along x, into shared memory).  Disparity i + 1 needs at
//            column j the right feature that i needed at column j - 1, so it
//            loads one left and one right feature per column for four costs.
//            A tile usually needs 17 real disparities: 200 units of 20
//            columns for 256 lanes;
//   phase 2: a thread per two vertical neighbours adds blockSize rows of
//            those sums for each, two labels per 32-bit add, from their
//            real-disparity offset.  The two have one parent and so one
//            offset, and share all but two of their window rows.
// Later passes of a tile hold few pixels: only the rows and the column
// halves with pixels of the cluster are staged and summed.
// Window sums are exact integers (at most 25 * 255 here, no intermediate
// clamp in the reference).  What is left after kTiClusters passes and wider
// windows evaluate each window directly.
// Bound by the integer pipe (seven instructions a cost; 62 %) and the
// barriers between the phases, three blocks per SM.  The base level of a
// 1080p pair: 158 us with direct sums for wide tiles, 98 with clusters, 94
// with four disparities a lane instead of two (which kept the shared-memory
// pipe at 64 %), 87 with the reductions, the staging and the shared rows as
// they are now.
// ---------------------------------------------------------------------------
constexpr int kTiX = 32, kTiY = 16, kTiMaxHalf = 2;
constexpr int kTiD = 16;         // labels of a pass
constexpr int kTiRn = 28;        // real disparities of a cluster
constexpr int kTiWarps = 8;
constexpr int kTiClusters = 8;   // passes of a tile
constexpr int kTiRows = kTiY + 2 * kTiMaxHalf;      // window rows at most
// Sums along x of a row: 14 words a column (7 pairs of words, odd, so that
// the columns' 8-byte reads hit distinct banks), the rows 10 words further
// (5 pairs: the writes of the lanes of five quads and three rows do too).
constexpr int kTiCs = kTiRn / 2, kTiRowS = kTiX * kTiCs + 10;
constexpr int kTiSeg = kTiX / 2;                    // columns a lane walks (without the window's border)
constexpr int kTiSL = kTiX + 2 * kTiMaxHalf;        // staged left features per window row
// Staged right features: pixel p of a row at (p & 3) * kTiSub + (p >> 2), so
// that lanes of adjacent quads read adjacent ones.
constexpr int kTiSub = 17, kTiSR = 4 * kTiSub - 1;
constexpr size_t kTiHs = (size_t)kTiRows * kTiRowS * 4;
constexpr size_t kTiSmem = kTiHs + (size_t)kTiRows * (kTiSL + kTiSR) * 16;
static_assert(kTiHs % 16 == 0, "the staged features are 16-byte aligned");
static_assert((kTiSL + kTiRn - 2) / 4 < kTiSub, "the right features of a row fit");
static_assert(kTiD + kTiRn % 4 <= kTiRn && kTiRn % 4 == 0, "whole quads");

// The part of a tile that a cluster's pixels cover.
struct TileArea {
    int r0, nr;     // window rows
    int seg0, ns;   // column halves
};

// Sums along x, for the 4 nq real disparities from rmin on, of the window
// rows and column halves of `a` (see above).
template <int HW>
__device__ __forceinline__ void bt_row_sums(const LevelDesc& J, uint32_t* hs, uint4* st, int x0, int y0, int rmin,
                                            int nq, const TileArea& a, int warp, int lane)
{
    constexpr int SW = kTiX + 2 * HW;    // window columns
    constexpr int NC = kTiSeg + 2 * HW;  // ... of a half
    constexpr int Q = HW > 0 ? 2 * HW : 1;
    const int W = J.w, H = J.h;
    uint4* sl = st;                      // [R][kTiSL]  left, columns x0 - HW + j (clamped)
    uint4* sr = st + kTiRows * kTiSL;    // [R][kTiSR]  right, columns xrs + p
    const int xrs = x0 - HW - (rmin + 4 * nq - 1);
    const int nsr = SW + 4 * nq - 1;
    // a warp per row; the columns (and which are outside) are those of every row
    const int gl0 = iclamp(x0 - HW + lane, 0, W - 1), gl1 = imin(x0 - HW + 32 + lane, W - 1);
    const int xr0 = xrs + lane, xr1 = xr0 + 32;
    const bool in0 = xr0 >= 0 && xr0 < W, in1 = xr1 >= 0 && xr1 < W, more = lane + 32 < nsr;
    for (int r = a.r0 + warp; r < a.r0 + a.nr; r += kTiWarps) {
        const size_t grow = (size_t)iclamp(y0 - HW + r, 0, H - 1) * W;
        const uint4 *fl = J.featL + grow, *fr = J.featR + grow;
        uint4* o = sr + r * kTiSR + (lane & 3) * kTiSub + (lane >> 2);
        tile_cp16(sl + r * kTiSL + lane, fl + gl0);
        if (lane < SW - 32) tile_cp16(sl + r * kTiSL + 32 + lane, fl + gl1);
        if (in0) tile_cp16(o, fr + xr0);
        else *o = bt_outside();
        if (more) {
            if (in1) tile_cp16(o + 8, fr + xr1);
            else o[8] = bt_outside();
        }
    }
    tile_commit_wait();
    __syncthreads();
    // no window column is clamped
    const bool interior = x0 - HW >= 0 && x0 + kTiX - 1 + HW < W;
    const int units = a.nr * nq * a.ns;
    for (int f = warp * 32 + lane; f < units; f += kTiWarps * 32) {
        const int t = f / nq, q = f - t * nq;
        const bool second = t >= a.nr;
        const int row = a.r0 + (second ? t - a.nr : t), j0 = (a.seg0 + (second ? 1 : 0)) * kTiSeg;
        const uint4* lp = sl + row * kTiSL + j0;
        const uint4* rrow = sr + row * kTiSR;
        uint2* out = reinterpret_cast<uint2*>(hs + row * kTiRowS + j0 * kTiCs + 2 * q);
        uint32_t h0[Q], h1[Q], s0 = 0, s1 = 0;   // the last 2 HW costs; their sums
#pragma unroll
        for (int i = 0; i < Q; ++i) h0[i] = h1[i] = 0;
        // add the four costs of window column j of the half (u: its place in the turn)
        auto column = [&](int j, int u, const uint32_t (&e)[4]) {
            const uint32_t p0 = e[0] | (e[1] << 16), p1 = e[2] | (e[3] << 16);
            s0 += p0;
            s1 += p1;
            if (j >= 2 * HW) {
                *out = make_uint2(s0, s1);
                out += kTiCs / 2;
            }
            s0 -= HW > 0 ? h0[u % Q] : p0;
            s1 -= HW > 0 ? h1[u % Q] : p1;
            h0[u % Q] = p0;
            h1[u % Q] = p1;
        };
        if (interior) {
            // disparity rmin + 4 q + i needs right pixel j0 + 4 (nq - q) - 1 + j - i at column j
            const uint4* rp = rrow + (j0 >> 2) + nq - 1 - q;
            uint4 win[4];   // right pixel p at p & 3
#pragma unroll
            for (int i = 1; i < 4; ++i) win[(3 - i) & 3] = rp[((3 - i) & 3) * kTiSub];
#pragma unroll 1
            for (int j = 0; j < NC; j += 4) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (NC % 4 != 0 && j + u >= NC) break;
                    const uint4 l = lp[j + u];
                    win[(3 + u) & 3] = rp[((3 + u) & 3) * kTiSub + ((3 + u) >> 2)];
                    uint32_t e[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) e[i] = bt_pixel(l, win[(3 + u - i) & 3]);
                    column(j + u, u, e);
                }
                ++rp;
            }
        } else {
#pragma unroll 1
            for (int j = 0; j < NC; j += Q) {
#pragma unroll
                for (int u = 0; u < Q; ++u) {
                    const int p = iclamp(x0 - HW + j0 + j + u, 0, W - 1) - (rmin + 4 * q) - xrs;
                    const uint4 l = lp[j + u];
                    uint32_t e[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) e[i] = bt_pixel(l, rrow[((p - i) & 3) * kTiSub + ((p - i) >> 2)]);
                    column(j + u, u, e);
                }
            }
        }
    }
}

template <int NJ>
__global__ void __launch_bounds__(256, 3) k_cost_bt_tiled(const __grid_constant__ Jobs<NJ> jobs)
{
    after_previous();
    const LevelDesc& J = jobs.d[blockIdx.z];
    const int x0 = blockIdx.x * kTiX, y0 = blockIdx.y * kTiY;
    if (x0 >= J.w || y0 >= J.h) return;
    const int W = J.w, H = J.h, D = J.D, h = J.bs / 2;
    extern __shared__ __align__(16) uint32_t hs[];   // [kTiRows] rows of sums, then the staged features
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint4* stg = reinterpret_cast<uint4*>(reinterpret_cast<unsigned char*>(hs) + kTiHs);
    __shared__ int wred[3][kTiWarps];
    // a thread's two pixels: (x0 + lane, y0 + 2 warp) and the one below
    const int x = x0 + lane;
    int yq[2], bq[2];
    bool inq[2], hasq[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        yq[i] = y0 + 2 * warp + i;
        inq[i] = x < W && yq[i] < H;
        bq[i] = inq[i] ? (int)J.base[(size_t)yq[i] * W + x] : (int)kNoParent;
        hasq[i] = inq[i] && bq[i] != kNoParent;
    }
    // lowest and highest base of the pixels in0, in1, and where they lie
    auto block_minmax = [&](bool in0, bool in1, int& mn, int& mx, TileArea& area) {
        const int a = __reduce_min_sync(0xffffffffu, imin(in0 ? bq[0] : INT_MAX, in1 ? bq[1] : INT_MAX));
        const int z = __reduce_max_sync(0xffffffffu, imax(in0 ? bq[0] : INT_MIN, in1 ? bq[1] : INT_MIN));
        const unsigned m = __ballot_sync(0xffffffffu, in0 || in1);
        __syncthreads();   // wred reused
        if (lane == 0) { wred[0][warp] = a; wred[1][warp] = z; wred[2][warp] = (int)m; }
        __syncthreads();
        const int l8 = lane & (kTiWarps - 1);
        mn = __reduce_min_sync(0xffffffffu, wred[0][l8]);
        mx = __reduce_max_sync(0xffffffffu, wred[1][l8]);
        const unsigned c = (unsigned)wred[2][l8], cols = __reduce_or_sync(0xffffffffu, c);
        const unsigned rows = __ballot_sync(0xffffffffu, c != 0) & ((1u << kTiWarps) - 1);
        const int first = __ffs((int)rows) - 1, last = 31 - __clz((int)rows);
        area.r0 = 2 * first;
        area.nr = 2 * (last - first + 1) + 2 * h;
        area.seg0 = (cols & 0xffffu) ? 0 : 1;
        area.ns = (cols & 0xffffu) && (cols >> 16) ? 2 : 1;
    };
    const bool vec = (D & 7) == 0;
    for (int dc = 0; dc < D; dc += kTiD) {
        const int nd = imin(kTiD, D - dc);
        // Clusters of bases, lowest first: the pixels whose real disparities
        // lie within kTiRn of the lowest one left.  11-26 % of the tiles of a
        // 1080p scene hold a depth edge or a wild parent and need more than
        // one; a pass costs less than the window sums of a few pixels, and
        // two passes at most left 1-2 % of the pixels to those (a seventh of
        // the kernel's instructions, in blocks that outlasted the others).
        const bool tiled = h >= 0 && h <= kTiMaxHalf;   // (a negative block size: an empty window)
        bool todo[2] = {hasq[0] && tiled, hasq[1] && tiled};
        for (int c = 0; c < kTiClusters; ++c) {
            int low, top;
            TileArea area;
            block_minmax(todo[0], todo[1], low, top, area);
            if (top == INT_MIN) break;
            if (top + nd - low > kTiRn) {
                const int last = low + kTiRn - nd;
                int lowest;
                block_minmax(todo[0] && bq[0] <= last, todo[1] && bq[1] <= last, lowest, top, area);
            }
            const int rmin = low + dc, nq = (top + nd - low + 3) >> 2;
            const bool mine[2] = {todo[0] && bq[0] <= top, todo[1] && bq[1] <= top};
            if (h == 2) bt_row_sums<2>(J, hs, stg, x0, y0, rmin, nq, area, warp, lane);
            else if (h == 1) bt_row_sums<1>(J, hs, stg, x0, y0, rmin, nq, area, warp, lane);
            else bt_row_sums<0>(J, hs, stg, x0, y0, rmin, nq, area, warp, lane);
            __syncthreads();
            // the 16 labels of pixel i from its pair sums, which start
            // `off` (0 to 3) halves before its first label
            auto put = [&](int i, uint32_t (&acc)[10], int off, int lo, int hi) {
                int16_t* out = J.C + ((size_t)yq[i] * W + x) * D + dc;
                if (!PG_IN(((size_t)yq[i] * W + x) * D, D, (size_t)W * H * D, 11)) return;
                const bool two = off & 2;
#pragma unroll
                for (int q = 0; q < 9; ++q) acc[q] = two ? acc[q + 1] : acc[q];
                const uint32_t sh = (uint32_t)(off & 1) * 16;
                uint32_t w[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) w[q] = __funnelshift_r(acc[q], acc[q + 1], sh);
                if (lo > dc || hi < dc + nd - 1) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const int d = dc + 2 * q;
                        if (d < lo || d > hi) w[q] = (w[q] & 0xffff0000u) | (uint32_t)kMax;
                        if (d + 1 < lo || d + 1 > hi) w[q] = (w[q] & 0xffffu) | ((uint32_t)kMax << 16);
                    }
                }
                if (vec) {
                    reinterpret_cast<uint4*>(out)[0] = make_uint4(w[0], w[1], w[2], w[3]);
                    if (nd > 8) reinterpret_cast<uint4*>(out)[1] = make_uint4(w[4], w[5], w[6], w[7]);
                } else {
#pragma unroll
                    for (int q = 0; q < 16; ++q)
                        if (q < nd) out[q] = (int16_t)((w[q >> 1] >> ((q & 1) * 16)) & 0xffffu);
                }
            };
            auto rowsum = [&](int k, int o, uint32_t (&v)[10]) {   // window row k, from disparity offset o & ~3
                const uint2* p = reinterpret_cast<const uint2*>(hs + k * kTiRowS + lane * kTiCs) + (o >> 2);
#pragma unroll
                for (int j = 0; j < 5; ++j) {
                    const uint2 a = p[j];
                    v[2 * j] = a.x;
                    v[2 * j + 1] = a.y;
                }
            };
            if (mine[0] && mine[1] && bq[0] == bq[1]) {
                int lo, hi;
                label_range(J, x, bq[0], lo, hi);
                const int o = bq[0] - low;
                uint32_t above[10], below[10];
#pragma unroll
                for (int j = 0; j < 10; ++j) below[j] = 0;
                for (int k = 1; k <= 2 * h; ++k) {   // the rows both windows hold
                    uint32_t v[10];
                    rowsum(2 * warp + k, o, v);
#pragma unroll
                    for (int j = 0; j < 10; ++j) below[j] += v[j];
                }
                uint32_t v[10];
                rowsum(2 * warp, o, above);
                rowsum(2 * warp + 2 * h + 1, o, v);
#pragma unroll
                for (int j = 0; j < 10; ++j) {
                    above[j] += below[j];
                    below[j] += v[j];
                }
                put(0, above, o & 3, lo, hi);
                put(1, below, o & 3, lo, hi);
            } else {
#pragma unroll 1
                for (int i = 0; i < 2; ++i) {
                    if (!(i ? mine[1] : mine[0])) continue;
                    const int bb = i ? bq[1] : bq[0];
                    int lo, hi;
                    label_range(J, x, bb, lo, hi);
                    uint32_t acc[10];
                    rowsum(2 * warp + i, bb - low, acc);
                    for (int k = 1; k <= 2 * h; ++k) {
                        uint32_t v[10];
                        rowsum(2 * warp + i + k, bb - low, v);
#pragma unroll
                        for (int j = 0; j < 10; ++j) acc[j] += v[j];
                    }
                    if (i) put(1, acc, (bb - low) & 3, lo, hi);
                    else put(0, acc, (bb - low) & 3, lo, hi);
                }
            }
            todo[0] = todo[0] && !mine[0];
            todo[1] = todo[1] && !mine[1];
            // (the next cluster's reductions come before its row sums overwrite hs)
        }
        // direct window per pixel (no parent, or in no cluster)
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
            const bool in = i ? inq[1] : inq[0], has = i ? hasq[1] : hasq[0], left = i ? todo[1] : todo[0];
            if (!in || (has && !left && tiled)) continue;
            const int y = i ? yq[1] : yq[0], b = i ? bq[1] : bq[0];
            int lo, hi;
            label_range(J, x, b, lo, hi);
            int16_t* out = J.C + ((size_t)y * W + x) * D;
            for (int d0 = dc; d0 < dc + nd; d0 += 8) {
                int sum[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                if (b != kNoParent) {
                    for (int dy = -h; dy <= h; ++dy) {
                        const int gy = iclamp(y + dy, 0, H - 1);
                        const uint4* lrow = J.featL + (size_t)gy * W;
                        const uint4* rrow = J.featR + (size_t)gy * W;
                        for (int dx = -h; dx <= h; ++dx) {
                            const int gx = iclamp(x + dx, 0, W - 1);
                            const uint4 lf = lrow[gx];
    #pragma unroll
                            for (int q = 0; q < 8; ++q) {
                                const int x2 = gx - (b + d0 + q);
                                sum[q] += (x2 >= 0 && x2 < W) ? (int)bt_pixel(lf, rrow[x2]) : 255;
                            }
                        }
                    }
                }
                uint32_t w[4];
    #pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int d = d0 + 2 * q;
                    const uint32_t v0 = (d >= lo && d <= hi) ? (uint32_t)imin(sum[2 * q], kMax - 1) : (uint32_t)kMax;
                    const uint32_t v1 =
                        (d + 1 >= lo && d + 1 <= hi) ? (uint32_t)imin(sum[2 * q + 1], kMax - 1) : (uint32_t)kMax;
                    w[q] = v0 | (v1 << 16);
                }
                if (vec) {
                    reinterpret_cast<uint4*>(out + d0)[0] = make_uint4(w[0], w[1], w[2], w[3]);
                } else {
                    for (int q = 0; q < 8 && d0 + q < D; ++q) out[d0 + q] = (int16_t)((w[q >> 1] >> ((q & 1) * 16)) & 0xffffu);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
template <int NB>
cudaError_t launch_pyrdown(const PyrDownBatch<NB>& b, int max_dw, int max_dh, cudaStream_t st)
{
    dim3 grid((max_dw + kPdX - 1) / kPdX, (max_dh + kPdY - 1) / kPdY, b.n);
    prof_begin(st);
    launch_after(k_pyrdown<NB>, grid, 256, 0, st, b);
    count_launch();
    if (prof_enabled()) {
        double by = 0;
        for (int i = 0; i < b.n; ++i) by += (double)b.d[i].sw * b.d[i].sh + (double)b.d[i].dw * b.d[i].dh;
        prof_end(PK_PYRDOWN, by, st);
    }
    return launched(st, "k_pyrdown");
}
template cudaError_t launch_pyrdown<1>(const PyrDownBatch<1>&, int, int, cudaStream_t);
template cudaError_t launch_pyrdown<2>(const PyrDownBatch<2>&, int, int, cudaStream_t);
template cudaError_t launch_pyrdown<kBatchPyr>(const PyrDownBatch<kBatchPyr>&, int, int, cudaStream_t);

cudaError_t launch_p2_table(int* lut, int P2, float alpha, float beta, float lower, float upper, cudaStream_t st)
{
    prof_begin(st);
    launch_after(k_p2_table, 1, 256, 0, st, lut, P2, alpha, beta, lower, upper);
    count_launch();
    prof_end(PK_P2TABLE, 1024.0, st);
    return launched(st, "k_p2_table");
}

template <int NJ>
cudaError_t launch_prepare(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st)
{
    dim3 gf((e.max_w + kFtX - 1) / kFtX, (e.max_h + kFtY - 1) / kFtY, 2 * jobs.n);
    prof_begin(st);
    launch_after(k_features<NJ>, gf, 256, 0, st, jobs);
    count_launch();
    if (prof_enabled()) {
        // read u8 and write features of both views, write the keys; refine
        // levels read the quarter-size parent and write the label base
        double by = 0;
        for (int i = 0; i < jobs.n; ++i) {
            const LevelDesc& d = jobs.d[i];
            const double px = (double)d.w * d.h;
            by += px * (2 * (1 + (d.cost == COST_CENSUS ? 4 : 16)) + 4 + (d.refine ? 2 + 6.0 / 4 : 0));
        }
        prof_end(PK_FEATURES, by, st);
    }
    return launched(st, "k_features");
}

template <int HW, int NJ>
cudaError_t launch_bt_strip(const Jobs<NJ>& jobs, cudaStream_t st)
{
    size_t smem = 0;
    int gx = 0, max_h = 0;
    long long tiles = 0;
    for (int i = 0; i < jobs.n; ++i) {
        const LevelDesc& d = jobs.d[i];
        const int nblk = (d.D + 63) / 64, db = ((d.D + nblk - 1) / nblk + 15) / 16 * 16;
        const int tx = kBsSeg * bs_segments(db), n = (d.w + tx - 1) / tx * nblk;
        gx = std::max(gx, n);
        max_h = std::max(max_h, d.h);
        tiles += n;
        smem = std::max(smem, bs_smem<HW>(db));
    }
    // strips of 8 k window rows: the k whose waves of blocks (3 per SM) take
    // the fewest turns of 8 rows
    int strip = 0;
    long long best = 0;
    for (int k = 2; k <= 16; ++k) {
        const int rows = k * kBsRows - 2 * HW;
        const long long blocks = tiles * ((max_h + rows - 1) / rows), slots = 3LL * sm_count();
        const long long turns = (blocks + slots - 1) / slots * k;
        if (strip == 0 || turns < best) {
            strip = rows;
            best = turns;
        }
    }
    const cudaError_t err = allow_smem(k_cost_bt_strip<HW, NJ>);
    if (err != cudaSuccess) return err;
    launch_after(k_cost_bt_strip<HW, NJ>, dim3(gx, (max_h + strip - 1) / strip, jobs.n), kBsThreads, smem, st, jobs, strip);
    return cudaGetLastError();
}

// BT cost of fixed disparities: by window size, 3 to 7 pixels in strips, any
// other through k_cost_bt_box.  The C entry points take any block size: a
// negative one has empty windows, whose sums are 0.
template <int NJ>
cudaError_t launch_bt_fixed(const Jobs<NJ>& jobs, cudaStream_t st)
{
    Jobs<NJ> part;
    int launches = 0;
    for (int half = 0; half <= 3; ++half) {
        part.n = 0;
        int maxHalf = 0, max_w = 0, max_h = 0, max_D = 0;
        for (int i = 0; i < jobs.n; ++i) {
            const LevelDesc& d = jobs.d[i];
            const int h = d.bs / 2;
            if ((h >= 1 && h <= 3 ? h : 0) != half) continue;
            if (h < 0) {
                const cudaError_t err = cudaMemsetAsync(d.C, 0, (size_t)d.w * d.h * d.D * sizeof(int16_t), st);
                if (err != cudaSuccess) return err;
                continue;
            }
            part.d[part.n++] = d;
            maxHalf = std::max(maxHalf, h);
            max_w = std::max(max_w, d.w);
            max_h = std::max(max_h, d.h);
            max_D = std::max(max_D, d.D);
        }
        if (part.n == 0) continue;
        if (launches++ > 0) count_launch();   // launch_cost counts one
        cudaError_t err = cudaSuccess;
        if (half == 1) err = launch_bt_strip<1, NJ>(part, st);
        else if (half == 2) err = launch_bt_strip<2, NJ>(part, st);
        else if (half == 3) err = launch_bt_strip<3, NJ>(part, st);
        else {
            const size_t SW = kBxX + 2 * (size_t)maxHalf, SH = kBxY + 2 * (size_t)maxHalf;
            const size_t smem = SH * SW * kBxD + SH * kBxX * kBxD * 2;
            if (smem > kSmemPerBlock) return cudaErrorInvalidValue;
            if (smem > 48 * 1024) err = allow_smem(k_cost_bt_box<NJ>);
            if (err != cudaSuccess) return err;
            const int nxt = (max_w + kBxX - 1) / kBxX;
            dim3 g(nxt * ((max_D + kBxD - 1) / kBxD), (max_h + kBxY - 1) / kBxY, part.n);
            launch_after(k_cost_bt_box<NJ>, g, 256, smem, st, part, maxHalf, nxt);
            err = cudaGetLastError();
        }
        if (err != cudaSuccess) return err;
    }
    return cudaSuccess;
}

// All jobs in `jobs` share the cost mode and the refine flag.
template <int NJ>
cudaError_t launch_cost(const Jobs<NJ>& jobs, const LevelExtent& e, cudaStream_t st)
{
    const LevelDesc& J0 = jobs.d[0];
    prof_begin(st);
    if (J0.cost == COST_CENSUS) {
        int chunks = 0;   // of eight labels, in the widest row
        for (int i = 0; i < jobs.n; ++i) chunks = std::max(chunks, jobs.d[i].w * (jobs.d[i].D / 8));
        dim3 g((chunks + 255) / 256, (e.max_h + kCnRows - 1) / kCnRows, jobs.n);
        launch_after(k_cost_census<NJ>, g, 256, 0, st, jobs);
    } else if (J0.refine) {
        cudaError_t err = cudaFuncSetAttribute(k_cost_bt_tiled<NJ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)kTiSmem);
        if (err != cudaSuccess) return err;
        dim3 g((e.max_w + kTiX - 1) / kTiX, (e.max_h + kTiY - 1) / kTiY, jobs.n);
        launch_after(k_cost_bt_tiled<NJ>, g, 256, kTiSmem, st, jobs);
    } else {
        const cudaError_t err = launch_bt_fixed(jobs, st);
        if (err != cudaSuccess) return err;
    }
    count_launch();
    // write the int16 volume, read both views' features (and the label base)
    prof_end(PK_COST, jobs_vox(jobs) * 2 + jobs_px(jobs) * ((J0.cost == COST_CENSUS ? 8 : 32) + (J0.refine ? 2 : 0)), st);
    return launched(st, J0.cost == COST_CENSUS ? "k_cost_census" : J0.refine ? "k_cost_bt_tiled" : "BT cost of fixed disparities");
}

#define PG_INST(NJ)                                                                          \
    template cudaError_t launch_prepare<NJ>(const Jobs<NJ>&, const LevelExtent&, cudaStream_t); \
    template cudaError_t launch_cost<NJ>(const Jobs<NJ>&, const LevelExtent&, cudaStream_t);
PG_INST(1)
PG_INST(kBatchJobs)
#undef PG_INST

}  // namespace pg
