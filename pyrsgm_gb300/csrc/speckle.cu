// speckle.cu -- opt-in speckle filter on an int16 disparity map, after the
// SGM path (no counterpart in the reference library; its benchmark turns
// OpenCV's filterSpeckles off, bench/pyrsgm_bench.cpp:312-323).  Semantics
// of cv::filterSpeckles: 4-neighbours belong to one region when neither
// holds new_val and their values differ by at most max_diff; every region
// of at most max_speckle_size pixels is set to new_val.
//
// GPU form: connected components by lock-free union-find (roots linked
// larger index -> smaller with atomicCAS).  Inside a 32x32 tile a row's runs
// are found with one ballot, so that a pixel starts at its run's first one,
// and a link to the row above is needed only where the pixel to the left
// has not made it already (on a disparity map, at few pixels); the tile
// leaves every pixel pointing at its tile-local root, and that root's size.
// Then the same across tile borders in global memory (a sixteenth of the
// pixels), the sizes of the tile roots added to their global roots, and one
// pass that clears small regions.  The partition into regions is unique, so
// the output is exactly that of a sequential flood fill.
// Bound by the dependent walks of the four launches, not by the 20 bytes a
// pixel they move (a 1080p map: 146 us a call with a label a pixel in 32x8
// tiles and every pixel in the border pass, 64 now).
#include <cuda_runtime.h>

#include <cstdint>

#include "pyrsgm/pyrsgm_gb300.h"
#include "sgm_launch.h"

namespace pg {
namespace {

// Root of x; path halving (each visited node is pointed at its grandparent,
// an ancestor, so concurrent halving keeps every pointer valid).  Parents
// only ever point to smaller indices, so the walk ends within x steps.
__device__ __forceinline__ int sp_find(int* lab, int x)
{
    for (;;) {
        const int p = *(volatile int*)&lab[x];
        if (p == x) return x;
        const int gp = *(volatile int*)&lab[p];
        if (gp != p) lab[x] = gp;
        x = p;
    }
}

// Link the sets of a and b.  Every failed CAS means another thread linked a
// root meanwhile (the number of roots only falls), so the loop is lock-free;
// the bound is a guard, not a wait.
__device__ __forceinline__ void sp_union(int* lab, int a, int b, int n)
{
    for (int it = 0; it <= n; ++it) {
        a = sp_find(lab, a);
        b = sp_find(lab, b);
        if (a == b) return;
        if (a < b) {
            const int t = a;
            a = b;
            b = t;
        }
        if (atomicCAS(&lab[a], a, b) == a) return;
    }
}

struct SpArgs {
    short* d;
    size_t pitch;   // elements
    int w, h;
    int new_val, max_size, max_diff;
    int* lab;
    int* size;
};

__device__ __forceinline__ int sp_at(const SpArgs& A, int x, int y) { return A.d[(size_t)y * A.pitch + x]; }
__device__ __forceinline__ bool sp_joined(const SpArgs& A, int u, int v)
{
    return u != A.new_val && v != A.new_val && abs(u - v) <= A.max_diff;
}

constexpr int kSpTile = 32, kSpRows = 4;   // tile side; rows of it per warp

// First pixel of a lane's run: the highest clear bit at or below the lane.
__device__ __forceinline__ int sp_first(unsigned runs, int lane)
{
    return 31 - __clz(~runs & (0xffffffffu >> (31 - lane)));
}

// Tile pass (see above): lab[p] = index of p's tile-local root, size[p] = its
// pixels in the tile at the root, 0 elsewhere.
__global__ void __launch_bounds__(256) k_sp_tile(const SpArgs A)
{
    let_next_in();
    after_previous();
    __shared__ int lab[kSpTile * kSpTile], cnt[kSpTile * kSpTile];
    __shared__ short val[kSpTile * kSpTile];
    __shared__ unsigned runs[kSpTile];   // bit x: pixel x continues the run of pixel x - 1
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x = blockIdx.x * kSpTile + lane, y0 = blockIdx.y * kSpTile + warp * kSpRows;
#pragma unroll
    for (int k = 0; k < kSpRows; ++k) {
        const int row = warp * kSpRows + k, i = row * kSpTile + lane, y = y0 + k;
        const int v = x < A.w && y < A.h ? sp_at(A, x, y) : A.new_val;
        const int left = __shfl_up_sync(0xffffffffu, v, 1);
        const bool on = lane > 0 && sp_joined(A, left, v);
        const unsigned m = __ballot_sync(0xffffffffu, on);
        if (lane == 0) runs[row] = m;
        val[i] = (short)v;
        if (!on) lab[i] = i;   // only the first pixels of runs have a label here
        cnt[i] = 0;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSpRows; ++k) {
        const int row = warp * kSpRows + k, i = row * kSpTile + lane;
        const bool up = row > 0 && sp_joined(A, row > 0 ? val[i - kSpTile] : A.new_val, val[i]);
        const unsigned ups = __ballot_sync(0xffffffffu, up);
        // left neighbour joined to this pixel and to its own upper one, that one to ours
        const unsigned made = runs[row] & (row > 0 ? runs[row - 1] : 0u) & (ups << 1);
        if (up && !((made >> lane) & 1u))
            sp_union(lab, row * kSpTile + sp_first(runs[row], lane), (row - 1) * kSpTile + sp_first(runs[row - 1], lane),
                     kSpTile * kSpTile);
    }
    __syncthreads();
    int root[kSpRows];
#pragma unroll
    for (int k = 0; k < kSpRows; ++k) {
        const int row = warp * kSpRows + k, i = row * kSpTile + lane;
        const unsigned m = runs[row];
        int r = -1;
        if (!((m >> lane) & 1u) && val[i] != A.new_val) {   // a run's first pixel finds its root and counts it
            r = sp_find(lab, i);
            const unsigned ends = ~m >> lane >> 1;           // clear bits after the lane: the next run
            atomicAdd(&cnt[r], ends ? __ffs(ends) : 32 - lane);
        }
        root[k] = __shfl_sync(0xffffffffu, r, sp_first(m, lane));
    }
    __syncthreads();
    if (x >= A.w) return;
#pragma unroll
    for (int k = 0; k < kSpRows; ++k) {
        const int i = (warp * kSpRows + k) * kSpTile + lane, y = y0 + k;
        if (y >= A.h) break;
        const int p = y * A.w + x, r = root[k];
        A.size[p] = r == i ? cnt[i] : 0;
        A.lab[p] = r < 0 ? -1 : ((int)blockIdx.y * kSpTile + r / kSpTile) * A.w + (int)blockIdx.x * kSpTile + r % kSpTile;
    }
}

// Border pass: links across the left edges of the tiles (thread i < nv: edge
// i / h, row i % h), then across their upper ones.
__global__ void __launch_bounds__(256) k_sp_link(const SpArgs A, int nv, int nh)
{
    let_next_in();
    after_previous();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= nv + nh) return;
    const bool side = i < nv;
    const int e = side ? i : i - nv, len = side ? A.h : A.w;
    const int x = side ? (e / len + 1) * kSpTile : e % len, y = side ? e % len : (e / len + 1) * kSpTile;
    const int dx = side ? 1 : 0, dy = side ? 0 : 1;     // towards the other tile: (x - dx, y - dy)
    const int v = sp_at(A, x, y), u = sp_at(A, x - dx, y - dy);
    if (!sp_joined(A, u, v)) return;
    // the pair before along the edge, in the same two tiles, has made it?
    if ((side ? y : x) % kSpTile != 0) {
        const int v1 = sp_at(A, x - dy, y - dx), u1 = sp_at(A, x - dx - dy, y - dy - dx);
        if (sp_joined(A, u1, v1) && sp_joined(A, v1, v) && sp_joined(A, u1, u)) return;
    }
    sp_union(A.lab, y * A.w + x, (y - dy) * A.w + x - dx, A.w * A.h);
}

// The tile roots' sizes to their global roots.
__global__ void __launch_bounds__(256) k_sp_count(const SpArgs A)
{
    let_next_in();
    after_previous();
    const long long p = (long long)blockIdx.x * 256 + threadIdx.x;
    if (p >= (long long)A.w * A.h) return;
    const int n = A.size[p];
    if (n == 0 || A.lab[p] == (int)p) return;   // (a global root's own pixels are counted)
    atomicAdd(&A.size[sp_find(A.lab, (int)p)], n);
}

__global__ void __launch_bounds__(256) k_sp_apply(const SpArgs A)
{
    let_next_in();
    after_previous();
    const int x = blockIdx.x * 32 + (threadIdx.x & 31), y = blockIdx.y * 8 + (threadIdx.x >> 5);
    if (x >= A.w || y >= A.h) return;
    int r = A.lab[y * A.w + x];
    if (r < 0) return;
    for (int q = A.lab[r]; q != r; q = A.lab[r]) r = q;
    if (A.size[r] <= A.max_size) A.d[(size_t)y * A.pitch + x] = (short)A.new_val;
}

}  // namespace
}  // namespace pg

extern "C" int pyrsgm_gb300_filter_speckles(short* d_disp, size_t pitch_bytes, int width, int height, short new_val,
                                            int max_speckle_size, int max_diff, cudaStream_t stream)
{
    if (!d_disp || width <= 0 || height <= 0 || pitch_bytes % sizeof(short) != 0 ||
        pitch_bytes < (size_t)width * sizeof(short) || max_diff < 0 || (long long)width * height > 0x7fffffffLL)
        return -1;
    if (max_speckle_size <= 0) return 0;
    const size_t n = (size_t)width * height;
    void* scratch = nullptr;
    if (cudaMallocAsync(&scratch, n * 8, stream) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    pg::SpArgs A{d_disp, pitch_bytes / sizeof(short), width, height, new_val, max_speckle_size, max_diff,
                 static_cast<int*>(scratch), static_cast<int*>(scratch) + n};
    const int tx = (width + pg::kSpTile - 1) / pg::kSpTile, ty = (height + pg::kSpTile - 1) / pg::kSpTile;
    const int nv = (tx - 1) * height, nh = (ty - 1) * width;   // border pixels: left edges, upper edges
    cudaError_t e;
    int launches = 3;
    pg::launch_after(pg::k_sp_tile, dim3(tx, ty), 256, 0, stream, A);
    e = pg::launched(stream, "k_sp_tile");
    if (e == cudaSuccess && nv + nh > 0) {
        pg::launch_after(pg::k_sp_link, (nv + nh + 255) / 256, 256, 0, stream, A, nv, nh);
        e = pg::launched(stream, "k_sp_link");
        ++launches;
        if (e == cudaSuccess) {
            pg::launch_after(pg::k_sp_count, (int)((n + 255) / 256), 256, 0, stream, A);
            e = pg::launched(stream, "k_sp_count");
        }
    } else {
        --launches;   // one tile: its sizes are final
    }
    if (e == cudaSuccess) {
        pg::launch_after(pg::k_sp_apply, dim3((width + 31) / 32, (height + 7) / 8), 256, 0, stream, A);
        e = pg::launched(stream, "k_sp_apply");
    }
    pg::count_launches(launches);
    cudaFreeAsync(scratch, stream);
    return e == cudaSuccess ? 0 : -1;
}
