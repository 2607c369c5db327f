// Planning of the ring tiles (ring.cuh).
#include <cub/cub.cuh>

#include <algorithm>

#include "ring.cuh"

namespace cfa {

namespace {

using Sort = cub::BlockRadixSort<int, kRingThreads, kRingCand / kRingThreads>;
using Scan = cub::BlockScan<int, kRingThreads>;

struct PlanSmem {
    union {
        typename Sort::TempStorage sort;
        typename Scan::TempStorage scan;
    } tmp;
    int cand[kRingCand];
    int ring[2][kRingHalo];
    int edge[kRingThreads];
    int count, over;
};

__device__ __forceinline__ int find_sorted(const int* a, int m, int v) {
    int lo = 0, hi = m;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (a[mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return lo < m && a[lo] == v ? lo : -1;
}

// Sorts the s.count candidates and keeps each once in out (at most cap); returns their number, -1
// when there are more. All threads call it.
__device__ int sort_unique(PlanSmem& s, int* out, int cap) {
    constexpr int K = kRingCand / kRingThreads;
    const int m = s.count;
    int key[K], first[K], rank[K], total = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int q = threadIdx.x * K + k;
        key[k] = q < m ? s.cand[q] : 0x7fffffff;
    }
    __syncthreads();
    Sort(s.tmp.sort).Sort(key);
    s.edge[threadIdx.x] = key[K - 1];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int prev = k > 0 ? key[k - 1] : threadIdx.x > 0 ? s.edge[threadIdx.x - 1] : -1;
        first[k] = key[k] != prev && key[k] != 0x7fffffff ? 1 : 0;
    }
    Scan(s.tmp.scan).ExclusiveSum(first, rank, total);
    if (total <= cap)
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (first[k]) out[rank[k]] = key[k];
    __syncthreads();
    return total <= cap ? total : -1;
}

__device__ __forceinline__ void add_candidate(PlanSmem& s, int j) {
    const int q = atomicAdd(&s.count, 1);
    if (q < kRingCand) s.cand[q] = j;
    else s.over = 1;
}

// Rings and sizes of one tile per block. flags: 0 a tile does not fit, 1 rows, 2 local vertices,
// 3 entries (largest).
__global__ void __launch_bounds__(kRingThreads)
k_ring_plan(int n, int rows, const int* __restrict__ rp, const int* __restrict__ ci, RingMeta* __restrict__ meta,
            int* __restrict__ halo, int* __restrict__ cnt, int* __restrict__ flags) {
    __shared__ PlanSmem s;
    CFA_GRID_DEP();
    const int r0 = blockIdx.x * rows, r1 = min(n, r0 + rows), nr = r1 - r0;
    const int p0 = rp[r0], p1 = rp[r1];
    int h1 = -1, h2 = -1;
    if (threadIdx.x == 0) s.count = s.over = 0;
    __syncthreads();
    for (int p = p0 + threadIdx.x; p < p1; p += kRingThreads) {
        const int j = ci[p];
        if (j < r0 || j >= r1) add_candidate(s, j);
    }
    __syncthreads();
    if (!s.over) h1 = sort_unique(s, s.ring[0], kRingHalo);
    __syncthreads();
    if (h1 >= 0) {
        if (threadIdx.x == 0) s.count = 0;
        __syncthreads();
        // eight lanes per ring 1 row
        for (int k = threadIdx.x / 8; k < h1; k += kRingThreads / 8)
            for (int p = rp[s.ring[0][k]] + (threadIdx.x & 7); p < rp[s.ring[0][k] + 1]; p += 8) {
                const int j = ci[p];
                if ((j < r0 || j >= r1) && find_sorted(s.ring[0], h1, j) < 0) add_candidate(s, j);
            }
        __syncthreads();
        if (!s.over) h2 = sort_unique(s, s.ring[1], kRingHalo - h1);
    }
    __syncthreads();
    const bool fits = h1 >= 0 && h2 >= 0 && nr + h1 <= kRingMaxRows;
    int len = 0;
    if (fits) {
        for (int k = threadIdx.x; k < h1; k += kRingThreads) len += rp[s.ring[0][k] + 1] - rp[s.ring[0][k]];
        for (int k = threadIdx.x; k < h1 + h2; k += kRingThreads)
            halo[(size_t)blockIdx.x * kRingHalo + k] = k < h1 ? s.ring[0][k] : s.ring[1][k - h1];
    }
    int before = 0, total = 0;
    Scan(s.tmp.scan).ExclusiveSum(len, before, total);
    if (threadIdx.x == 0) {
        const int ne = fits ? p1 - p0 + total : 0;
        meta[blockIdx.x] = {fits ? h1 : 0, fits ? h2 : 0, ne, 0, 0};
        cnt[blockIdx.x] = (ne + 7) & ~7;
        if (!fits || ne > 0xffff) flags[0] = 1;
        else {
            atomicMax(&flags[1], nr + h1);
            atomicMax(&flags[2], nr + h1 + h2);
            atomicMax(&flags[3], ne);
        }
    }
}

// Row offsets, local columns and values of one tile per block.
__global__ void __launch_bounds__(kRingThreads)
k_ring_fill(int n, int rows, const int* __restrict__ rp, const int* __restrict__ ci, const double* __restrict__ v,
            RingMeta* __restrict__ meta, const int* __restrict__ off, const int* __restrict__ halo, int rp_stride,
            unsigned short* __restrict__ trp, unsigned short* __restrict__ tci, float* __restrict__ v32,
            double* __restrict__ v64) {
    constexpr int K = kRingMaxRows / kRingThreads;
    __shared__ typename Scan::TempStorage tmp;
    __shared__ int ring[kRingHalo];
    __shared__ int start[kRingMaxRows + 1];
    CFA_GRID_DEP();
    const int r0 = blockIdx.x * rows, r1 = min(n, r0 + rows), nr = r1 - r0;
    const RingMeta m = meta[blockIdx.x];
    const int R = nr + m.h1;
    const long long e0 = off[blockIdx.x];
    for (int k = threadIdx.x; k < m.h1 + m.h2; k += kRingThreads) ring[k] = halo[(size_t)blockIdx.x * kRingHalo + k];
    __syncthreads();
    int len[K], at[K], total = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int lr = threadIdx.x * K + k;
        const int row = lr < nr ? r0 + lr : lr < R ? ring[lr - nr] : -1;
        len[k] = row >= 0 ? rp[row + 1] - rp[row] : 0;
    }
    Scan(tmp).ExclusiveSum(len, at, total);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int lr = threadIdx.x * K + k;
        if (lr <= R) {
            start[lr] = at[k];
            trp[(size_t)blockIdx.x * rp_stride + lr] = (unsigned short)at[k];
        }
    }
    if (R == kRingMaxRows && threadIdx.x == 0) {   // the last offset falls beyond the scan's items
        start[R] = total;
        trp[(size_t)blockIdx.x * rp_stride + R] = (unsigned short)total;
    }
    __syncthreads();
    // four lanes per row
    for (int lr = threadIdx.x / 4; lr < R; lr += kRingThreads / 4) {
        const int row = lr < nr ? r0 + lr : ring[lr - nr];
        const int q0 = rp[row], q1 = rp[row + 1];
        for (int q = q0 + (threadIdx.x & 3); q < q1; q += 4) {
            const int j = ci[q];
            int c;
            if (j >= r0 && j < r1) c = j - r0;
            else {
                c = find_sorted(ring, m.h1, j);
                c = c >= 0 ? nr + c : nr + m.h1 + find_sorted(ring + m.h1, m.h2, j);
            }
            const long long e = e0 + start[lr] + (q - q0);
            tci[e] = (unsigned short)c;
            if (v32) v32[e] = (float)v[q];
            if (v64) v64[e] = v[q];
        }
    }
    if (threadIdx.x == 0) meta[blockIdx.x].e0 = e0;
}

}  // namespace

// Rows per tile, 0 where one sweep per pass is the better form. A pair of sweeps saves a kernel
// boundary, but its gathers go through shared memory, some 21 wavefronts for a warp's 32 entries (columns,
// values and vector), no fewer than the one-sweep kernels' through L1, and its ring repeats work, so it pays while a sweep is mostly
// launch and latency. CG iteration with one against two sweeps per pass, best rows, FP64 / mixed:
// 8k vertices 38.8 -> 33.2 / 36.4 -> 30.7 us, 37k 54.2 -> 51.3 / 51.6 -> 49.4 us, 69k 62.1 -> 59.8 /
// 58.9 -> 56.8 us; 141k 89.1 -> 91.4 / 85.7 -> 85.6 us, 651k 236 -> 258 / 210 -> 218 us. The line lies
// at two tiles of 256 rows per SM; below it the tiles shrink while there is less than one per SM
// (8k: 64 rows 33.2, 256 rows 36.4 us; 37k: 128 rows 51.3, 64 rows 55.6 us).
static int ring_rows(int n, int num_sms) {
    int r = 256;
    if ((long long)n > 2LL * r * num_sms) return 0;
    while (r > 64 && (long long)n < (long long)num_sms * r) r /= 2;
    return r;
}

cfa_status build_ring(cfa_ctx* ctx, int n, int nnz, const int* rp, const int* ci, const double* v, bool f32, bool f64,
                      RingTiles& R) {
    R.ok = false;
    R.n = n;
    R.rows = ring_rows(n, ctx->num_sms);
    if (R.rows == 0) return CFA_OK;
    R.ntiles = ceil_div(n, R.rows);
    CFA_CUDA(R.meta.ensure(R.ntiles));
    CFA_CUDA(R.halo.ensure((size_t)R.ntiles * kRingHalo));
    CFA_CUDA(R.cnt.ensure(R.ntiles + 1));
    CFA_CUDA(R.off.ensure(R.ntiles + 1));
    CFA_CUDA(R.flags.ensure(4));
    CFA_CUDA(cudaMemsetAsync(R.flags.p, 0, 4 * sizeof(int), ctx->stream));
    CFA_CUDA(cudaMemsetAsync(R.cnt.p + R.ntiles, 0, sizeof(int), ctx->stream));
    CFA_LAUNCH(ctx, k_ring_plan, R.ntiles, kRingThreads, 0, n, R.rows, rp, ci, R.meta.p, R.halo.p, R.cnt.p, R.flags.p);
    size_t tmp = 0;
    CFA_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp, R.cnt.p, R.off.p, R.ntiles + 1, ctx->stream));
    CFA_CUDA(R.tmp.ensure(tmp + 16));
    CFA_CUDA(cub::DeviceScan::ExclusiveSum(R.tmp.p, tmp, R.cnt.p, R.off.p, R.ntiles + 1, ctx->stream));
    int h[5] = {0, 0, 0, 0, 0};
    CFA_CUDA(cudaMemcpyAsync(h, R.flags.p, 4 * sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    CFA_CUDA(cudaMemcpyAsync(h + 4, R.off.p + R.ntiles, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    CFA_CUDA(cudaStreamSynchronize(ctx->stream));
    if (h[0]) return CFA_OK;
    R.max_rows = h[1];
    R.max_local = h[2];
    R.max_ne = h[3];
    R.total = h[4];
    if (ring_smem(R, f64 ? 8 : 4, 8) > kRingMaxSmem) return CFA_OK;
    R.rp_stride = (R.max_rows + 1 + 7) & ~7;
    CFA_CUDA(R.rp.ensure((size_t)R.ntiles * R.rp_stride));
    CFA_CUDA(R.ci.ensure(R.total + 8));
    if (f32) CFA_CUDA(R.v32.ensure(R.total + 8));
    if (f64) CFA_CUDA(R.v64.ensure(R.total + 8));
    CFA_CUDA(R.b.ensure(n));
    CFA_LAUNCH(ctx, k_ring_fill, R.ntiles, kRingThreads, 0, n, R.rows, rp, ci, v, R.meta.p, (const int*)R.off.p,
               (const int*)R.halo.p, R.rp_stride, R.rp.p, R.ci.p, f32 ? R.v32.p : (float*)nullptr,
               f64 ? R.v64.p : (double*)nullptr);
    tile_fence(ctx);
    CFA_CHECK_LAUNCH();
    R.ok = true;
    return CFA_OK;
}

}  // namespace cfa
