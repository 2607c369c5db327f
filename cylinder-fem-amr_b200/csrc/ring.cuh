// Ring tiles: two consecutive sweeps over one sparse matrix in one pass.
//
// A tile is a block of consecutive rows together with the rows its rows couple to (ring 1) and the
// columns those couple to (ring 2). A block of threads brings the tile's vector into shared memory,
// computes the first sweep on its own rows and on ring 1, and the second sweep on its own rows
// from there: the matrix is read once for both sweeps (plus the ring's share), the vector of the
// second sweep never leaves the SM, and a kernel boundary goes. Columns are 16-bit places in the
// tile's vector. Every row sums its entries in CSR order, as the one-sweep kernels do.
#pragma once

#include "internal.cuh"
#include "tiled.cuh"

namespace cfa {

constexpr int kRingThreads = 256;
constexpr int kRingHalo = 1024;           // ring 1 and ring 2 vertices a tile may have
constexpr int kRingCand = 8 * kRingThreads;   // candidates a ring's sort takes
constexpr int kRingMaxRows = 6 * kRingThreads;   // own and ring 1 rows of a tile
constexpr int kRingMaxSmem = 100 * 1024;  // dynamic shared memory a block may take (two per SM)

struct RingMeta {
    int h1, h2, ne, pad;      // ring sizes, entries of the own and ring 1 rows
    long long e0;             // the tile's first entry (multiple of 8)
};

struct RingTiles {
    bool ok = false;
    int n = 0, rows = 0, ntiles = 0;
    int max_rows = 0, max_local = 0, max_ne = 0;   // largest tile
    long long total = 0;      // entries stored, paddings included
    DevBuf<RingMeta> meta;
    DevBuf<int> halo;                 // [ntiles][kRingHalo]: ring 1, then ring 2, each ascending
    DevBuf<unsigned short> rp;        // [ntiles][rp_stride]
    int rp_stride = 0;
    DevBuf<unsigned short> ci;        // [total]
    DevBuf<float> v32;
    DevBuf<double> v64;
    DevBuf<double> b;                 // [n]: the right-hand side of an apply in place
    DevBuf<int> cnt;                  // planning: padded entries per tile, then their offsets
    DevBuf<int> off, flags;
    DevBuf<unsigned char> tmp;
};

template <class V>
struct RingView {
    int n, rows, ntiles, rp_stride, max_rows, max_local, max_ne;
    const RingMeta* meta;
    const int* halo;
    const unsigned short *rp, *ci;
    const V* v;
    int* err;
};

inline const float* ring_values(const RingTiles& R, float) { return R.v32.p; }
inline const double* ring_values(const RingTiles& R, double) { return R.v64.p; }

// Dynamic shared memory of a two-sweep kernel with values of vb and vectors of tb bytes: the bulk
// copied row offsets, columns and values, then x (own, ring 1, ring 2), the first sweep's result,
// b and omega D^-1 (own, ring 1), and the ring's vertices.
struct RingSmem {
    int rp, ci, v, x, y, b, od, hl, bytes;
};
__host__ __device__ inline RingSmem ring_smem_layout(int max_rows, int max_local, int max_ne, int vb, int tb) {
    RingSmem s;
    int o = 0;
    auto take = [&](long long bytes) { const int at = o; o += (int)align16(bytes); return at; };
    const int ne = (max_ne + 7) & ~7;
    s.rp = take(2LL * (max_rows + 8));
    s.ci = take(2LL * ne);
    s.v = take((long long)vb * ne);
    s.x = take((long long)tb * max_local);
    s.y = take((long long)tb * max_rows);
    s.b = take((long long)tb * max_rows);
    s.od = take((long long)tb * max_rows);
    s.hl = take(4LL * max_local);
    s.bytes = o;
    return s;
}
inline int ring_smem(const RingTiles& R, int vb, int tb) {
    return ring_smem_layout(R.max_rows, R.max_local, R.max_ne, vb, tb).bytes;
}

// Plans and fills the ring tiles of a device CSR matrix with FP32 and / or FP64 values. ok stays
// false where the two-sweep pass does not apply (see ring.cu); synchronises.
cfa_status build_ring(cfa_ctx* ctx, int n, int nnz, const int* rp, const int* ci, const double* v, bool f32, bool f64,
                      RingTiles& R);

}  // namespace cfa
