// Element tiles of the row gathers: the elements that touch a block of consecutive rows, each
// once, and for every row and CSR entry of the block the places of its contributions among them.
//
// A row gather that recomputes its elements meets every element three times (once per vertex);
// at 402k vertices the pressure rows spent 358 us that way, latency- and division-bound, against
// 32 us for their bytes. With a tile the block computes each of its elements once into shared
// memory (about 1.35 times every element at 96 rows, the halo included) and rows and entries then
// sum from there, in ascending element order as the gathers do, so the sums keep their order.
//
// The plan is connectivity only (made with the mesh handle); coordinates and fields are read at
// every call.
#pragma once

#include "internal.cuh"

namespace cfa {

constexpr int kEtThreads = 256;
constexpr int kEtRows = 96;                    // rows of a tile
constexpr int kEtMaxInc = 12 * kEtThreads;     // incidences of a tile that the plan can sort
constexpr int kEtLongRow = 24;                  // incidences of a row that one thread of the plan takes
constexpr int kEtMaxSmem = 200 * 1024;         // bytes of shared memory a tile may need
constexpr int kEtMaxRec = 19;                  // doubles per element of the largest records

struct ElemTiles {
    bool ok = false;          // false: some tile is too large, the row gathers run instead
    int rows = 0;             // rows per tile
    int ntiles = 0;
    int max_elems = 0;        // largest tile's element count, rounded up to a multiple of 4
    DevBuf<int> elems;        // [3 ne]: tile t's elements ascending, from inc_ptr[first row]
    DevBuf<int> count;        // [ntiles]
    DevBuf<unsigned short> rcode;   // [3 ne]: incidence s -> local element << 2 | local vertex
    DevBuf<unsigned short> ecode;   // [9 ne]: entries' contributions, local element << 4 | a << 2 | b
    DevBuf<unsigned short> eoff;    // [nnz]: an entry's first contribution, from its tile's first
};

struct ElemTileView {
    int rows, ntiles, stride;       // stride: elements per record array in shared memory
    const int *elems, *count, *inc_ptr;
    const unsigned short *rcode, *ecode, *eoff;
};

// Rows per tile: 96 rows of a triangulation touch about 250 elements, one per thread of the block.
// At 402k vertices, momentum / pressure rows in us: 32 rows 222 / 212, 64 rows 144 / 154, 96 rows
// 130 / 148, 128 rows 120 / 170, 192 rows 102 / 206, 256 rows 134 / 202: a taller tile repeats fewer
// elements, but its records leave fewer blocks per SM, which the pressure's 19 doubles an element
// feel first. Meshes with fewer than two such tiles per SM take 64 rows (22.5k vertices: 13.3 / 10.8
// against 13.3 / 13.3 us).
inline int elem_tile_rows(int n, int num_sms) { return n < 2 * num_sms * kEtRows ? 64 : kEtRows; }

// One tile of this block: rows [r0, r1), incidences [i0, i1), ne elements.
struct EtBlock {
    int r0, r1, i0, i1, ne;
};
__device__ __forceinline__ EtBlock et_block(const ElemTileView& v, int n) {
    EtBlock b;
    b.r0 = blockIdx.x * v.rows;
    b.r1 = min(n, b.r0 + v.rows);
    b.i0 = v.inc_ptr[b.r0];
    b.i1 = v.inc_ptr[b.r1];
    b.ne = v.count[blockIdx.x];
    return b;
}
inline int et_smem_bytes(const ElemTiles& t, int nrec) { return nrec * t.max_elems * (int)sizeof(double); }

}  // namespace cfa
