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
// every call. It takes 43 bytes an element (65 as the buffers are sized), beside 50 (75) of the handle's
// incidences and positions; a mesh whose kernels all take the row gathers gives it back.
#pragma once

#include "internal.cuh"

namespace cfa {

constexpr int kEtThreads = 256;
constexpr int kEtRows = 96;                    // rows of a tile
constexpr int kEtMaxInc = 12 * kEtThreads;     // incidences of a tile that the plan can sort
constexpr int kEtLongRow = 24;                  // incidences of a row that one thread of the plan takes
constexpr int kEtMaxSmem = 200 * 1024;         // bytes of shared memory a tile may need
constexpr int kEtMaxRec = 19;                  // doubles per element of the largest records
// Elements of all tiles over elements of the mesh (ElemTiles::repeats): 1.42 in the mesh's own order, 1.9
// in reverse Cuthill-McKee's, 2.1 to 2.8 sorted by x, 3 (nothing shared) in a random one. Tiles against
// gathers in us: sorted by x, 402k vertices: momentum 239 / 169, pressure 303 / 396, projection 105 / 89;
// Cuthill-McKee: 153 / 153, 185 / 370, 67 / 75; random, 37k: 48 / 36, 60 / 51, 42 / 28, and pressure at
// 4.2M 13.96 / 9.89 ms. Small meshes (64-row tiles) gain in any order: random, 22k: 29 / 36, 41 / 51, 24 / 28.
constexpr double kEtRepeats = 2.0;             // most that the momentum and gradient kernels take
constexpr double kEtRepeatsPressure = 2.9;     // ... the pressure's, and with it any

struct ElemTiles {
    bool ok = false;          // false: the row gathers run instead (a tile too large, elements hardly shared)
    int rows = 0;             // rows per tile
    int ntiles = 0;
    int max_elems = 0;        // largest tile's element count, rounded up to a multiple of 4
    int max_row = 0;          // most elements around one vertex
    double repeats = 0.0;     // elements of all tiles / elements of the mesh
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

// Whether a kernel's tiles are its better form on this mesh. Both forms take whole waves of blocks, and
// a wave of tiles costs a share of a wave of gathers that the kernel's comment states: tile_blocks and
// row_blocks are the blocks an SM holds of each, num / den the most waves of tiles per wave of gathers.
// A gather runs a long row in one thread (0.25 to 1.1 us an element), which tiles share. max_elems: the
// largest tile sizes every block's shared memory, so one scattered tile (vertices appended by a
// refinement and never renumbered) takes the L1 from all; the momentum's large records feel it.
struct EtForm {
    int tile_blocks, row_blocks, num, den;
    int max_elems = 1 << 30;
};
constexpr int kEtHubRow = 31;
inline bool et_better(const ElemTiles& t, int n, int num_sms, const EtForm& f) {
    if (!t.ok || (t.rows == kEtRows && t.repeats > kEtRepeats)) return false;
    if (t.max_row > kEtHubRow) return true;
    if (t.max_elems > f.max_elems) return false;
    const long long tiles = ceil_div(t.ntiles, f.tile_blocks * num_sms);
    const long long gathers = ceil_div(ceil_div(n, kThreads), f.row_blocks * num_sms);
    return tiles * f.den <= gathers * f.num;
}

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
