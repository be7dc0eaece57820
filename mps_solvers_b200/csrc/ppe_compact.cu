// ppe_compact.cu -- the PPE matrix in a compact 16-bit layout and the
// persistent PCG solve over it.
//
// Same system as ppe.cu (MPS_CPU::buildPoisson, MPS_CAL_v4.0/MPS_CPU.cpp:619-710,
// solved as MPS_CPU::DoCG's CG, :829-888, with diagonal scaling and FP64
// defect correction).  The layout is built around tiles:
//
//  * the R non-Dirichlet rows are numbered 0..R-1 along a Hilbert curve over
//    the reference's linked cells (edge max(r0, rlap); the fast arithmetic's
//    halved cells are grouped back into them), so a run of consecutive rows
//    is a compact lump of the fluid;
//  * a tile is such a run, one per block of the solver up to C16_TILE_ROWS
//    rows on average, cut where the tiles carry equal shares of the matrix.
//    Its rows couple to few distinct columns (the lump and a shell of one
//    kernel radius around it: 2,900 columns for 920 rows of the 310,912-
//    particle dam break, 6,100 for 1,840 rows of a 1.6 M-particle scene; the
//    same runs in cell order have 5,200 and 11,800), which the tile lists;
//  * an entry is the column's position in its tile's list, times 4, in 16
//    bits, beside its FP32 weight: 6 bytes.  Slices of 8 rows, a warp takes
//    one with 4 lanes per row; lane L = 8 q + r holds, in every chunk of 16
//    entries of row r, entries 4 q to 4 q + 3.  A chunk is 768 contiguous
//    bytes: 512 of weights, then 256 of codes;
//  * a column past the tile's list (C16_COLS columns) is coded 65535 and read
//    from the assembly's row-major columns; only rows with far more neighbours
//    than a lattice has get there.
//
// In every product a block first brings the tile's columns of the vector
// into shared memory, in coalesced runs, and then reads each entry's operand
// from there: the product streams the matrix, and its gathers never leave
// the SM.  Before, each entry gathered 8 bytes through L1 from a vector the
// whole grid reads, and the wait for those gathers set the pace.
#include <algorithm>
#include <cstring>
#include <vector>

#include <cuda_bf16.h>

#include "cellsort.cuh"
#include "ppe.cuh"
#include "ppe_device.cuh"

namespace mpsb {

namespace {

inline uint32_t cblocks(uint32_t n, uint32_t t) { return (n + t - 1) / t; }

constexpr uint32_t C16_ROWS = 8;            // rows per slice
constexpr uint32_t C16_CHUNK_BYTES = 768;   // a chunk, 128 entries (8 rows x 16): weights, then codes
constexpr uint32_t C16_ESC = 0xffffu;       // escaped code
// Rows of a tile on average, and a slice's cost beside its chunks (1 to 32 of
// them) when tiles are cut: a tile then has at most 37 / 5 of the average,
// 11,904 rows, which fit its column list, and the list as doubles and the
// row sums fit a block's shared memory.
constexpr uint32_t C16_TILE_ROWS = 1600;
constexpr uint32_t C16_SLICE_COST = 5;
// The limits past which an entry is escaped and a tile is done by one warp;
// builds of the tests lower them, so that small scenes get there.
#ifndef MPS_C16_COLS
#define MPS_C16_COLS 12288
#endif
#ifndef MPS_C16_PAGES
#define MPS_C16_PAGES 512
#endif
#ifndef MPS_C16_WHOLE
#define MPS_C16_WHOLE 0
#endif
constexpr uint32_t C16_COLS = MPS_C16_COLS;  // columns a tile lists (4 x 12,287 is below the escape code)
constexpr uint32_t C16_PAGE = 256;           // rows per page of the tile's column set
constexpr uint32_t C16_PAGES = MPS_C16_PAGES;  // pages a tile's column set holds
constexpr bool C16_WHOLE = MPS_C16_WHOLE != 0;  // every tile by one warp
constexpr uint32_t C16_NONE = 0xffffffffu;
constexpr int C16_THREADS = 512;            // a solver block
constexpr int C16_PACK_THREADS = 1024;
constexpr int C16_BATCH = 4;                // chunks a warp loads at a time, twice buffered
constexpr int C16_BATCH64 = 3;              // (6 of them: 5 % slower; 768 threads with 3: 2 to 10 % slower)
// A matrix of several L2s comes from memory: every warp has the batch after
// the next fetched into L2, 3 KB at a time, before it loads it.  Where L2 holds
// a good part of the matrix the fetches are in its way; with S', which L2
// holds too, up to a larger one.  ms a solve without and with them, by rows
// (1.45 KB of entries each): 303,860 4.46 and 4.56 (S' 4.54, 4.78), 374,952
// 5.49 and 5.57 (5.53, 5.85), 419,968 6.15 and 6.10 (6.20, 6.44), 468,160 7.03
// and 6.86 (7.05, 7.08), 531,196 8.12 and 7.88 (8.43, 8.17), 689,132 10.34 and
// 10.06 (10.89, 10.45): they cross at 4.5 and 5 times the L2.
// 8, 16 and 24 chunks ahead: 15.8, 15.9 and 16.1 ms at 1,088,346 rows with S',
// 4 15.5; none (the loaded batch itself) 15.8.
constexpr uint32_t C16_AHEAD = 4;
constexpr uint32_t C16_AHEAD_FROM = 9, C16_AHEAD_FROM_SP = 10;  // half L2s of entries
constexpr uint32_t C16_STATS = 4;
constexpr uint32_t C16_SP_SLICES = C16_COLS / 32 + 1;  // S' slices (32 rows) a tile can have, and one

// One tile: slices [s0, s1), its columns (its own rows first, then the others
// in ascending order), whether entries are escaped, its longest slice and,
// in a batch, its scene.
struct C16Tile {
    uint32_t s0, s1, ncol, esc, wmax, scene, pad[2];
};

// Tiles of R rows for G solver blocks: the same number for every block.  The
// scenes of a batch (ns, 0 for a single scene) have tiles of their own; one
// tile of each is spoken for before the rows are shared out.
__host__ __device__ __forceinline__ uint32_t c16_tiles(uint32_t R, uint32_t G, uint32_t ns) {
    const uint32_t t = (R + C16_TILE_ROWS - 1) / C16_TILE_ROWS + ns;
    const uint32_t k = (t + G - 1) / G;
    return G * (k > 0 ? k : 1u);
}

// ---------------------------------------------------------------- row order
// Whether particle i has a row (is not Dirichlet), as the assembly's test:
// n < beta n0 in double exactly when n < the least float >= beta n0.
struct C16Flag {
    const float4* pos;
    const float* n;
    const uint32_t* id;
    const uint32_t* sid_of_id;  // batch: the scene of each particle id
    const PpeScene* scenes;
    double bthr;
    bool fluid;                 // the viscosity's system: a row for every fluid particle
};

__device__ __forceinline__ bool c16_is_row(const C16Flag& F, uint32_t i) {
    if (F.fluid) return ptype(F.pos[i]) == T_FLUID;
    double b = F.bthr;
    if (F.scenes) {
        const PpeScene& s = F.scenes[F.sid_of_id[F.id[i]]];
        b = s.beta * s.n0;
    }
    return ptype(F.pos[i]) != T_DUMMY && !((double)F.n[i] < b);
}

// Grids of many linked cells, most of them empty (c16_lists): the ones that hold
// particles as a list, in any order (the counts of the others are 0).
__global__ void __launch_bounds__(256) k_c16_occupied(const uint32_t* __restrict__ cells, uint32_t nsuper,
                                                      const uint32_t* __restrict__ cs, uint32_t* __restrict__ base,
                                                      uint32_t* __restrict__ list, uint32_t* __restrict__ list_n) {
    after_previous();
    const uint32_t h = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    bool some = false;
    if (h < nsuper) {
        const uint4 c4 = *reinterpret_cast<const uint4*>(cells + 4 * (size_t)h);
        const uint32_t c[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (c[u] != C16_NONE) some |= cs[c[u]] != cs[c[u] + 1];
    }
    if (h <= nsuper) base[h] = 0u;
    const uint32_t m = __ballot_sync(0xffffffffu, some);
    uint32_t at = 0;
    if (lane == 0 && m) at = atomicAdd(list_n, __popc(m));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (some) list[at + __popc(m & ((1u << lane) - 1u))] = h;
}

// The linked cell of a warp: its own number, or its place in the list of
// occupied ones (list not null; C16_NONE past the end of either).
__device__ __forceinline__ uint32_t c16_cell_of(uint32_t warp, uint32_t nsuper, const uint32_t* __restrict__ list,
                                                const uint32_t* __restrict__ list_n) {
    if (!list) return warp < nsuper ? warp : C16_NONE;
    return warp < *list_n ? list[warp] : C16_NONE;
}

// Rows of linked cell h (its up to 4 cells of the sorted grid).
__global__ void __launch_bounds__(256) k_c16_count(C16Flag F, const uint32_t* __restrict__ cells, uint32_t nsuper,
                                                   const uint32_t* __restrict__ list,
                                                   const uint32_t* __restrict__ list_n,
                                                   const uint32_t* __restrict__ cs, uint32_t* __restrict__ base,
                                                   uint32_t* __restrict__ stats) {
    after_previous();
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t lane = threadIdx.x & 31;
    if (blockIdx.x == 0 && threadIdx.x < C16_STATS) stats[threadIdx.x] = 0u;
    if (warp == nsuper && !list && lane == 0) base[nsuper] = 0u;  // the scan leaves R there
    const uint32_t h = c16_cell_of(warp, nsuper, list, list_n);
    if (h == C16_NONE) return;
    uint32_t n = 0;
    const uint4 c4 = *reinterpret_cast<const uint4*>(cells + 4 * (size_t)h);
    const uint32_t c[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
    for (int u = 0; u < 4; u++) {
        if (c[u] == C16_NONE) continue;
        const uint32_t lo = cs[c[u]], hi = cs[c[u] + 1];
        for (uint32_t i = lo + lane; i < hi; i += 32) n += c16_is_row(F, i) ? 1u : 0u;
    }
    n = __reduce_add_sync(0xffffffffu, n);
    if (lane == 0) base[h] = n;
}

// A batch: the scenes' rows start at multiples of 8, so that no slice (and no
// tile) spans two scenes.  dense: the scanned counts; base: the linked
// cells' first rows with the scenes' starts moved up; srow: the scenes'
// first rows and the end.  The up to 7 places left at a scene's end have no
// row (C16_NONE in the row list).
__global__ void __launch_bounds__(256) k_c16_shift(const uint32_t* __restrict__ dense, uint32_t nsuper,
                                                   const uint32_t* __restrict__ sfirst, uint32_t ns,
                                                   uint32_t* __restrict__ base, uint32_t* __restrict__ srow,
                                                   uint32_t* __restrict__ rowlist, uint32_t* __restrict__ rowcell,
                                                   uint32_t* __restrict__ nrows) {
    after_previous();
    __shared__ uint32_t first[PPE_MAX_SCENES + 1], at[PPE_MAX_SCENES + 1];
    for (uint32_t x = threadIdx.x; x <= ns; x += blockDim.x) first[x] = sfirst[x];
    if (threadIdx.x < 32) {
        uint32_t carry = 0;
        for (uint32_t s0 = 0; s0 < ns; s0 += 32) {
            const uint32_t s = s0 + threadIdx.x;
            const uint32_t v = s < ns ? (dense[sfirst[s + 1]] - dense[sfirst[s]] + 7u) & ~7u : 0u;
            uint32_t x = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, x, o);
                if ((int)threadIdx.x >= o) x += t;
            }
            if (s < ns) at[s] = carry + x - v;
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
        if (threadIdx.x == 0) at[ns] = carry;
    }
    __syncthreads();
    const uint32_t h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h <= nsuper) {
        uint32_t lo = 0, hi = ns;  // the scene of cell h (past the last: the end)
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (first[mid] <= h) lo = mid;
            else hi = mid;
        }
        base[h] = h == nsuper ? at[ns] : dense[h] - dense[first[lo]] + at[lo];
    }
    if (blockIdx.x == 0) {
        for (uint32_t s = threadIdx.x; s <= ns; s += blockDim.x) {
            srow[s] = at[s];
            if (s < ns)
                for (uint32_t k = at[s] + dense[first[s + 1]] - dense[first[s]]; k < at[s + 1]; k++)
                    rowlist[k] = rowcell[k] = C16_NONE;
        }
        if (threadIdx.x == 0) *nrows = at[ns];
    }
}

// After the scan: row numbers and the row list (in a batch also the list
// without the scenes' gaps, of dense_n rows).  A particle without a row gets
// the identity row of the particle-indexed arrays.
struct C16RowArgs {
    const uint32_t *cells, *cs, *base;
    uint32_t nsuper;
    const uint32_t *list, *list_n;  // occupied linked cells (k_c16_occupied), or null
    const uint32_t* dense;  // batch: first row of every linked cell without the gaps
    uint32_t* rowcell;      // linked cell of every row
    uint32_t *cpos, *rowlist, *nrows, *dense_list, *dense_n, *rlen;
    double* diag64;
};

__global__ void __launch_bounds__(256) k_c16_rows(C16Flag F, C16RowArgs A) {
    after_previous();
    const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (A.dense) *A.dense_n = A.dense[A.nsuper];
        else *A.nrows = A.base[A.nsuper];
    }
    const uint32_t h = c16_cell_of((blockIdx.x * blockDim.x + threadIdx.x) >> 5, A.nsuper, A.list, A.list_n);
    if (h == C16_NONE) return;
    uint32_t at = A.base[h];
    const uint32_t dd = A.dense ? at - A.dense[h] : 0u;  // gaps before this cell
    const uint4 c4 = *reinterpret_cast<const uint4*>(A.cells + 4 * (size_t)h);
    const uint32_t c[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
    for (int u = 0; u < 4; u++) {
        if (c[u] == C16_NONE) continue;
        const uint32_t lo = A.cs[c[u]], hi = A.cs[c[u] + 1];
        for (uint32_t i0 = lo; i0 < hi; i0 += 32) {
            const uint32_t i = i0 + lane;
            const bool f = i < hi && c16_is_row(F, i);
            const uint32_t m = __ballot_sync(0xffffffffu, f);
            if (f) {
                const uint32_t k = at + __popc(m & lt);
                A.cpos[i] = k;
                A.rowlist[k] = i;
                A.rowcell[k] = h;
                if (A.dense) A.dense_list[k - dd] = i;
            } else if (i < hi) {
                A.cpos[i] = C16_NONE;
                A.rlen[i] = PPE_DIRICHLET;
                A.diag64[i] = 1.0;
            }
            at += __popc(m);
        }
    }
}

// ---------------------------------------------------------------- assembly
struct C16AsmArgs {
    StageArgs a;
    C16Assemble K;
    const PpeScene* scenes;
    const uint32_t* rowlist;
    const uint32_t* nrows;
    const uint32_t* cpos;
    uint32_t* cols;   // row-major, PPE_W a row
    float* wrm;
    uint32_t* clen;
    uint32_t* rlen;   // by particle: entries of its row
    unsigned* bar;
    double *diag64, *cb64, *cx64, *cdiag64;
    float *cdiag32, *cinv_diag, *cdsq;
    uint32_t* width;
    uint32_t maxslices;
};

// A warp a row: the neighbours within rlap of type != 2 in ascending particle
// index, those with rows appended as row numbers, every weight added to the
// diagonal (MPS_CAL_v4.0/MPS_CPU.cpp:651-698).  Bound by issued instructions:
// of some 640 candidates a third is within rlap.  The walk only tests a
// candidate; the hits collect in shared memory, and every 32 of them are
// weighed, looked up and appended together.  136,582 rows: 300 -> 240 us
// against all of it for every batch of candidates, with the row's divisions
// (now k_c16_rowend's, a thread a row).  Two and four rows a warp over the
// union of their candidates take fewer instructions and more registers:
// 20 us slower and 60 us slower.
template <bool EX, bool BT>
__global__ void __launch_bounds__(256) k_c16_assemble(C16AsmArgs A) {
    after_previous();
    __shared__ __align__(512) char rings[8][512];
    const StageArgs& a = A.a;
    const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    const uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (blockIdx.x == 0 && threadIdx.x == 0) A.bar[0] = 0u;  // the 8-byte solvers' barrier starts empty
    if (k >= *A.nrows) return;
    const uint32_t i = __ldg(A.rowlist + k);
    if (BT && i == C16_NONE) return;  // a gap between two scenes' rows
    HitRing hits(rings[threadIdx.x >> 5]);
    const float4* __restrict__ pos = a.cur.pos;
    const float4 pi = pos[i];
    const Local L = local_of<BT>(a, i);
    const Phys P = phys_of<BT>(a, L.s);
    const float re = P.rlap, thr = P.rlap_thr;
    uint32_t* cols = A.cols + (size_t)k * PPE_W;
    float* wrow = A.wrm + (size_t)k * PPE_W;
    uint32_t count = 0;
    float diag_lane = 0.f;  // a lane's few weights, then a FP64 sum over the warp
    auto weigh = [&](uint32_t at, uint32_t m) {
        const float2 h = hits.get(at + lane);
        float w = 0.f;
        uint32_t col = PPE_DIRICHLET;
        if (lane < m) {
            w = weight_rr<EX>(re, h.y);
            if (w > 0.f) col = __ldg(A.cpos + __float_as_uint(h.x));
        }
        diag_lane += w;
        const uint32_t ma = __ballot_sync(0xffffffffu, col != PPE_DIRICHLET);
        const uint32_t to = count + __popc(ma & lt);
        if (col != PPE_DIRICHLET && to < PPE_W) {
            cols[to] = col;
            wrow[to] = w;
        }
        count += __popc(ma);
    };
    const CellNear nr = cell_near(L.g, L.c, pi.x, pi.y, pi.z, re);
    flat_batches(flat_walk(L.g, L.cs, L.c, nr, lane), lane, [&](uint32_t j, bool in) {
        const float4 pj = __ldg(pos + j);
        const float dx = fsub<EX>(pj.x, pi.x), dy = fsub<EX>(pj.y, pi.y), dz = fsub<EX>(pj.z, pi.z);
        const float rr = dot3<EX>(dx, dy, dz, dx, dy, dz);
        const bool hit = in && ptype(pj) != T_DUMMY && rr < thr && j != i;
        hits.add(lane, hit, j, rr, weigh);
    });
    hits.rest(weigh);
    const double d = warp_sum_d((double)diag_lane);
    if (lane) return;
    if (count > PPE_W) {
        atomicOr(&a.sc->err, ERR_CAPACITY);  // more than PPE_W neighbours
        count = PPE_W;
    }
    A.clen[k] = count;
    A.rlen[i] = count;
    A.cdiag64[k] = d;
}

// chunks of the slice of rows k / 8 (every thread of a warp calls it)
__device__ __forceinline__ void c16_slice_width(uint32_t k, uint32_t len, const C16AsmArgs& A) {
#pragma unroll
    for (int o = 1; o < (int)C16_ROWS; o <<= 1) len = max(len, __shfl_xor_sync(0xffffffffu, len, o));
    const uint32_t s = k / C16_ROWS;
    if (k % C16_ROWS == 0 && s <= A.maxslices) A.width[s] = (len + 15u) / 16u;
}

// A thread a row: its diagonal from the weights' sum and its vectors; and the
// chunks of every slice (the longest of its 8 rows), scanned next.  A gap
// between two scenes' rows is an identity row with b = 0.
template <bool BT>
__global__ void __launch_bounds__(256) k_c16_rowend(C16AsmArgs A) {
    after_previous();
    const StageArgs& a = A.a;
    const uint32_t R = *A.nrows;
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t i = k < R ? A.rowlist[k] : C16_NONE;
    uint32_t len = 0;
    if (i != C16_NONE) {
        len = A.clen[k];
        double n0 = A.K.n0, b_tmp = A.K.b_tmp, rlan0 = A.K.rho_lambda_alpha_n0;
        uint32_t s = 0;
        if (BT) {
            s = a.batch.sid_of_id[a.cur.id[i]];
            const PpeScene& ps = A.scenes[s];
            n0 = ps.n0;
            b_tmp = ps.b_tmp;
            rlan0 = ps.rho_lambda_alpha_n0;
        }
        const double dt = (double)dt_of<BT>(a, s);
        const double dg = -A.cdiag64[k] - rlan0 / (A.K.dim2 * dt * dt);
        A.diag64[i] = dg;
        A.cdiag64[k] = dg;
        A.cdiag32[k] = (float)dg;
        A.cinv_diag[k] = (float)(1.0 / dg);
        A.cdsq[k] = (float)(1.0 / sqrt(-dg));
        A.cb64[k] = b_tmp * (n0 - (double)a.cur.n[i]);
        A.cx64[k] = (double)a.cur.press[i];
    } else if (BT && k < R) {
        A.clen[k] = 0;
        A.cdiag64[k] = -1.0;
        A.cdiag32[k] = -1.f;
        A.cinv_diag[k] = -1.f;
        A.cdsq[k] = 1.f;
        A.cb64[k] = 0.0;
        A.cx64[k] = 0.0;
    }
    c16_slice_width(k, len, A);
}

// ---------------------------------------------------------------- Crank-Nicolson viscosity
// The system of ppe.cu's k_cn_assemble (every neighbour in the diagonal, the
// ones that are no rows moved to the right-hand side) for the rows of this
// layout: hits weighed 32 at a time as in k_c16_assemble.
struct C16CnArgs {
    C16AsmArgs A;
    int c;                          // velocity component
    uint32_t* moved;                // by component (cn_reach)
    double lambda_n0_over_dim_niu;  // 1/R = this / dt
};

__device__ __forceinline__ float c16_comp(const float4& v, int c) { return c == 0 ? v.x : (c == 1 ? v.y : v.z); }

template <bool EX>
__global__ void __launch_bounds__(256) k_c16_cn_assemble(C16CnArgs C) {
    after_previous();
    __shared__ __align__(512) char rings[8][512];
    const C16AsmArgs& A = C.A;
    const StageArgs& a = A.a;
    const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    const uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (blockIdx.x == 0 && threadIdx.x == 0) C.moved[C.c] = 0u;
    if (k >= *A.nrows) return;
    const uint32_t i = __ldg(A.rowlist + k);
    HitRing hits(rings[threadIdx.x >> 5]);
    const float4* __restrict__ pos = a.cur.pos;
    const float4* __restrict__ vel = a.cur.vel;
    const float4 pi = pos[i];
    const double ui = (double)c16_comp(vel[i], C.c);
    const Local L = local_of<false>(a, i);
    const float re = a.P.rlap, thr = a.P.rlap_thr;
    uint32_t* cols = A.cols + (size_t)k * PPE_W;
    float* wrow = A.wrm + (size_t)k * PPE_W;
    uint32_t count = 0;
    double diag = 0.0, bi = 0.0;
    auto weigh = [&](uint32_t at, uint32_t m) {
        const float2 h = hits.get(at + lane);
        uint32_t col = C16_NONE;
        float w = 0.f;
        if (lane < m) w = weight_rr<EX>(re, h.y);
        if (w > 0.f) {
            const uint32_t j = __float_as_uint(h.x);
            const double uj = (double)c16_comp(__ldg(vel + j), C.c);
            col = __ldg(A.cpos + j);
            bi -= (uj - ui) * (double)w;
            if (col == C16_NONE) bi -= (double)w * uj;
        }
        diag += (double)w;
        const uint32_t ma = __ballot_sync(0xffffffffu, col != C16_NONE);
        const uint32_t to = count + __popc(ma & lt);
        if (col != C16_NONE && to < PPE_W) {
            cols[to] = col;
            wrow[to] = w;
        }
        count += __popc(ma);
    };
    const CellNear nr = cell_near(L.g, L.c, pi.x, pi.y, pi.z, cn_reach(re, C.moved, C.c));
    flat_batches(flat_walk(L.g, L.cs, L.c, nr, lane), lane, [&](uint32_t j, bool in) {
        const float4 pj = __ldg(pos + j);
        const float dx = fsub<EX>(pj.x, pi.x), dy = fsub<EX>(pj.y, pi.y), dz = fsub<EX>(pj.z, pi.z);
        const float rr = dot3<EX>(dx, dy, dz, dx, dy, dz);
        hits.add(lane, in && rr < thr && j != i, j, rr, weigh);
    });
    hits.rest(weigh);
    diag = warp_sum_d(diag);
    bi = warp_sum_d(bi);
    if (lane) return;
    if (count > PPE_W) {
        atomicOr(&a.sc->err, ERR_CAPACITY);
        count = PPE_W;
    }
    A.clen[k] = count;
    A.cdiag64[k] = diag;
    A.cb64[k] = bi;
}

__global__ void __launch_bounds__(256) k_c16_cn_rowend(C16CnArgs C) {
    after_previous();
    const C16AsmArgs& A = C.A;
    const StageArgs& a = A.a;
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    const bool row = k < *A.nrows;
    if (row) {
        const double ui = (double)c16_comp(a.cur.vel[A.rowlist[k]], C.c);
        const double one_over_R = C.lambda_n0_over_dim_niu / (double)a.sc->dt;
        const double dg = -A.cdiag64[k] - one_over_R;
        A.cdiag64[k] = dg;
        A.cdiag32[k] = (float)dg;
        A.cinv_diag[k] = (float)(1.0 / dg);
        A.cb64[k] -= one_over_R * ui + C.lambda_n0_over_dim_niu * (double)a.sc->g_eff[C.c];
        A.cx64[k] = ui;
    }
    c16_slice_width(k, row ? A.clen[k] : 0u, A);
}

// MPS_CPU_IMPL::updatePosVel<dir> (MPS_CAL_v4.0/MPS_CPU_IMPL.cpp:129-190):
// fluid u_c = x, x_c += dt u_c.
__global__ void __launch_bounds__(256) k_c16_cn_finish(const double* __restrict__ cx64, const uint32_t* __restrict__ cpos,
                                                       State s, int c, const Scalars* __restrict__ sc,
                                                       uint32_t* __restrict__ moved) {
    after_previous();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t k = i < sc->np ? cpos[i] : C16_NONE;
    float step = 0.f;
    if (k != C16_NONE) {
        const float x = (float)cx64[k];
        float4 u = s.vel[i], p = s.pos[i];
        step = __fmul_rn(sc->dt, x);
        const float at = __fadd_rn(c16_comp(p, c), step);
        if (c == 0) { u.x = x; p.x = at; }
        else if (c == 1) { u.y = x; p.y = at; }
        else { u.z = x; p.z = at; }
        s.vel[i] = u;
        s.pos[i] = p;
    }
    block_max_abs(step, moved + c);
}

// Weight of the slices before s when tiles are cut.
__device__ __forceinline__ uint64_t c16_weight(const uint32_t* __restrict__ off, uint32_t s) {
    return (uint64_t)__ldg(off + s) + (uint64_t)C16_SLICE_COST * s;
}

// A batch's tiles: tb[s] = first tile of scene s, tb[ns] = all of them.  One
// tile a scene, the rest by weight, what rounding leaves to the scenes with
// the heaviest tiles.
__global__ void __launch_bounds__(32) k_c16_cut(const uint32_t* __restrict__ off, const uint32_t* __restrict__ srow,
                                                const uint32_t* __restrict__ nrows, uint32_t ns, uint32_t G,
                                                uint32_t* __restrict__ tb) {
    after_previous();
    constexpr uint32_t PER = PPE_MAX_SCENES / 32;
    const uint32_t lane = threadIdx.x, R = *nrows, T = c16_tiles(R, G, ns);
    const double W = (double)c16_weight(off, R / C16_ROWS);
    double w[PER];
    uint32_t n[PER], given = 0;
#pragma unroll
    for (uint32_t u = 0; u < PER; u++) {
        const uint32_t s = u * 32 + lane;
        w[u] = s < ns ? (double)(c16_weight(off, srow[s + 1] / C16_ROWS) - c16_weight(off, srow[s] / C16_ROWS)) : -1.0;
        n[u] = s < ns ? 1u + (W > 0.0 ? (uint32_t)((double)(T - ns) * (w[u] / W)) : 0u) : 0u;
        given += n[u];
    }
    given = __reduce_add_sync(0xffffffffu, given);
    for (; given < T; given++) {
        double most = -2.0;
        uint32_t at = 0;
#pragma unroll
        for (uint32_t u = 0; u < PER; u++) {
            const double load = n[u] ? w[u] / n[u] : -2.0;
            if (load > most) { most = load; at = u * 32 + lane; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double m2 = __shfl_xor_sync(0xffffffffu, most, o);
            const uint32_t a2 = __shfl_xor_sync(0xffffffffu, at, o);
            if (m2 > most || (m2 == most && a2 < at)) { most = m2; at = a2; }
        }
#pragma unroll
        for (uint32_t u = 0; u < PER; u++)
            if (at == u * 32 + lane) n[u]++;
    }
    uint32_t carry = 0;
#pragma unroll
    for (uint32_t u = 0; u < PER; u++) {
        uint32_t x = n[u];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, x, o);
            if ((int)lane >= o) x += t;
        }
        if (u * 32 + lane <= ns) tb[u * 32 + lane] = carry + x - n[u];
        carry += __shfl_sync(0xffffffffu, x, 31);
    }
    if (lane == 0) tb[ns] = carry;
}

// ---------------------------------------------------------------- pack
// smallest x in [0, n] with x == n or f(x) >= v, f ascending; a whole warp
// probes 32 places a round
template <class F>
__device__ __forceinline__ uint32_t warp_lower(uint32_t n, uint64_t v, F f) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t x = lo + lane * step;
        const uint32_t below = __popc(__ballot_sync(0xffffffffu, x < hi && f(x) < v));
        if (below == 0) break;
        hi = min(hi, lo + below * step);
        lo += (below - 1) * step + 1;
    }
    return lo;
}

struct C16PackArgs {
    const uint32_t* cols_rm;  // row numbers of the columns, row-major by row
    const float* w_rm;
    const uint32_t* clen;
    const uint32_t* nrows;
    const uint32_t* off;
    const uint32_t* base;     // first row of every linked cell
    const uint32_t* nbr;      // 27 linked cells around each (C16_NONE: outside)
    const uint32_t* rowcell;  // linked cell of every row
    uint32_t blocks;
    uint32_t ns;              // scenes of a batch (0: a single scene)
    const uint32_t* srow;     // their first rows
    const uint32_t* tb;       // and first tiles
    C16Tile* tiles;
    uint32_t* collist;        // C16_COLS per tile
    unsigned char* ent;
    uint32_t* stats;          // [0] entries beyond a 16-bit offset from their slice, [1] most columns, [2] most rows,
                              // [3] fours of S' given out
    // learned S' (LRN)
    const uint32_t* rowlist;
    const uint32_t* cpos;
    const uint32_t* idv;      // GEO index of each particle
    const uint32_t* index_of_id;
    const float* dsq;         // 1 / sqrt(-diagonal) by row
    const uint32_t* s_cnt;
    const uint32_t* s_col;
    const float* s_val;
    const float* s_diag;
    uint32_t np;
    const Scalars* sc;
    uint32_t* sp_first;       // C16_SP_SLICES per tile
    uint32_t* sp_ent;
    uint32_t* sp_side;
    float* sp_diag;
};

// exclusive scan of one value per thread over the block; *total the sum
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* ws, uint32_t* total) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, x, o);
        if ((int)lane >= o) x += t;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    uint32_t w = lane < nw ? ws[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, w, o);
        if ((int)lane >= o) w += t;
    }
    const uint32_t prev = __shfl_sync(0xffffffffu, w, warp ? warp - 1 : 0u);
    *total = __shfl_sync(0xffffffffu, w, 31);
    __syncthreads();
    return (warp ? prev : 0u) + x - v;
}

__device__ __forceinline__ uint32_t sp_bf16_bits(float v) {
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v));
}

// S' of a tile: 32-row slices of its rows, each as wide as its longest row,
// in fours of words; four f of local row k is at first[k / 32] + 32 f + k % 32.
// One block per tile.  The rows its entries can name are those of the linked
// cells around its own ones; their 256-row pages get consecutive slots, the
// columns in use (other than its own rows) a bit each in their page's slot,
// and a column's position in the tile's list is the number of bits before
// it.  With the learned preconditioner the columns of S' are marked too, and
// S' is coded the same way, one thread per row.
template <bool LRN>
__global__ void __launch_bounds__(C16_PACK_THREADS) k_c16_pack(C16PackArgs A) {
    after_previous();
    extern __shared__ uint16_t page_slot[];  // slot of every page of rows (0xffff: none)
    __shared__ uint2 bits[C16_PAGES * 8];    // columns in use, and those before the word
    __shared__ uint32_t slot_page[C16_PAGES];
    __shared__ uint32_t ws[32], found[2], cell[C16_PACK_THREADS], ncell;
    const uint32_t R = *A.nrows;
    const uint32_t nsl = (R + C16_ROWS - 1) / C16_ROWS;
    const uint32_t T = c16_tiles(R, A.blocks, A.ns);
    const uint32_t t = blockIdx.x, tid = threadIdx.x, nthr = blockDim.x;
    const uint32_t lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
    if (t >= T) return;
    // equal shares of the chunks of the tile's scene, a slice counting
    // C16_SLICE_COST more
    uint32_t scene = 0, t0 = 0, t1 = T, lo = 0, hi = nsl;
    if (A.ns) {
        scene = warp_lower(A.ns, (uint64_t)t + 1, [&](uint32_t x) { return (uint64_t)__ldg(A.tb + x); }) - 1;
        t0 = __ldg(A.tb + scene);
        t1 = __ldg(A.tb + scene + 1);
        lo = __ldg(A.srow + scene) / C16_ROWS;
        hi = __ldg(A.srow + scene + 1) / C16_ROWS;
    }
    if (warp < 2) {
        const uint64_t w0 = c16_weight(A.off, lo), w1 = c16_weight(A.off, hi);
        const uint32_t s = warp_lower(nsl, w0 + (w1 - w0) * (t - t0 + warp) / (t1 - t0),
                                      [&](uint32_t x) { return c16_weight(A.off, x); });
        if (lane == 0) found[warp] = t + warp == t1 ? hi : s;
    }
    const uint32_t npages = (R + C16_PAGE - 1) / C16_PAGE;
    for (uint32_t p = tid; p < npages; p += nthr) page_slot[p] = 0;
    __syncthreads();
    const uint32_t s0 = found[0], s1 = found[1];
    if (s0 >= s1) {
        if (tid == 0) A.tiles[t] = C16Tile{s0, s0, 0u, 0u, 0u, scene, {0u, 0u}};
        return;
    }
    const uint32_t r0 = s0 * C16_ROWS, r1 = min(s1 * C16_ROWS, R), rows = r1 - r0;
    // the linked cells of its rows, a thread a row, and what is around each
    for (uint32_t k0 = r0; k0 < r1; k0 += nthr) {
        if (tid == 0) ncell = 0u;
        __syncthreads();
        const uint32_t k = k0 + tid;
        const uint32_t h = k < r1 ? __ldg(A.rowcell + k) : C16_NONE;
        if (h != C16_NONE && (k == r0 || __ldg(A.rowcell + k - 1) != h)) cell[atomicAdd(&ncell, 1u)] = h;
        __syncthreads();
        for (uint32_t x = tid; x < ncell * 27u; x += nthr) {
            const uint32_t nb = __ldg(A.nbr + (size_t)cell[x / 27u] * 27 + x % 27u);
            if (nb == C16_NONE) continue;
            const uint32_t lo = __ldg(A.base + nb), hi = __ldg(A.base + nb + 1);
            if (lo < hi)
                for (uint32_t p = lo / C16_PAGE; p <= (hi - 1) / C16_PAGE; p++) page_slot[p] = 1;
        }
        __syncthreads();
    }
    // slots in page order
    uint32_t nslots;
    {
        const uint32_t per = (npages + nthr - 1) / nthr;
        const uint32_t p0 = min(tid * per, npages), p1 = min(p0 + per, npages);
        uint32_t c = 0;
        for (uint32_t p = p0; p < p1; p++) c += page_slot[p];
        uint32_t slot = block_scan(c, ws, &nslots);
        for (uint32_t p = p0; p < p1; p++) {
            if (page_slot[p] && slot < C16_PAGES) {
                slot_page[slot] = p;
                page_slot[p] = (uint16_t)slot++;
            } else {
                page_slot[p] = 0xffffu;
            }
        }
        nslots = min(nslots, C16_PAGES);
    }
    const uint32_t words = nslots * 8;
    for (uint32_t w = tid; w < words; w += nthr) bits[w].x = 0u;
    __syncthreads();
    auto mark = [&](uint32_t col) {
        if (col - r0 < rows) return;
        const uint32_t s = page_slot[col / C16_PAGE];
        if (s == 0xffffu) return;
        uint32_t* w = &bits[s * 8 + ((col / 32) & 7u)].x;
        const uint32_t b = 1u << (col & 31u);
        if (!(*(volatile uint32_t*)w & b)) atomicOr(w, b);
    };
    // a warp per row, eight of a lane's entries at a time
    for (uint32_t k = r0 + warp; k < r1; k += nwarps) {
        const uint32_t* rc = A.cols_rm + (size_t)k * PPE_W;
        const uint32_t len = __ldg(A.clen + k);
        for (uint32_t e0 = lane; e0 < len; e0 += 256) {
            uint32_t col[8];
#pragma unroll
            for (int u = 0; u < 8; u++) col[u] = e0 + 32u * u < len ? __ldg(rc + e0 + 32u * u) : r0;
#pragma unroll
            for (int u = 0; u < 8; u++) mark(col[u]);
        }
    }
    // the row of stored neighbour u of a row with GEO index id (C16_NONE: none now)
    auto sp_row_of = [&](uint32_t id, uint32_t u) -> uint32_t {
        const uint32_t j = __ldg(A.index_of_id + __ldg(A.s_col + (size_t)id * LP_GW + u));
        return j < A.sc->np ? __ldg(A.cpos + j) : C16_NONE;
    };
    if (LRN) {
        for (uint32_t x = tid; x < rows * 8u; x += nthr) {  // eight threads a row
            const uint32_t i = __ldg(A.rowlist + r0 + x / 8u);
            if (i == C16_NONE) continue;
            const uint32_t id = __ldg(A.idv + i);
            const uint32_t n = __ldg(A.s_cnt + id);
            for (uint32_t u = x & 7u; u < n; u += 8) {
                const uint32_t col = sp_row_of(id, u);
                if (col != C16_NONE) mark(col);
            }
        }
    }
    __syncthreads();
    // the columns before every word, the list
    uint32_t* list = A.collist + (size_t)t * C16_COLS;
    for (uint32_t k = tid; k < rows; k += nthr) list[k] = r0 + k;
    const uint32_t wper = (words + nthr - 1) / nthr;
    const uint32_t w0 = min(tid * wper, words), w1 = min(w0 + wper, words);
    uint32_t c = 0, ncol;
    for (uint32_t w = w0; w < w1; w++) c += __popc(bits[w].x);
    uint32_t at = rows + block_scan(c, ws, &ncol);
    for (uint32_t w = w0; w < w1; w++) {
        bits[w].y = at;
        uint32_t m = bits[w].x;
        const uint32_t c0 = slot_page[w >> 3] * C16_PAGE + (w & 7u) * 32u;
        while (m) {
            const uint32_t b = __ffs(m) - 1;
            m &= m - 1;
            if (at < C16_COLS) list[at] = c0 + b;
            at++;
        }
    }
    ncol = min(ncol + rows, C16_COLS);
    __syncthreads();
    // position of a column in the list, C16_NONE when it is not there
    auto local_of = [&](uint32_t col) -> uint32_t {
        if (col - r0 < rows) return col - r0;
        const uint32_t s = page_slot[col / C16_PAGE];
        if (s == 0xffffu) return C16_NONE;
        const uint2 b = bits[s * 8 + ((col / 32) & 7u)];
        const uint32_t p = b.y + __popc(b.x & ((1u << (col & 31u)) - 1u));
        return p < C16_COLS ? p : C16_NONE;
    };
    uint32_t far = 0, nesc = 0, wmax = 0;
    for (uint32_t s = s0 + warp; s < s1; s += nwarps) {
        const uint32_t r = lane & 7u, q = lane >> 3;
        const uint32_t g0 = __ldg(A.off + s), nch = __ldg(A.off + s + 1) - g0;
        wmax = max(wmax, nch);
        const uint32_t k = s * C16_ROWS + r;
        const uint32_t len = k < R ? __ldg(A.clen + k) : 0u;
        const uint4* rc = reinterpret_cast<const uint4*>(A.cols_rm + (size_t)min(k, R - 1) * PPE_W);
        const float4* rw = reinterpret_cast<const float4*>(A.w_rm + (size_t)min(k, R - 1) * PPE_W);
        const uint32_t padcode = 4u * min(k - r0, rows - 1);  // the row itself, weight 0
#pragma unroll 2
        for (uint32_t x = 0; x < nch; x++) {
            const uint32_t e = 16u * x + 4u * q;
            uint4 cv = make_uint4(0, 0, 0, 0);
            float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
            if (e < len) {
                cv = __ldg(rc + 4u * x + q);
                w = __ldg(rw + 4u * x + q);
            }
            const uint32_t cc[4] = {cv.x, cv.y, cv.z, cv.w};
            uint32_t code[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                code[u] = padcode;
                if (e + u >= len) continue;
                const uint32_t p = local_of(cc[u]);
                const int d = (int)cc[u] - (int)(s * C16_ROWS) + 32768;
                if (d < 0 || d >= (int)C16_ESC) far++;
                if (p == C16_NONE) {
                    code[u] = C16_ESC;
                    nesc++;
                } else {
                    code[u] = 4u * p;
                }
            }
            if (e + 1 >= len) w.y = 0.f;
            if (e + 2 >= len) w.z = 0.f;
            if (e + 3 >= len) w.w = 0.f;
            unsigned char* dst = A.ent + (size_t)(g0 + x) * C16_CHUNK_BYTES;
            *reinterpret_cast<float4*>(dst + 16u * lane) = w;
            *reinterpret_cast<uint2*>(dst + 512u + 8u * lane) =
                make_uint2(code[0] | (code[1] << 16), code[2] | (code[3] << 16));
        }
    }
    if (LRN) {
        // the widths from the stored counts (rows' kept entries are at most
        // those; the rest are zeros), then the tile's place in the array
        __shared__ uint32_t first[C16_SP_SLICES + 1];
        const uint32_t nsp = (rows + SP_SLICE - 1) / SP_SLICE;
        for (uint32_t j = warp; j < nsp; j += nwarps) {
            const uint32_t k = j * SP_SLICE + lane;
            const uint32_t i = k < rows ? __ldg(A.rowlist + r0 + k) : C16_NONE;
            const uint32_t n = i != C16_NONE ? (__ldg(A.s_cnt + __ldg(A.idv + i)) + 3u) / 4u : 0u;
            const uint32_t w = __reduce_max_sync(0xffffffffu, n);
            if (lane == 0) first[j + 1] = w * SP_SLICE;
        }
        __syncthreads();
        if (tid == 0) {
            uint32_t n = 0;
            for (uint32_t j = 0; j < nsp; j++) n += first[j + 1];
            first[0] = atomicAdd(A.stats + 3, n);
            for (uint32_t j = 0; j < nsp; j++) first[j + 1] += first[j];
        }
        __syncthreads();
        for (uint32_t j = tid; j <= nsp; j += nthr) A.sp_first[(size_t)t * C16_SP_SLICES + j] = first[j];
        // a pair without a row now is left out (of both its rows), which
        // keeps S' symmetric and diagonally dominant
        for (uint32_t k = tid; k < rows; k += nthr) {
            const uint32_t i = __ldg(A.rowlist + r0 + k);
            const uint32_t id = i != C16_NONE ? __ldg(A.idv + i) : 0u;
            const uint32_t n = i != C16_NONE ? __ldg(A.s_cnt + id) : 0u;
            const float di = __ldg(A.dsq + r0 + k);
            A.sp_diag[r0 + k] = i != C16_NONE ? __ldg(A.s_diag + id) * (di * di) : 1.f;
            const uint32_t f0 = first[k / SP_SLICE], words = (first[k / SP_SLICE + 1] - f0) / SP_SLICE * 4u;
            auto place = [&](uint32_t w) { return ((size_t)f0 + w / 4u * SP_SLICE + k % SP_SLICE) * 4u + (w & 3u); };
            uint32_t m = 0;
            for (uint32_t u0 = 0; u0 < n; u0 += 8) {
                uint32_t col[8];
#pragma unroll
                for (uint32_t b = 0; b < 8; b++) col[b] = u0 + b < n ? sp_row_of(id, u0 + b) : C16_NONE;
                float v[8];
#pragma unroll
                for (uint32_t b = 0; b < 8; b++)
                    v[b] = col[b] == C16_NONE
                               ? 0.f
                               : __ldg(A.s_val + (size_t)id * LP_GW + u0 + b) * (di * __ldg(A.dsq + col[b]));
#pragma unroll
                for (uint32_t b = 0; b < 8; b++) {
                    if (col[b] == C16_NONE) continue;
                    const uint32_t p = local_of(col[b]);
                    if (p == C16_NONE) {
                        A.sp_side[place(m)] = col[b];
                        nesc++;
                    }
                    A.sp_ent[place(m)] = ((p == C16_NONE ? C16_ESC : 4u * p) << 16) | sp_bf16_bits(v[b]);
                    m++;
                }
            }
            for (; m < words; m++) A.sp_ent[place(m)] = 0u;
        }
    }
    far = __reduce_add_sync(0xffffffffu, far);
    if (lane == 0 && far) atomicAdd(A.stats, far);
    if (lane == 0) ws[warp] = wmax;
    const int any = __syncthreads_or((int)nesc);
    if (tid == 0) {
        for (uint32_t w = 0; w < nwarps; w++) wmax = max(wmax, ws[w]);
        A.tiles[t] = C16Tile{s0, s1, ncol, any ? 1u : 0u, wmax, scene, {0u, 0u}};
        atomicMax(A.stats + 1, ncol);
        atomicMax(A.stats + 2, rows);
    }
}

// p = max(x, 0) for the rows, 0 for Dirichlet particles (pressCorr,
// MPS_CAL_v4.0/MPS_CPU.cpp:734-743).
__global__ void __launch_bounds__(256) k_c16_finish(const double* __restrict__ cx64, const uint32_t* __restrict__ cpos,
                                                    float* __restrict__ press, const Scalars* __restrict__ sc) {
    after_previous();
    const uint32_t n = sc->np;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float p = 0.f;
    const uint32_t k = cpos[i];
    if (k != C16_NONE) {
        p = (float)cx64[k];
        if (p < 0.f) p = 0.f;
    }
    press[i] = p;
}

// Export: the stored entries of every row as particle indices, at
// row_start[i] (the particle's list) in stored order.  One block per tile.
__global__ void __launch_bounds__(256) k_c16_export(const C16Tile* __restrict__ tiles,
                                                    const uint32_t* __restrict__ collist, uint32_t blocks, uint32_t ns,
                                                    const uint32_t* __restrict__ clen,
                                                    const uint32_t* __restrict__ rowlist,
                                                    const uint32_t* __restrict__ nrows, const uint32_t* __restrict__ off,
                                                    const unsigned char* __restrict__ ent,
                                                    const uint32_t* __restrict__ cols_rm,
                                                    const uint32_t* __restrict__ row_start, uint32_t* __restrict__ cols,
                                                    float* __restrict__ out_w) {
    const uint32_t R = *nrows;
    if (blockIdx.x >= c16_tiles(R, blocks, ns)) return;
    const C16Tile ti = tiles[blockIdx.x];
    const uint32_t lane = threadIdx.x & 31, r = lane & 7u, q = lane >> 3;
    for (uint32_t s = ti.s0 + (threadIdx.x >> 5); s < ti.s1; s += blockDim.x >> 5) {
        const uint32_t k = s * C16_ROWS + r;
        if (k >= R) continue;
        const uint32_t g0 = off[s], W = off[s + 1] - g0;
        const uint32_t len = clen[k];
        if (len == 0) continue;
        const uint32_t o = row_start[rowlist[k]];
        for (uint32_t x = 0; x < W; x++)
            for (uint32_t u = 0; u < 4; u++) {
                const uint32_t e = 16u * x + 4u * q + u;  // the pack's order (k_c16_pack)
                if (e >= len) continue;
                const unsigned char* src = ent + (size_t)(g0 + x) * C16_CHUNK_BYTES;
                const uint32_t c = reinterpret_cast<const uint16_t*>(src + 512)[4u * lane + u];
                const uint32_t col = c == C16_ESC ? cols_rm[(size_t)k * PPE_W + e]
                                                  : collist[(size_t)blockIdx.x * C16_COLS + c / 4u];
                cols[o + e] = rowlist[col];
                out_w[o + e] = reinterpret_cast<const float*>(src)[4u * lane + u];
            }
    }
}

// ---------------------------------------------------------------- learned S'
// S' (its layout: ppe_device.cuh) of the current rows, from S kept by GEO
// index (learned.cuh): row position k holds its FP32 diagonal and its stored
// neighbours that are rows now.  A pair whose columns lie farther apart than
// 32,767 is left out from both its rows, which keeps S' symmetric and
// diagonally dominant (S is built dominant with a 1 % margin, more than BF16
// rounding of the entries takes away, so S' stays SPD).  Columns are particle
// indices in every solver.
struct SpArgs {
    const uint32_t* rowlist;
    const uint32_t* nrows;
    const uint32_t* idv;       // GEO index of each particle
    const uint32_t* index_of_id;
    const uint32_t* rlen;
    const double* diag64;      // particle-indexed diagonal of A
    const uint32_t* s_cnt;
    const uint32_t* s_col;
    const float* s_val;
    const float* s_diag;
    const Scalars* sc;
    uint32_t* off;             // widths (entries), then the scanned first entries
    uint32_t* ent;
    float* diag;
    uint32_t maxslices;
};

// The pack takes a thread per row (lane = row of the 32-row slice, so the
// packed words leave as coalesced 128-byte rows) and eight of its stored
// neighbours at a time, their loads issued together: the chain s_col ->
// index_of_id -> rlen, diag64 costs three dependent rounds per eight
// entries instead of per entry.
constexpr uint32_t SP_BATCH = 8;

// the batch [u0, u0 + 8) of the stored neighbours of a row with own column
// c: kept or not, the column offset and the neighbour's particle index
__device__ __forceinline__ void sp_batch(const SpArgs& A, uint32_t id, uint32_t n, uint32_t u0, uint32_t np,
                                         uint32_t c, bool (&ok)[SP_BATCH], int (&d)[SP_BATCH],
                                         uint32_t (&j)[SP_BATCH]) {
    uint32_t jd[SP_BATCH];
#pragma unroll
    for (uint32_t b = 0; b < SP_BATCH; b++)
        jd[b] = u0 + b < n ? __ldg(A.s_col + (size_t)id * LP_GW + u0 + b) : 0u;
#pragma unroll
    for (uint32_t b = 0; b < SP_BATCH; b++) j[b] = u0 + b < n ? __ldg(A.index_of_id + jd[b]) : np;
    uint32_t len[SP_BATCH];
#pragma unroll
    for (uint32_t b = 0; b < SP_BATCH; b++) {
        len[b] = j[b] < np ? __ldg(A.rlen + j[b]) : PPE_DIRICHLET;
    }
#pragma unroll
    for (uint32_t b = 0; b < SP_BATCH; b++) {
        d[b] = (int)j[b] - (int)c;
        ok[b] = len[b] != PPE_DIRICHLET && d[b] >= -32767 && d[b] <= 32767;
    }
}

// Pass 1: off[s] = 32 x (the most stored entries of a row of slice s), every
// slice up to maxslices.  The stored count bounds the kept entries (the pack
// leaves out neighbours that are not rows now and far pairs, and pads the
// row with zeros), so this pass reads one count a row instead of following
// every entry to its row.
__global__ void __launch_bounds__(256) k_sp_width(SpArgs A) {
    after_previous();
    const uint32_t R = *A.nrows;
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t s = k / SP_SLICE;
    uint32_t cnt = 0;
    if (k < R) cnt = __ldg(A.s_cnt + __ldg(A.idv + __ldg(A.rowlist + k)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt = max(cnt, __shfl_xor_sync(0xffffffffu, cnt, o));
    if ((threadIdx.x & 31) == 0 && s <= A.maxslices) A.off[s] = cnt * SP_SLICE;
}

// Pass 2 (after the scan of off): the kept entries of row k in stored order,
// then zeros up to the slice's width.
__global__ void __launch_bounds__(256) k_sp_pack(SpArgs A) {
    after_previous();
    const uint32_t R = *A.nrows, np = A.sc->np;
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t s = k / SP_SLICE, lane = k % SP_SLICE;
    if (s >= (R + SP_SLICE - 1) / SP_SLICE) return;
    const uint32_t base = A.off[s], W = (A.off[s + 1] - base) / SP_SLICE;
    uint32_t t = 0;
    if (k < R) {
        const uint32_t i = __ldg(A.rowlist + k);
        const uint32_t id = __ldg(A.idv + i);
        const uint32_t n = __ldg(A.s_cnt + id);
        const float di = (float)(1.0 / sqrt(-__ldg(A.diag64 + i)));
        A.diag[k] = __ldg(A.s_diag + id) * (di * di);
        for (uint32_t u0 = 0; u0 < n; u0 += SP_BATCH) {
            bool ok[SP_BATCH];
            int d[SP_BATCH];
            uint32_t j[SP_BATCH];
            sp_batch(A, id, n, u0, np, i, ok, d, j);
            double dg[SP_BATCH];
            float sv[SP_BATCH];
#pragma unroll
            for (uint32_t b = 0; b < SP_BATCH; b++) {
                dg[b] = ok[b] ? __ldg(A.diag64 + j[b]) : -1.0;
                sv[b] = ok[b] ? __ldg(A.s_val + (size_t)id * LP_GW + u0 + b) : 0.f;
            }
#pragma unroll
            for (uint32_t b = 0; b < SP_BATCH; b++) {
                if (!ok[b]) continue;
                const float dj = (float)(1.0 / sqrt(-dg[b]));
                const float v = sv[b] * (di * dj);
                A.ent[base + SP_SLICE * t + lane] = ((uint32_t)(d[b] & 0xffff) << 16) | sp_bf16_bits(v);
                t++;
            }
        }
    }
    for (; t < W; t++) A.ent[base + SP_SLICE * t + lane] = 0u;
}

// ---------------------------------------------------------------- solve
struct C16Args {
    const uint32_t* nrows;
    const uint32_t* off;        // first chunk of every slice
    const unsigned char* ent;
    const uint32_t* cols_rm;    // the assembly's columns, PPE_W a row (of escaped entries)
    const C16Tile* tiles;
    const uint32_t* collist;
    const uint32_t* stats;      // [1] most columns and [2] most rows of a tile
    uint32_t ns;                // scenes of a batch (0: a single scene)
    const uint32_t* tb;         // their first tiles
    double* tsum;               // a batch's sums of every tile, two buffers
    int *iters, *outers;        // a batch's results by scene
    double* srel;
    const double* b64;
    const double* diag64;
    const float* diag32;
    const float* inv_diag;
    double* x64;
    float *p, *r;               // direction and residual (a block of several tiles keeps them here)
    float4* pub0;               // what other blocks read of a row, current and next
    float4* pub1;
    ulonglong2* slots;          // grid sums: the blocks' inboxes, twice
    unsigned long long* epoch;  // epochs used by the launches so far
    Scalars* sc;
    double tol, eta_min;
    uint32_t keep;              // chunks read as evict_last, over all tiles
    uint32_t ahead_from;        // chunks of the smallest matrix fetched ahead (C16_AHEAD_FROM)
    int max_iter, inner_cap, max_outer;
    uint32_t smem_chunks;       // most chunks a block holds in shared memory
    uint32_t smem_bytes;        // its dynamic shared memory
    // learned S' (LRN): codes into the tile's columns, by row
    const uint32_t* sp_first;
    const uint32_t* sp_ent;
    const uint32_t* sp_side;
    const float* sp_diag;
};

__device__ __forceinline__ uint2 ld_codes(const uint2* p, uint64_t pol) {
    uint2 v;
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.u32 {%0, %1}, [%2], %3;"
        : "=r"(v.x), "=r"(v.y)
        : "l"(p), "l"(pol));
    return v;
}

// Grid-wide sum of K doubles fused with a grid barrier, in one crossing of
// the chip: every block has an inbox with a place for each block, a block
// writes its sums into all inboxes as (value, epoch) pairs, single 16-byte
// accesses, and waits for its own inbox to fill.  No place is read by more
// than one block: with one shared place per block, 148 readers polling each
// delayed the writes to 11 us.  The sums are added in block order by a fixed
// tree, so they are the same in every block and every run.  Two inboxes: a
// block writes those of epoch e + 2 only after every block has read those of
// epoch e.  The wait is bounded: after the budget (1 s) it sets
// ERR_DEVICE_TIMEOUT and returns false.
struct C16Sync {
    ulonglong2* slots;
    unsigned long long epoch;
    Scalars* sc;
};
constexpr uint32_t C16_SUMS = 3;

template <int K>
__device__ __forceinline__ bool c16_sum(const double (&v)[K], C16Sync& sy, double* got, double (&out)[K]) {
    __shared__ double part[C16_SUMS][32];
    __shared__ double tot[C16_SUMS];
    __shared__ int bad;
    const uint32_t G = gridDim.x, tid = threadIdx.x;
    const uint32_t lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    sy.epoch++;
    ulonglong2* buf = sy.slots + (size_t)(sy.epoch & 1ull) * G * G * C16_SUMS;
#pragma unroll
    for (int k = 0; k < K; k++) {
        const double t = warp_sum_d(v[k]);
        if (lane == 0) part[k][warp] = t;
    }
    if (tid == 0) bad = 0;
    __syncthreads();
    if (warp < K) {
        const double t = warp_sum_d(lane < nw ? part[warp][lane] : 0.0);
        if (lane == 0) tot[warp] = t;
    }
    __syncthreads();
    if (tid < G * K) __threadfence();  // this block's writes before its sums
    for (uint32_t x = tid; x < G * K; x += blockDim.x)
        asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(
                         buf + ((size_t)(x / K) * G + blockIdx.x) * C16_SUMS + x % K),
                     "l"(__double_as_longlong(tot[x % K])), "l"(sy.epoch)
                     : "memory");
    for (uint32_t x = tid; x < G * K; x += blockDim.x) {
        const ulonglong2* at = buf + ((size_t)blockIdx.x * G + x / K) * C16_SUMS + x % K;
        uint64_t t0 = 0;
        for (;;) {
            long long val;
            unsigned long long ep;
            asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                         : "=l"(val), "=l"(ep)
                         : "l"(at)
                         : "memory");
            if (ep == sy.epoch) {
                got[x] = __longlong_as_double(val);
                break;
            }
            uint64_t t1;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
            if (t0 == 0) t0 = t1;
            if (t1 - t0 > wait_budget_ns(sy.sc)) {
                atomicOr(&sy.sc->err, ERR_DEVICE_TIMEOUT);
                bad = 1;
                break;
            }
        }
    }
    if (tid < G * K) __threadfence();  // the other blocks' writes after their sums
    __syncthreads();
    if (warp < K) {
        double t = 0.0;
        for (uint32_t b = lane; b < G; b += 32) t += got[b * K + warp];
        t = warp_sum_d(t);
        if (lane == 0) tot[warp] = t;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; k++) out[k] = tot[k];
    return bad == 0;
}

// What a block needs of one of its tiles (uniform over the block).
struct C16View {
    uint32_t s0, r0, rows, ns, ncol, c0, nch;
    uint32_t cpw;     // chunks per warp: the tile's chunks in equal contiguous shares
    uint32_t nseg;    // most pieces this cuts a slice into
    // of a warp's share, the last resw chunks are resident in shared memory
    // and the first keepw are read as evict_last (mat_policy; 0xFFFFFFFF:
    // default policy), so that every warp has the same mix of near and far
    uint32_t resw, keepw;
    uint32_t ahead;   // chunks a warp fetches into L2 before it loads them (C16_AHEAD)
    uint32_t esc;
    const uint32_t* cl;
    const uint32_t* spf;  // its S' slices (k_c16_pack)
    uint32_t tile, scene;
};

constexpr uint32_t C16_SEGS = 4;  // most pieces a slice's chunks are cut into

__device__ __forceinline__ uint32_t c16_align(uint32_t v) { return (v + 15u) & ~15u; }

__device__ __forceinline__ C16View c16_view(const C16Args& S, uint32_t t, uint32_t R, uint32_t C, uint32_t nwarps,
                                             uint32_t keep) {
    const C16Tile ti = S.tiles[t];
    C16View v;
    v.s0 = ti.s0;
    v.ns = ti.s1 - ti.s0;
    v.r0 = ti.s0 * C16_ROWS;
    v.rows = min(ti.s1 * C16_ROWS, R) - min(v.r0, R);
    v.ncol = ti.ncol;
    v.esc = ti.esc;
    v.c0 = __ldg(S.off + ti.s0);
    const uint32_t c1 = __ldg(S.off + ti.s1);
    v.nch = c1 - v.c0;
    // no slice in more than C16_SEGS pieces
    v.cpw = max((v.nch + nwarps - 1) / nwarps, (ti.wmax + C16_SEGS - 2) / (C16_SEGS - 1));
    v.cpw = max(v.cpw, 1u);
    v.nseg = ti.wmax ? (ti.wmax + v.cpw - 2) / v.cpw + 1 : 1u;
    v.resw = 0;
    v.keepw = keep == 0xffffffffu ? keep : (uint32_t)((uint64_t)v.cpw * min(keep, C) / C);
    v.ahead = C >= S.ahead_from ? C16_AHEAD : 0x7fffffffu;
    v.cl = S.collist + (size_t)t * C16_COLS;
    v.spf = S.sp_first + (size_t)t * C16_SP_SLICES;
    v.tile = t;
    v.scene = ti.scene;
    return v;
}

// Slice offsets of the tile, from its first chunk, and the pieces of each.
__device__ __forceinline__ void c16_slices(const C16Args& S, const C16View& v, uint32_t* soff, unsigned char* sseg) {
    for (uint32_t s = threadIdx.x; s <= v.ns; s += blockDim.x) {
        const uint32_t a = __ldg(S.off + v.s0 + s) - v.c0;
        soff[s] = a;
        if (s < v.ns) {
            const uint32_t b = __ldg(S.off + v.s0 + s + 1) - v.c0;
            sseg[s] = (unsigned char)(b > a ? (b - 1) / v.cpw - a / v.cpw + 1 : 0u);
        }
    }
}

// [p, p + bytes) into L2 ahead of its loads, by one thread of the warp
__device__ __forceinline__ void c16_fetch(const unsigned char* p, uint32_t bytes, uint64_t pol) {
    if ((threadIdx.x & 31) == 0)
        asm volatile("cp.async.bulk.prefetch.L2.global.L2::cache_hint [%0], %1, %2;" ::"l"(p), "r"(bytes), "l"(pol));
}

// The row sums of a tile's product over the staged vector (at vecb): warp w
// takes chunks [w cpw, (w + 1) cpw) whichever slices they belong to, four
// chunks' loads in flight at a time, and leaves each slice's sums (or its
// piece's) in q[piece * rs + row].  REMOTE gives the operand of a column that
// is not in the tile's list.
template <class T, bool ESC, class REMOTE>
__device__ __forceinline__ void c16_product(const C16Args& S, const C16View& v, const unsigned char* vecb,
                                            const uint32_t* soff, T* q, uint32_t rs, const unsigned char* res,
                                            REMOTE remote) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = warp * v.cpw;
    const uint32_t x1 = min(x + v.cpw, v.nch);
    if (x >= x1) return;
    uint32_t s = 0;  // the slice of chunk x: the last one that starts at or before it
    {
        uint32_t hi = v.ns;
        while (hi - s > 1) {
            const uint32_t mid = (s + hi) >> 1;
            if (soff[mid] <= x) s = mid;
            else hi = mid;
        }
    }
    uint32_t seg = warp - soff[s] / v.cpw, send = soff[s + 1];
    T a0 = 0, a1 = 0;
    auto add = [&](const uint2 cw, const float4 w, uint32_t at) {
        T o[4];
        const uint32_t c[4] = {cw.x & 0xffffu, cw.x >> 16, cw.y & 0xffffu, cw.y >> 16};
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (ESC && c[u] == C16_ESC)
                o[u] = remote(__ldg(S.cols_rm + (size_t)((v.s0 + s) * C16_ROWS + (lane & 7u)) * PPE_W +
                                    16u * (at - soff[s]) + 4u * (lane >> 3) + u));
            else
                o[u] = *reinterpret_cast<const T*>(vecb + c[u] * (sizeof(T) / 4));
        }
        a0 += (T)w.x * o[0];
        a1 += (T)w.y * o[1];
        a0 += (T)w.z * o[2];
        a1 += (T)w.w * o[3];
        if (at + 1 == send) {  // the slice ends here
            T t = a0 + a1;
            t += __shfl_xor_sync(0xffffffffu, t, 8);
            t += __shfl_xor_sync(0xffffffffu, t, 16);
            if (lane < C16_ROWS) q[seg * rs + s * C16_ROWS + lane] = t;
            a0 = 0;
            a1 = 0;
            seg = 0;
            if (at + 1 < x1) {
                do s++;
                while (soff[s + 1] == at + 1);
                send = soff[s + 1];
            }
        }
    };
    const uint32_t nres = min(v.resw, x1 - x), xs = x1 - nres;
    const uint32_t xk = v.keepw == 0xffffffffu ? v.keepw : x + v.keepw;
    // streamed chunks, in two batches of registers: one is consumed while the
    // other is on its way
    constexpr int UN = sizeof(T) == 4 ? C16_BATCH : C16_BATCH64;
    const unsigned char* src = S.ent + (size_t)(v.c0 + x) * C16_CHUNK_BYTES + 16u * lane;
    const unsigned char* srcc = src + 512u - 8u * lane;
    const uint64_t near = mat_policy(0u, xk == 0xffffffffu ? xk : 1u), far = mat_policy(1u, xk == 0xffffffffu ? xk : 0u);
    float4 wa[UN], wb[UN];
    uint2 ca[UN], cb[UN];
    uint32_t ahead = min(v.keepw, xs - x) + x + v.ahead;
    auto load = [&](float4 (&w)[UN], uint2 (&c)[UN], uint32_t at) {
        const uint64_t pol = at < xk ? near : far;
        if (ahead < xs) {
            c16_fetch(S.ent + (size_t)(v.c0 + ahead) * C16_CHUNK_BYTES,
                      min((uint32_t)UN, xs - ahead) * C16_CHUNK_BYTES, far);
            ahead += UN;
        }
#pragma unroll
        for (int u = 0; u < UN; u++) {
            w[u] = ld_mat(reinterpret_cast<const float4*>(src + u * C16_CHUNK_BYTES), pol);
            c[u] = ld_codes(reinterpret_cast<const uint2*>(srcc + u * C16_CHUNK_BYTES), pol);
        }
        src += UN * C16_CHUNK_BYTES;
        srcc += UN * C16_CHUNK_BYTES;
    };
    auto use = [&](const float4 (&w)[UN], const uint2 (&c)[UN], uint32_t at) {
#pragma unroll
        for (int u = 0; u < UN; u++) add(c[u], w[u], at + u);
    };
    uint32_t nb = (xs - x) / UN;  // whole batches
    if (nb) {
        load(wa, ca, x);
        for (; nb > 2; nb -= 2) {
            load(wb, cb, x + UN);
            use(wa, ca, x);
            load(wa, ca, x + 2 * UN);
            use(wb, cb, x + UN);
            x += 2 * UN;
        }
        if (nb == 2) {
            load(wb, cb, x + UN);
            use(wa, ca, x);
            use(wb, cb, x + UN);
        } else {
            use(wa, ca, x);
        }
        x += nb * UN;
    }
    for (; x < xs; x++) {  // and the chunks left
        const uint64_t pol = x < xk ? near : far;
        const float4 w = ld_mat(reinterpret_cast<const float4*>(src), pol);
        const uint2 c = ld_codes(reinterpret_cast<const uint2*>(srcc), pol);
        src += C16_CHUNK_BYTES;
        srcc += C16_CHUNK_BYTES;
        add(c, w, x);
    }
#pragma unroll 2
    for (; x < x1; x++) {
        const unsigned char* ch = res + (size_t)(warp * v.resw + (x - xs)) * C16_CHUNK_BYTES;
        const float4 w = *reinterpret_cast<const float4*>(ch + 16u * lane);
        const uint2 cw = *reinterpret_cast<const uint2*>(ch + 512u + 8u * lane);
        add(cw, w, x);
    }
    if (x1 < send) {  // the share ends inside its last slice
        T t = a0 + a1;
        t += __shfl_xor_sync(0xffffffffu, t, 8);
        t += __shfl_xor_sync(0xffffffffu, t, 16);
        if (lane < C16_ROWS) q[seg * rs + s * C16_ROWS + lane] = t;
    }
}

// row sum of the tile's row k (its slice's pieces in order)
template <class T>
__device__ __forceinline__ T c16_rowsum(const T* q, uint32_t rs, const unsigned char* sseg, uint32_t k) {
    const uint32_t n = sseg[k / C16_ROWS];
    T t = 0;
    for (uint32_t g = 0; g < n; g++) t += q[g * rs + k];
    return t;
}

// vec[c] = op(column c's number) for the tile's columns, four at a time so
// that op's loads overlap
template <class T, class OP>
__device__ __forceinline__ void c16_stage(T* vec, const uint32_t* cl, uint32_t ncol, OP op) {
    const uint32_t nthr = blockDim.x;
    for (uint32_t c = threadIdx.x; c < ncol; c += 4 * nthr) {
        uint32_t j[4];
#pragma unroll
        for (int u = 0; u < 4; u++) j[u] = cl[min(c + u * nthr, ncol - 1)];
        T v[4];
        op(j, v);
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (c + u * nthr < ncol) vec[c + u * nthr] = v[u];
    }
}

// A block's shared memory for tiles of at most ncol columns and rows rows in
// nseg pieces a slice: the staged vector (at 0; doubles in the FP64 pass),
// the row sums, the tile's slice offsets, the inbox read by the grid sums,
// and, in a block of one tile
// (single), its column list and its rows' state, which then never leave the
// SM.  The rest holds chunks of the matrix.
// The solve of the scene a tile belongs to (a batch; every tile has a copy).
struct C16Scene {
    double alpha, beta, gamma, stop, relres;
    int total, outers, it, phase;
    uint32_t flip;  // which of the published buffers is read
    uint32_t pad;
};

struct C16Plan {
    uint32_t q, soff, sseg, got, views, scn, cl, row, res;  // byte offsets
    uint32_t rs;                           // row stride of the sums and the state
};
constexpr uint32_t C16_ROW_BYTES = 32;     // x in double; r, w, s, 1 / diagonal, p, diagonal

__device__ __forceinline__ C16Plan c16_plan(uint32_t ncol, uint32_t rows, uint32_t nseg, uint32_t ntiles, bool single,
                                            bool batch) {
    C16Plan p;
    const uint32_t ns = (rows + C16_ROWS - 1) / C16_ROWS;
    p.rs = ns * C16_ROWS;
    p.q = c16_align(max(ncol, 1u) * 8u);
    p.soff = p.q + c16_align(p.rs * nseg * 8u);
    p.sseg = p.soff + c16_align((ns + 1) * 4u);
    p.got = p.sseg + c16_align(ns);
    p.views = p.got + c16_align(gridDim.x * C16_SUMS * 8u);
    p.scn = p.views + c16_align(single ? 0u : ntiles * (uint32_t)sizeof(C16View));
    p.cl = p.scn + c16_align(batch ? ntiles * (uint32_t)sizeof(C16Scene) : 0u);
    p.row = p.cl + (single ? c16_align(ncol * 4u) : 0u);
    p.res = c16_align(p.row + (single ? p.rs * C16_ROW_BYTES : 0u));
    return p;
}

// [p, p + bytes) towards L2, spread over the block
__device__ __forceinline__ void c16_ahead(const void* p, uint32_t bytes) {
    const unsigned char* a = reinterpret_cast<const unsigned char*>(p);
    for (uint32_t x = threadIdx.x * 128u; x < bytes; x += blockDim.x * 128u)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a + x));
}

// One block of a solver: its tiles, its shared memory and, when it has one
// tile, that tile's view.  Rows' state is in shared memory (single) or in
// the global arrays.
struct C16Block {
    const C16Args& S;
    unsigned char* sm;
    uint32_t R, C, G, ntiles;
    bool single, whole;
    bool sp_res;       // S' of the block's rows is in shared memory
    uint32_t sp_at, sp_words;  // its diagonal and first four of each 32 rows, and its entries
    C16Plan pl;
    C16View v;

    __device__ __forceinline__ C16Block(const C16Args& S_, unsigned char* sm_, bool learned) : S(S_), sm(sm_) {
        R = *S.nrows;
        G = gridDim.x;
        ntiles = c16_tiles(R, G, S.ns) / G;
        C = max(__ldg(S.off + (R + C16_ROWS - 1) / C16_ROWS), 1u);
        v = c16_view(S, blockIdx.x + G * (ntiles - 1), R, C, blockDim.x >> 5, S.keep);
        single = false;
        whole = false;
        if (ntiles == 1) {
            pl = c16_plan(v.ncol, v.rows, v.nseg, 1u, true, S.ns != 0u);
            single = pl.res <= S.smem_bytes && !C16_WHOLE;
        }
        if (!single) {
            // a tile with so many rows and columns that the pieces do not fit
            // is done by one warp, slices whole: slow, but right
            pl = c16_plan(__ldg(S.stats + 1), __ldg(S.stats + 2), C16_SEGS, ntiles, false, S.ns != 0u);
            whole = pl.res > S.smem_bytes || C16_WHOLE;
            if (whole) pl = c16_plan(__ldg(S.stats + 1), __ldg(S.stats + 2), 1u, ntiles, false, S.ns != 0u);
        }
        if (whole) v.cpw = max(v.nch, 1u);
        sp_res = false;
        if (learned && single) resident_sp();
        // the end of every warp's share of the last tile stays in shared memory
        const uint32_t nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        v.resw = min((S.smem_bytes - pl.res) / C16_CHUNK_BYTES, S.smem_chunks) / nw;
        v.resw = min(v.resw, v.cpw);
        {
            const uint32_t x0 = min(warp * v.cpw, v.nch), x1 = min(x0 + v.cpw, v.nch), n = min(v.resw, x1 - x0);
            const uint4* src = reinterpret_cast<const uint4*>(S.ent + (size_t)(v.c0 + x1 - n) * C16_CHUNK_BYTES);
            uint4* dst = reinterpret_cast<uint4*>(sm + pl.res + (size_t)warp * v.resw * C16_CHUNK_BYTES);
            for (uint32_t x = lane; x < n * (C16_CHUNK_BYTES / 16); x += 32) dst[x] = __ldg(src + x);
        }
        if (!single) {
            // half the L2 budget less the rows' vectors (48 bytes a row) and
            // S', which are read again every iteration too: with all of it
            // 293,971 rows take 4.19 (learned 4.49) ms a solve, so 4.08 (4.23)
            uint32_t keep = S.keep;
            if (keep != 0xffffffffu) {
                const uint64_t other = (uint64_t)R * 48u + (learned ? (uint64_t)__ldg(S.stats + 3) * 16u : 0u);
                const uint32_t n = (uint32_t)min(other / C16_CHUNK_BYTES, (uint64_t)0x7fffffffu);
                keep = keep / 2u > n ? keep / 2u - n : 0u;
            }
            C16View* views = reinterpret_cast<C16View*>(sm + pl.views);
            for (uint32_t m = threadIdx.x; m < ntiles; m += blockDim.x) {
                C16View t = c16_view(S, blockIdx.x + G * m, R, C, nw, keep);
                if (whole) t.cpw = max(t.nch, 1u);
                if (m == ntiles - 1) t.resw = v.resw;
                views[m] = t;
            }
        }
        if (single) {
            c16_slices(S, v, soff(), sseg());
            uint32_t* cl = reinterpret_cast<uint32_t*>(sm + pl.cl);
            for (uint32_t c = threadIdx.x; c < v.ncol; c += blockDim.x) cl[c] = __ldg(v.cl + c);
            v.cl = cl;
            for (uint32_t k = threadIdx.x; k < v.rows; k += blockDim.x) {
                rx()[k] = S.x64[v.r0 + k];
                rf(C16_INV)[k] = S.inv_diag[v.r0 + k];
                rf(C16_DG)[k] = S.diag32[v.r0 + k];
            }
        }
        __syncthreads();
    }
    // S' of the rows into shared memory, 32-row interleaved, when it fits: it
    // is read once an iteration by one thread a row, and the wait for those
    // few loads cost more than the chunks it displaces
    __device__ __forceinline__ void resident_sp() {
        const uint32_t nsp = (v.rows + SP_SLICE - 1) / SP_SLICE;
        const uint32_t f0 = __ldg(v.spf), n = __ldg(v.spf + nsp) - f0;
        const uint32_t head = c16_align(pl.res + (nsp * (SP_SLICE + 1) + 1) * 4u);
        if (head + n * 16u > S.smem_bytes) return;
        float* diag = reinterpret_cast<float*>(sm + pl.res);
        uint32_t* first = reinterpret_cast<uint32_t*>(diag + nsp * SP_SLICE);
        for (uint32_t j = threadIdx.x; j <= nsp; j += blockDim.x) first[j] = __ldg(v.spf + j) - f0;
        for (uint32_t k = threadIdx.x; k < v.rows; k += blockDim.x) diag[k] = __ldg(S.sp_diag + v.r0 + k);
        const uint4* src = reinterpret_cast<const uint4*>(S.sp_ent) + f0;
        uint4* w = reinterpret_cast<uint4*>(sm + head);
        for (uint32_t x = threadIdx.x; x < n; x += blockDim.x) w[x] = __ldg(src + x);
        sp_res = true;
        sp_at = pl.res;
        sp_words = head;
        pl.res = head + n * 16u;
    }
    __device__ __forceinline__ uint32_t* soff() const { return reinterpret_cast<uint32_t*>(sm + pl.soff); }
    __device__ __forceinline__ unsigned char* sseg() const { return sm + pl.sseg; }
    __device__ __forceinline__ double* got() const { return reinterpret_cast<double*>(sm + pl.got); }
    __device__ __forceinline__ double* rx() const { return reinterpret_cast<double*>(sm + pl.row); }
    __device__ __forceinline__ float* rf(uint32_t f) const {
        return reinterpret_cast<float*>(sm + pl.row + pl.rs * 8u) + f * pl.rs;
    }
    enum : uint32_t { C16_R = 0, C16_W, C16_S, C16_INV, C16_P, C16_DG };

    // body(view) for each of the block's tiles; the slice offsets are loaded
    // (the body's first barrier publishes them).  While a tile is worked on,
    // ahead(view) brings what the next one reads once into L2.
    template <class P, class F, class W>
    __device__ __forceinline__ void tiles(P ahead, F body, W want) const {
        const C16View* views = reinterpret_cast<const C16View*>(sm + pl.views);
        for (uint32_t m = 0; m < ntiles; m++) {
            if (m + 1 < ntiles && want(m + 1)) {
                const C16View& n = views[m + 1];
                c16_ahead(n.cl, n.ncol * 4u);
                c16_ahead(S.off + n.s0, (n.ns + 1) * 4u);
                ahead(n);
            }
            if (!want(m)) continue;
            C16View t = v;
            if (!single) {
                t = views[m];
                __syncthreads();
                c16_slices(S, t, soff(), sseg());
            }
            body(t);  // the only call: the compiler inlines it
        }
    }
    template <class P, class F>
    __device__ __forceinline__ void tiles(P ahead, F body) const {
        tiles(ahead, body, [](uint32_t) { return true; });
    }
    __device__ __forceinline__ const C16View& view(uint32_t m) const {
        return single ? v : reinterpret_cast<const C16View*>(sm + pl.views)[m];
    }
    // the tile's products over the staged vector, barriers included; row k's
    // sum is then rowsum<T>(k)
    template <class T, class REMOTE>
    __device__ __forceinline__ void product(const C16View& t, REMOTE remote) const {
        __syncthreads();
        T* q = reinterpret_cast<T*>(sm + pl.q);
        if (t.esc) c16_product<T, true>(S, t, sm, soff(), q, pl.rs, sm + pl.res, remote);
        else c16_product<T, false>(S, t, sm, soff(), q, pl.rs, sm + pl.res, remote);
        __syncthreads();
    }
    template <class T>
    __device__ __forceinline__ T rowsum(uint32_t k) const {
        return c16_rowsum(reinterpret_cast<const T*>(sm + pl.q), pl.rs, sseg(), k);
    }
    // r64 = b - A x64 of the tile's rows in FP64, |r64|^2 and |b|^2;
    // body(k, r64)
    template <class F>
    __device__ __forceinline__ void residual(const C16View& t, double (&acc)[C16_SUMS], F body) const {
        c16_stage(reinterpret_cast<double*>(sm), t.cl, t.ncol, [&](const uint32_t (&j)[4], double (&o)[4]) {
#pragma unroll
            for (int u = 0; u < 4; u++) o[u] = __ldcg(S.x64 + j[u]);
        });
        product<double>(t, [&](uint32_t col) { return __ldcg(S.x64 + col); });
        for (uint32_t k = threadIdx.x; k < t.rows; k += blockDim.x) {
            const uint32_t g = t.r0 + k;
            const double bi = __ldg(S.b64 + g);
            const double x = reinterpret_cast<const double*>(sm)[k];
            const double ri = bi - (__ldg(S.diag64 + g) * x + rowsum<double>(k));
            acc[0] += ri * ri;
            acc[1] += bi * bi;
            body(k, ri);
        }
    }
    // what that reads of a tile once
    __device__ __forceinline__ void ahead_residual(const C16View& n) const {
        c16_ahead(S.b64 + n.r0, n.rows * 8u);
        c16_ahead(S.diag64 + n.r0, n.rows * 8u);
    }
};

// the reduction one FP32 inner solve is asked for, squared
__device__ __forceinline__ double inner_target(const C16Args& S, double relres) {
    double eta = 0.3 * S.tol / relres;
    if (eta < S.eta_min) eta = S.eta_min;
    if (eta > 0.5) eta = 0.5;
    return eta * eta;
}

// ---- a tile's part of an iteration with diagonal scaling
// CG in the single-reduction form of Chronopoulos and Gear (1989): with u =
// D^-1 r and w = A u, one sum of (r.u, w.u, r.r) gives the next alpha and
// beta, and s = w + beta s, p = u + beta p follow by recurrence.  A row
// publishes (r, w, s, 1 / diagonal); whoever needs its next u forms it from
// those while staging (16 bytes per staged column, not per entry), so an
// iteration has one grid-wide wait.  The same iterates as CG's in exact
// arithmetic; the FP64 true residual ends the solve.  pc is read, pn written.
__device__ __forceinline__ void c16_start_row(const C16Args& S, const C16Block& B, const C16View& t, uint32_t k,
                                              double ri, float4* pc) {
    const float r = (float)ri;
    if (B.single) {
        B.rf(C16Block::C16_R)[k] = r;
        B.rf(C16Block::C16_W)[k] = 0.f;
        B.rf(C16Block::C16_S)[k] = 0.f;
        B.rf(C16Block::C16_P)[k] = 0.f;
        pc[t.r0 + k] = make_float4(r, 0.f, 0.f, B.rf(C16Block::C16_INV)[k]);
    } else {
        S.p[t.r0 + k] = 0.f;
        pc[t.r0 + k] = make_float4(r, 0.f, 0.f, __ldg(S.inv_diag + t.r0 + k));
    }
}

__device__ __forceinline__ void c16_iterate(const C16Args& S, const C16Block& B, const C16View& t, double alpha,
                                            double beta, const float4* pc, float4* pn, double (&g)[C16_SUMS]) {
    float* vec = reinterpret_cast<float*>(B.sm);
    const float af = (float)alpha, bf = (float)beta;
    auto next_u = [&](const float4& v) { return v.w * fmaf(-af, fmaf(bf, v.z, v.y), v.x); };
    c16_stage(vec, t.cl, t.ncol, [&](const uint32_t (&j)[4], float (&o)[4]) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = __ldcg(pc + j[u]);
#pragma unroll
        for (int u = 0; u < 4; u++) o[u] = next_u(v[u]);
    });
    B.product<float>(t, [&](uint32_t col) { return next_u(__ldcg(pc + col)); });
    for (uint32_t k = threadIdx.x; k < t.rows; k += blockDim.x) {
        const uint32_t gk = t.r0 + k;
        float4 o;
        float p, dg;
        double x;
        if (B.single) {
            o = make_float4(B.rf(C16Block::C16_R)[k], B.rf(C16Block::C16_W)[k], B.rf(C16Block::C16_S)[k],
                            B.rf(C16Block::C16_INV)[k]);
            p = B.rf(C16Block::C16_P)[k];
            dg = B.rf(C16Block::C16_DG)[k];
            x = B.rx()[k];
        } else {
            o = pc[gk];
            p = S.p[gk];
            dg = __ldg(S.diag32 + gk);
            x = S.x64[gk];
        }
        const float sn = fmaf(bf, o.z, o.y);
        p = fmaf(bf, p, o.w * o.x);
        x += alpha * (double)p;
        const float r = fmaf(-af, sn, o.x);
        const float u = vec[k];
        const float w = fmaf(dg, u, B.rowsum<float>(k));
        pn[gk] = make_float4(r, w, sn, o.w);
        S.x64[gk] = x;
        if (B.single) {
            B.rf(C16Block::C16_R)[k] = r;
            B.rf(C16Block::C16_W)[k] = w;
            B.rf(C16Block::C16_S)[k] = sn;
            B.rf(C16Block::C16_P)[k] = p;
            B.rx()[k] = x;
        } else {
            S.p[gk] = p;
        }
        g[0] += (double)r * (double)u;
        g[1] += (double)w * (double)u;
        g[2] += (double)r * (double)r;
    }
}

__device__ __forceinline__ void c16_ahead_iterate(const C16Args& S, const C16View& n) {
    c16_ahead(S.x64 + n.r0, n.rows * 8u);
    c16_ahead(S.p + n.r0, n.rows * 4u);
    c16_ahead(S.diag32 + n.r0, n.rows * 4u);
}

// ---- and with the learned preconditioner z = S' r
// Row k of S' x over the staged x (own rows first in the tile's list); an
// escaped column's x comes from remote.  S' is in shared memory or read
// again every iteration.
template <class REMOTE>
__device__ __forceinline__ float c16_sp_row(const C16Args& S, const C16Block& B, const C16View& t, const float* vec,
                                            uint32_t k, REMOTE remote) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    auto add = [&](uint32_t e, size_t at, float& a) {
        const uint32_t c = e >> 16;
        float x;
        if (t.esc && c == C16_ESC) x = remote(__ldg(S.sp_side + at));
        else x = vec[c >> 2];
        a = fmaf(__uint_as_float(e << 16), x, a);
    };
    auto four = [&](const uint4& e, uint32_t f, float& a0, float& a1, float& a2, float& a3) {  // four f of the array
        add(e.x, 4 * (size_t)f, a0);
        add(e.y, 4 * (size_t)f + 1, a1);
        add(e.z, 4 * (size_t)f + 2, a2);
        add(e.w, 4 * (size_t)f + 3, a3);
    };
    float dg;
    if (B.sp_res) {
        const float* diag = reinterpret_cast<const float*>(B.sm + B.sp_at);
        const uint32_t nsp = (t.rows + SP_SLICE - 1) / SP_SLICE;
        const uint32_t* first = reinterpret_cast<const uint32_t*>(diag + nsp * SP_SLICE) + k / SP_SLICE;
        const uint32_t a = first[0] + k % SP_SLICE, b = first[1];
        const uint4* w = reinterpret_cast<const uint4*>(B.sm + B.sp_words);
        dg = diag[k];
        uint32_t f = a;
        for (; f + SP_SLICE < b; f += 2 * SP_SLICE) {
            four(w[f], __ldg(t.spf) + f, acc[0], acc[1], acc[2], acc[3]);
            four(w[f + SP_SLICE], __ldg(t.spf) + f + SP_SLICE, acc[4], acc[5], acc[6], acc[7]);
        }
        if (f < b) four(w[f], __ldg(t.spf) + f, acc[0], acc[1], acc[2], acc[3]);
    } else {
        constexpr int UN = 8;  // fours in flight: a whole row mostly
        const uint32_t a = __ldg(t.spf + k / SP_SLICE) + k % SP_SLICE, b = __ldg(t.spf + k / SP_SLICE + 1);
        dg = __ldg(S.sp_diag + t.r0 + k);
        const uint4* w = reinterpret_cast<const uint4*>(S.sp_ent);
        for (uint32_t f = a; f < b; f += UN * SP_SLICE) {
            uint4 e[UN];
#pragma unroll
            for (int u = 0; u < UN; u++) e[u] = __ldg(w + (f + u * SP_SLICE < b ? f + u * SP_SLICE : f));
#pragma unroll
            for (int u = 0; u < UN; u++)
                if (f + u * SP_SLICE < b) four(e[u], f + u * SP_SLICE, acc[4 * (u & 1)], acc[4 * (u & 1) + 1], acc[4 * (u & 1) + 2],
                                               acc[4 * (u & 1) + 3]);
        }
    }
    const float offd = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]));
    return fmaf(dg, vec[k], offd);
}

// An iteration is two passes, each ending in a grid-wide sum: the update
// (residuals r - alpha q staged, x, z = S' r, r.z and r.r) and the product
// (directions z + beta p staged, q = A p, p.q).  A row publishes (z, p) in
// the first and (r, q) in the second, each read by the other blocks only in
// the other pass.
__device__ __forceinline__ void c16_update(const C16Args& S, const C16Block& B, const C16View& t, double alpha,
                                           float2* zp, const float2* rq, double (&g)[C16_SUMS]) {
    float* vec = reinterpret_cast<float*>(B.sm);
    const float af = (float)alpha;
    auto next_r = [&](const float2& v) { return fmaf(-af, v.y, v.x); };
    c16_stage(vec, t.cl, t.ncol, [&](const uint32_t (&j)[4], float (&o)[4]) {
        float2 v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = __ldcg(rq + j[u]);
#pragma unroll
        for (int u = 0; u < 4; u++) o[u] = next_r(v[u]);
    });
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < t.rows; k += blockDim.x) {
        const uint32_t gk = t.r0 + k;
        const float r = vec[k];
        const float p = B.single ? B.rf(C16Block::C16_P)[k] : S.p[gk];
        const double x = (B.single ? B.rx()[k] : S.x64[gk]) + alpha * (double)p;
        const float z = c16_sp_row(S, B, t, vec, k, [&](uint32_t col) { return next_r(__ldcg(rq + col)); });
        zp[gk] = make_float2(z, p);
        S.x64[gk] = x;
        if (B.single) {
            B.rx()[k] = x;
            B.rf(C16Block::C16_R)[k] = r;
        } else {
            S.r[gk] = r;
        }
        g[0] += (double)r * (double)z;
        g[1] += (double)r * (double)r;
    }
}

__device__ __forceinline__ void c16_ahead_update(const C16Args& S, const C16View& n) {
    const uint32_t nsp = (n.rows + SP_SLICE - 1) / SP_SLICE;
    const uint32_t f = __ldg(n.spf);
    c16_ahead(S.sp_ent + 4 * (size_t)f, (__ldg(n.spf + nsp) - f) * 16u);
    c16_ahead(n.spf, (nsp + 1) * 4u);
    c16_ahead(S.sp_diag + n.r0, n.rows * 4u);
    c16_ahead(S.x64 + n.r0, n.rows * 8u);
    c16_ahead(S.p + n.r0, n.rows * 4u);
}

__device__ __forceinline__ void c16_direction(const C16Args& S, const C16Block& B, const C16View& t, float beta,
                                              const float2* zp, float2* rq, double& pq) {
    float* vec = reinterpret_cast<float*>(B.sm);
    auto next_p = [&](const float2& v) { return fmaf(beta, v.y, v.x); };
    c16_stage(vec, t.cl, t.ncol, [&](const uint32_t (&j)[4], float (&o)[4]) {
        float2 v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = __ldcg(zp + j[u]);
#pragma unroll
        for (int u = 0; u < 4; u++) o[u] = next_p(v[u]);
    });
    B.product<float>(t, [&](uint32_t col) { return next_p(__ldcg(zp + col)); });
    for (uint32_t k = threadIdx.x; k < t.rows; k += blockDim.x) {
        const uint32_t gk = t.r0 + k;
        const float p = vec[k];
        const float dg = B.single ? B.rf(C16Block::C16_DG)[k] : __ldg(S.diag32 + gk);
        const float q = fmaf(dg, p, B.rowsum<float>(k));
        if (B.single) B.rf(C16Block::C16_P)[k] = p;
        else S.p[gk] = p;
        rq[gk] = make_float2(B.single ? B.rf(C16Block::C16_R)[k] : S.r[gk], q);
        pq += (double)p * (double)q;
    }
}

__device__ __forceinline__ void c16_ahead_direction(const C16Args& S, const C16View& n) {
    c16_ahead(S.diag32 + n.r0, n.rows * 4u);
    c16_ahead(S.r + n.r0, n.rows * 4u);
}

// the start of an inner solve from r64: r published, p = 0
__device__ __forceinline__ void c16_start_row_learned(const C16Args& S, const C16Block& B, const C16View& t,
                                                      uint32_t k, double ri, float2* rq) {
    rq[t.r0 + k] = make_float2((float)ri, 0.f);
    if (B.single) B.rf(C16Block::C16_P)[k] = 0.f;
    else S.p[t.r0 + k] = 0.f;
}

// ---- one scene
// ok: every grid sum completed (else the timeout is the error)
__device__ __forceinline__ void c16_finish_solve(const C16Args& S, const C16Sync& sy, int total, int outers,
                                                 double relres, bool converged, bool ok) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    *S.epoch = sy.epoch + 2;  // past every epoch any block has used
    if (!ok) return;
    S.sc->cg_iters = total;
    S.sc->cg_outer = outers;
    S.sc->cg_relres = relres;
    if (!converged) atomicOr(&S.sc->err, ERR_CG_NOT_CONVERGED);
}

template <bool LRN>
__global__ void __launch_bounds__(C16_THREADS, 1) k_ppe_solve_c16(C16Args S) {
    extern __shared__ __align__(16) unsigned char c16_sm[];
    C16Sync sy{S.slots, *S.epoch, S.sc};
    const C16Block B(S, c16_sm, LRN);
    float4* pc = S.pub0;  // published rows: read by this iteration
    float4* pn = S.pub1;  // and written
    float2* zp = reinterpret_cast<float2*>(S.pub0);
    float2* rq = reinterpret_cast<float2*>(S.pub1);
    int total = 0, outers = 0;
    double relres = 0.0;
    bool converged = false, ok = true;
    for (int outer = 0; outer < S.max_outer; outer++) {
        double acc[C16_SUMS] = {0.0, 0.0, 0.0};
        B.tiles([&](const C16View& n) { B.ahead_residual(n); },
                [&](const C16View& t) {
                    B.residual(t, acc, [&](uint32_t k, double ri) {
                        if (LRN) c16_start_row_learned(S, B, t, k, ri, rq);
                        else c16_start_row(S, B, t, k, ri, pc);
                    });
                });
        const double two[2] = {acc[0], acc[1]};
        double tot[2];
        ok = c16_sum<2>(two, sy, B.got(), tot);
        if (!ok) break;
        outers++;
        relres = tot[1] > 0.0 ? sqrt(tot[0] / tot[1]) : 0.0;
        if (relres <= S.tol) {
            converged = true;
            break;
        }
        if (total >= S.max_iter) break;
        const double stop = inner_target(S, relres) * tot[0];
        double alpha = 0.0, beta = 0.0, gamma = 0.0;
        // it = -1: w = A u, or z = S' r, of the start; nothing moves (alpha = beta = 0)
        for (int it = -1;; it++) {
            double g[C16_SUMS] = {0.0, 0.0, 0.0};
            if (LRN) {
                B.tiles([&](const C16View& n) { c16_ahead_update(S, n); },
                        [&](const C16View& t) { c16_update(S, B, t, alpha, zp, rq, g); });
                const double v2[2] = {g[0], g[1]};
                double gt[2];
                ok = c16_sum<2>(v2, sy, B.got(), gt);
                if (!ok) break;
                beta = 0.0;
                if (it >= 0) {
                    total++;
                    if (gt[1] <= stop) break;
                    beta = gt[0] / gamma;
                }
                gamma = gt[0];
                if (it + 1 >= S.inner_cap || total >= S.max_iter) break;
                double pq[1] = {0.0}, tp[1];
                B.tiles([&](const C16View& n) { c16_ahead_direction(S, n); },
                        [&](const C16View& t) { c16_direction(S, B, t, (float)beta, zp, rq, pq[0]); });
                ok = c16_sum<1>(pq, sy, B.got(), tp);
                if (!ok) break;
                alpha = gamma / tp[0];
            } else {
                B.tiles([&](const C16View& n) { c16_ahead_iterate(S, n); },
                        [&](const C16View& t) { c16_iterate(S, B, t, alpha, beta, pc, pn, g); });
                double gt[C16_SUMS];
                ok = c16_sum<C16_SUMS>(g, sy, B.got(), gt);
                if (!ok) break;
                float4* x = pc;
                pc = pn;
                pn = x;
                if (it >= 0) {
                    total++;
                    if (gt[2] <= stop) break;
                    beta = gt[0] / gamma;
                    alpha = gt[0] / (gt[1] - beta * gt[0] / alpha);
                } else {
                    alpha = gt[0] / gt[1];
                }
                gamma = gt[0];
                if (it + 1 >= S.inner_cap || total >= S.max_iter) break;
            }
        }
        if (!ok) break;
    }
    c16_finish_solve(S, sy, total, outers, relres, converged, ok);
}

// ---- the scenes of a batch
// Every scene runs its own solve, with its own FP64 passes and stop, and its
// tiles are spread over the blocks.  In a round every tile does what its
// scene is at (the FP64 residual, the start, an iteration; with the learned
// form an update or a product) and leaves its sums; after one grid-wide
// barrier every block adds up the sums of its tiles' scenes, in tile order,
// and moves them on.  A scene that is done is skipped; the barrier's own sum
// counts the scenes that are not.
enum : int { SCN_RESID = 0, SCN_START, SCN_ITER, SCN_PROD, SCN_DONE };

// the block's sum of g to out[0 .. C16_SUMS)
__device__ __forceinline__ void c16_tile_sum(const double (&g)[C16_SUMS], double* out) {
    __shared__ double part[C16_SUMS][32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < (int)C16_SUMS; k++) {
        const double t = warp_sum_d(g[k]);
        if (lane == 0) part[k][warp] = t;
    }
    __syncthreads();
    if (warp < C16_SUMS) {
        const double t = warp_sum_d(lane < nw ? part[warp][lane] : 0.0);
        if (lane == 0) out[warp] = t;
    }
}

// a scene's next step from the sums of its last one (g); true when it ends
template <bool LRN>
__device__ __forceinline__ void c16_advance(const C16Args& S, C16Scene& c, const double (&g)[C16_SUMS], bool* failed) {
    switch (c.phase) {
        case SCN_RESID:
            c.outers++;
            c.relres = g[1] > 0.0 ? sqrt(g[0] / g[1]) : 0.0;
            if (c.relres <= S.tol) {
                c.phase = SCN_DONE;
            } else if (c.total >= S.max_iter || c.outers >= S.max_outer) {
                c.phase = SCN_DONE;
                *failed = true;
            } else {
                c.stop = inner_target(S, c.relres) * g[0];
                c.alpha = c.beta = c.gamma = 0.0;
                c.it = -1;
                c.phase = SCN_START;
            }
            return;
        case SCN_PROD:
            c.alpha = c.gamma / g[0];
            c.it++;
            c.phase = SCN_ITER;
            return;
        default: break;
    }
    const bool started = c.phase == SCN_ITER;
    if (started) c.total++;
    if (LRN) {
        if (started && g[1] <= c.stop) {
            c.phase = SCN_RESID;
            return;
        }
        c.beta = started ? g[0] / c.gamma : 0.0;
        c.gamma = g[0];
        c.phase = c.it + 1 >= S.inner_cap || c.total >= S.max_iter ? SCN_RESID : SCN_PROD;
    } else {
        c.flip ^= 1u;
        if (started && g[2] <= c.stop) {
            c.phase = SCN_RESID;
            return;
        }
        if (started) {
            c.beta = g[0] / c.gamma;
            c.alpha = g[0] / (g[1] - c.beta * g[0] / c.alpha);
        } else {
            c.alpha = g[0] / g[1];
        }
        c.gamma = g[0];
        c.phase = c.it + 1 >= S.inner_cap || c.total >= S.max_iter ? SCN_RESID : SCN_ITER;
        c.it++;
    }
}

template <bool LRN>
__global__ void __launch_bounds__(C16_THREADS, 1) k_ppe_solve_c16_batch(C16Args S) {
    extern __shared__ __align__(16) unsigned char c16_sm[];
    C16Sync sy{S.slots, *S.epoch, S.sc};
    const C16Block B(S, c16_sm, LRN);
    C16Scene* scn = reinterpret_cast<C16Scene*>(c16_sm + B.pl.scn);
    __shared__ int open_s;  // scenes not done whose first tile is this block's
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t T = B.ntiles * B.G;
    for (uint32_t m = threadIdx.x; m < B.ntiles; m += blockDim.x) {
        C16Scene c;
        c.alpha = c.beta = c.gamma = c.stop = c.relres = 0.0;
        c.total = c.outers = 0;
        c.it = -1;
        c.phase = SCN_RESID;
        c.flip = 0;
        scn[m] = c;
    }
    auto own = [&](uint32_t m) { return __ldg(S.tb + B.view(m).scene) == B.view(m).tile; };
    auto count_open = [&] {  // thread 0
        int n = 0;
        for (uint32_t m = 0; m < B.ntiles; m++) n += scn[m].phase != SCN_DONE && own(m) ? 1 : 0;
        open_s = n;
    };
    __syncthreads();
    if (threadIdx.x == 0) count_open();
    __syncthreads();
    float2* zp = reinterpret_cast<float2*>(S.pub0);
    float2* rq = reinterpret_cast<float2*>(S.pub1);
    bool ok;
    for (uint32_t round = 0;; round++) {
        double* ts = S.tsum + (size_t)(round & 1u) * T * C16_SUMS;
        auto index = [&](const C16View& t) { return (t.tile - blockIdx.x) / B.G; };
        B.tiles(
            [&](const C16View& n) {
                const int ph = scn[index(n)].phase;
                if (ph == SCN_RESID) B.ahead_residual(n);
                else if (!LRN) c16_ahead_iterate(S, n);
                else if (ph == SCN_PROD) c16_ahead_direction(S, n);
                else c16_ahead_update(S, n);
            },
            [&](const C16View& t) {
                const C16Scene& c = scn[index(t)];
                double g[C16_SUMS] = {0.0, 0.0, 0.0};
                if (c.phase == SCN_RESID) {
                    float4* pc = c.flip ? S.pub1 : S.pub0;
                    B.residual(t, g, [&](uint32_t k, double ri) {
                        if (LRN) c16_start_row_learned(S, B, t, k, ri, rq);
                        else c16_start_row(S, B, t, k, ri, pc);
                    });
                } else if (!LRN) {
                    c16_iterate(S, B, t, c.alpha, c.beta, c.flip ? S.pub1 : S.pub0, c.flip ? S.pub0 : S.pub1, g);
                } else if (c.phase == SCN_PROD) {
                    c16_direction(S, B, t, (float)c.beta, zp, rq, g[0]);
                } else {
                    c16_update(S, B, t, c.alpha, zp, rq, g);
                }
                c16_tile_sum(g, ts + (size_t)t.tile * C16_SUMS);
            },
            [&](uint32_t m) { return scn[m].phase != SCN_DONE; });
        const double open[1] = {threadIdx.x == 0 ? (double)open_s : 0.0};
        double left[1];
        ok = c16_sum<1>(open, sy, B.got(), left);
        if (!ok || left[0] == 0.0) break;
        // a scene's sums once for its consecutive tiles here; the others copy
        auto leads = [&](uint32_t m) { return m == 0 || B.view(m - 1).scene != B.view(m).scene; };
        for (uint32_t m = warp; m < B.ntiles; m += nw) {
            if (scn[m].phase == SCN_DONE || !leads(m)) continue;
            const uint32_t s = B.view(m).scene, t0 = __ldg(S.tb + s), t1 = __ldg(S.tb + s + 1);
            double g[C16_SUMS] = {0.0, 0.0, 0.0};
            for (uint32_t t = t0 + lane; t < t1; t += 32)
#pragma unroll
                for (int k = 0; k < (int)C16_SUMS; k++) g[k] += __ldcg(ts + (size_t)t * C16_SUMS + k);
#pragma unroll
            for (int k = 0; k < (int)C16_SUMS; k++) g[k] = warp_sum_d(g[k]);
            if (lane == 0) {
                bool failed = false;
                c16_advance<LRN>(S, scn[m], g, &failed);
                if (failed) atomicOr(&S.sc->err, ERR_CG_NOT_CONVERGED);
            }
        }
        __syncthreads();
        for (uint32_t m = threadIdx.x; m < B.ntiles; m += blockDim.x) {
            uint32_t l = m;
            while (!leads(l)) l--;
            if (l != m) scn[m] = scn[l];
        }
        __syncthreads();
        if (threadIdx.x == 0) count_open();
        for (uint32_t m = threadIdx.x; m < B.ntiles; m += blockDim.x)
            if (own(m)) {
                const uint32_t s = B.view(m).scene;
                S.iters[s] = scn[m].total;
                S.outers[s] = scn[m].outers;
                S.srel[s] = scn[m].relres;
            }
        __syncthreads();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *S.epoch = sy.epoch + 2;
        if (ok) {
            int mi = 0, mo = 0;
            double mr = 0.0;
            for (uint32_t s = 0; s < S.ns; s++) {
                mi = max(mi, __ldcg(S.iters + s));
                mo = max(mo, __ldcg(S.outers + s));
                mr = fmax(mr, __ldcg(S.srel + s));
            }
            S.sc->cg_iters = mi;
            S.sc->cg_outer = mo;
            S.sc->cg_relres = mr;
        }
    }
}

template <class T>
bool c16_alloc(T** p, size_t count) {
    return cudaMalloc((void**)p, (count ? count : 1) * sizeof(T)) == cudaSuccess;
}

// Several arrays in one allocation (each starts at 256 bytes): a cudaMalloc
// costs 0.1 ms and more, and a handle has some thirty of these arrays.
struct C16Arrays {
    size_t bytes = 0;
    std::vector<std::pair<void**, size_t>> at;
    template <class T>
    void add(T** p, size_t count) {
        at.push_back({(void**)p, bytes});
        bytes += (count * sizeof(T) + 255) / 256 * 256;
    }
    bool get(unsigned char** block) {
        if (!c16_alloc(block, bytes)) return false;
        for (const auto& a : at) *a.first = *block + a.second;
        return true;
    }
};

// The linked cells of a grid (the fast arithmetic's halved cells grouped)
struct C16Cells {
    uint32_t f, nx, ny, nz;  // cells of the sorted grid in one along y and z; linked cells
    C16Cells(const Grid& g)
        : f((uint32_t)g.reach), nx(g.cdx), ny((g.cdy + f - 1) / f), nz((g.cdz + f - 1) / f) {}
    uint64_t count() const { return (uint64_t)nx * ny * nz; }
};

// The cells of a box along the Hilbert curve of the cube around it.  The
// curve is the one of J. Skilling, "Programming the Hilbert curve" (AIP Conf.
// Proc. 707, 2004), unrolled from its top level down: in the curve's frame
// (axis a is the box's axis p[a], mirrored where f[a]) the octants come in
// Gray code order, backwards in cubes of odd parity; a set bit of axis a
// mirrors axis 0 of the octant's own frame, a clear one swaps axes 0 and a.
// Octants outside the box are passed over.  79,950 cells take 1.4 ms of host
// time; computing and sorting the cells' positions took 11.8.
struct C16Curve {
    uint32_t n[3];
    uint32_t* out;  // (z ny + y) nx + x of each cell
    void cube(const uint32_t (&at)[3], uint32_t edge, const uint32_t (&p0)[3], const uint32_t (&f0)[3], bool odd) {
        if (edge == 1) {
            *out++ = (at[2] * n[1] + at[1]) * n[0] + at[0];
            return;
        }
        for (uint32_t d = 0; d < 8; d++) {
            const uint32_t v = odd ? 7u - d : d;
            const uint32_t b[3] = {v >> 2, ((v >> 1) ^ (v >> 2)) & 1u, (v ^ (v >> 1)) & 1u};
            uint32_t o[3] = {at[0], at[1], at[2]}, p[3] = {p0[0], p0[1], p0[2]}, f[3] = {f0[0], f0[1], f0[2]};
            for (int a = 0; a < 3; a++) o[p[a]] += b[a] != f[a] ? edge / 2 : 0u;
            if (o[0] >= n[0] || o[1] >= n[1] || o[2] >= n[2]) continue;
            for (int a = 0; a < 3; a++) {
                if (b[a]) {
                    f[0] ^= 1u;
                } else {
                    std::swap(p[0], p[a]);
                    std::swap(f[0], f[a]);
                }
            }
            cube(o, edge / 2, p, f, odd != ((v & 1u) != 0u));
        }
    }
};

void curve_order(const C16Cells& c, uint32_t* out) {
    C16Curve w{{c.nx, c.ny, c.nz}, out};
    uint32_t edge = 2;
    while (edge < std::max(c.nx, std::max(c.ny, c.nz))) edge *= 2;
    w.cube({0, 0, 0}, edge, {0, 1, 2}, {0, 0, 0}, false);
}

// The place of every linked cell on the curve (first: the grid's first one).
__global__ void __launch_bounds__(256) k_c16_rank(const uint32_t* __restrict__ order, uint32_t n, uint32_t first,
                                                  uint32_t* __restrict__ rank) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) rank[order[k]] = first + k;
}

// A warp a linked cell: the 27 linked cells around it (C16_NONE: outside) and
// its up to 4 cells of the sorted grid (global ids).
__global__ void __launch_bounds__(256) k_c16_links(Grid g, C16Cells c, const uint32_t* __restrict__ order, uint32_t n,
                                                   const uint32_t* __restrict__ rank, uint32_t* __restrict__ cells,
                                                   uint32_t* __restrict__ nbr) {
    const uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (k >= n) return;
    const uint32_t lin = order[k], cx = lin % c.nx, cy = lin / c.nx % c.ny, cz = lin / c.nx / c.ny;
    if (lane < 27) {
        const uint32_t x = cx + lane % 3 - 1, y = cy + lane / 3 % 3 - 1, z = cz + lane / 9 - 1;  // below 0 wraps
        const bool in = x < c.nx && y < c.ny && z < c.nz;
        nbr[27 * (size_t)k + lane] = in ? rank[(z * c.ny + y) * c.nx + x] : C16_NONE;
    } else if (lane < 31) {
        const uint32_t a = (lane - 27) & 1u, b = (lane - 27) >> 1, y = cy * c.f + a, z = cz * c.f + b;
        const bool in = a < c.f && b < c.f && y < g.cdy && z < g.cdz;
        cells[4 * (size_t)k + lane - 27] = in ? g.base + z * g.sheet + y * g.cdx + cx : C16_NONE;
    }
}

// shared memory of the pack's page table and of a solver block (the rest of
// an SM's 228 KB stays L1 and the kernels' static arrays)
size_t c16_page_bytes(uint32_t cap) { return (((size_t)cap + C16_PAGE - 1) / C16_PAGE + 1) * sizeof(uint16_t); }
constexpr size_t C16_PAGE_BYTES_MAX = 160 * 1024;
constexpr size_t C16_SMEM = 220 * 1024;

}  // namespace

static bool c16_solver_smem() {
    for (const void* f : {(const void*)k_ppe_solve_c16<false>, (const void*)k_ppe_solve_c16<true>,
                          (const void*)k_ppe_solve_c16_batch<false>, (const void*)k_ppe_solve_c16_batch<true>})
        if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C16_SMEM) != cudaSuccess)
            return false;
    return true;
}

static uint64_t c16_cells(const Grid* grids, uint32_t ngrids) {
    uint64_t n = 0;
    for (uint32_t s = 0; s < ngrids; s++) n += C16Cells(grids[s]).count();
    return n;
}

// the pack's page table is in shared memory: 20 M particles; a warp a linked
// cell in 32-bit thread numbers
bool ppe_c16_takes(uint32_t cap, const Grid* grids, uint32_t ngrids) {
    for (uint32_t s = 0; s < ngrids; s++)
        if (grids[s].reach > 2) return false;
    return c16_cells(grids, ngrids) < (1u << 26) &&
           c16_page_bytes(ppe_rows_cap(cap, ngrids)) <= C16_PAGE_BYTES_MAX;
}

// The links of a linked cell take 132 bytes.  The tiles are the faster layout in
// nearly empty grids too (70,912 particles with one far away, ms a step over
// tiles and in the 8-byte layout: 2 cells a particle 0.52 and 0.78, 16 0.63 and
// 0.87, 64 0.99 and 1.16; with S' at 64 1.17 and 1.38), but past 64 cells a
// particle the links are more than both layouts' matrices.  A tank full of
// water has 0.02 cells a particle, one half full 0.04.
constexpr uint64_t C16_FEW_CELLS = 65536;
bool ppe_c16_prefers(uint32_t cap, const Grid* grids, uint32_t ngrids) {
    return ppe_c16_takes(cap, grids, ngrids) &&
           c16_cells(grids, ngrids) <= std::max<uint64_t>(64ull * cap, C16_FEW_CELLS);
}

// Whether the numbering lists the occupied cells first (k_c16_occupied): three
// launches more and a scan by many blocks, 16 us, where a warp for every cell
// costs 0.6 us a thousand: 27,700 particles in 19,683 cells 0.424 ms a step with
// and 0.42 without, in 59,319 0.428 and 0.437; of 70,913 in 287,496 0.54 and
// 0.68.  Not where most cells are full.
static bool c16_lists(const PpeWork& w) { return w.c16_nsuper > 32768u && w.c16_nsuper > w.cap / 8u; }

int ppe_c16_enable(PpeWork& w, const Grid* grids, uint32_t ngrids, const PpeWork* same, cudaStream_t st,
                   std::string* err) {
    if (w.c16_ready) return MPS_OK;
    const uint32_t ns = w.nscenes;
    if (!ppe_c16_takes(w.cap, grids, ngrids)) {
        if (err) *err = "the compact PPE layout does not take this grid";
        return MPS_ERR_INVALID;
    }
    const size_t cap = ppe_rows_cap(w.cap, ns);
    const size_t vec = cap + 8;
    const size_t slices = (cap + C16_ROWS - 1) / C16_ROWS + 2;
    const size_t chunks = slices * ((PPE_W + 15) / 16);
    const size_t tiles = c16_tiles((uint32_t)cap, (uint32_t)w.sms, ns);
    C16Arrays A;
    w.c16_shared = same && same->c16_ready;
    std::vector<uint32_t> sfirst(1, 0u);
    for (uint32_t s = 0; s < ngrids; s++) sfirst.push_back(sfirst.back() + (uint32_t)C16Cells(grids[s]).count());
    w.c16_nsuper = sfirst.back();
    if (w.c16_shared) {
        w.c16_cells = same->c16_cells;
        w.c16_nbr = same->c16_nbr;
    } else {
        A.add(&w.c16_cells, 5 * (size_t)w.c16_nsuper);  // and the curve order, behind
        A.add(&w.c16_nbr, 27 * (size_t)w.c16_nsuper);
    }
    A.add(&w.c16_base, (size_t)w.c16_nsuper + 2);
    if (c16_lists(w)) {
        A.add(&w.c16_list, std::min<size_t>(w.c16_nsuper, w.cap));
        A.add(&w.c16_list_n, 1);
        A.add(&w.c16_sums, scan_sums(w.c16_nsuper + 1));
    }
    A.add(&w.c16_rowcell, vec);
    if (ns) {
        A.add(&w.c16_dense, (size_t)w.c16_nsuper + 2);
        A.add(&w.c16_sfirst, ns + 1);
        A.add(&w.c16_srow, ns + 1);
        A.add(&w.c16_tb, PPE_MAX_SCENES + 1);
        A.add(&w.c16_rowlist, vec);
        A.add(&w.c16_nrows, 1);
        A.add(&w.c16_tsum, 2 * tiles * C16_SUMS);
    }
    A.add(&w.cpos, cap);
    A.add(&w.clen, vec);
    A.add(&w.c16_off, slices + 2);
    A.add(&w.c16_ent, chunks * C16_CHUNK_BYTES);
    A.add(&w.c16_tile, tiles * (sizeof(C16Tile) / sizeof(uint32_t)));
    A.add(&w.c16_collist, tiles * C16_COLS);
    A.add(&w.c16_stats, C16_STATS);
    A.add(&w.cb64, vec);
    A.add(&w.cx64, vec);
    A.add(&w.cdiag64, vec);
    A.add(&w.cdiag32, vec);
    A.add(&w.cinv_diag, vec);
    A.add(&w.cdsq, vec);
    A.add(&w.cr, vec);
    A.add(&w.cp, vec);
    A.add(&w.cpub[0], vec);
    A.add(&w.cpub[1], vec);
    A.add(&w.c16_slots, 2 * (size_t)w.sms * w.sms * C16_SUMS);
    A.add(&w.c16_epoch, 1);
    const bool have = A.get(&w.c16_block);
    if (!have) {
        ppe_c16_free(w);
        if (err) *err = "cudaMalloc failed for the compact PPE layout";
        return MPS_ERR_CUDA;
    }
    bool ok = true;
    cudaMemsetAsync(w.c16_stats, 0, C16_STATS * sizeof(uint32_t), st);
    cudaMemsetAsync(w.c16_epoch, 0, sizeof(unsigned long long), st);
    cudaMemsetAsync(w.c16_slots, 0, 2 * (size_t)w.sms * w.sms * C16_SUMS * sizeof(ulonglong2), st);
    if (!w.c16_shared) {
        std::vector<uint32_t> order(w.c16_nsuper);
        for (uint32_t s = 0; s < ngrids; s++) curve_order(C16Cells(grids[s]), order.data() + sfirst[s]);
        uint32_t* dev = w.c16_cells + 4 * (size_t)w.c16_nsuper;
        ok = cudaMemcpyAsync(dev, order.data(), order.size() * 4, cudaMemcpyHostToDevice, st) == cudaSuccess;
        for (uint32_t s = 0; s < ngrids && ok; s++) {
            const uint32_t first = sfirst[s], n = sfirst[s + 1] - first;
            uint32_t* rank = w.c16_base + first;  // each step writes the array anew
            k_c16_rank<<<cblocks(n, 256), 256, 0, st>>>(dev + first, n, first, rank);
            k_c16_links<<<cblocks(n, 8), 256, 0, st>>>(grids[s], C16Cells(grids[s]), dev + first, n, rank,
                                                       w.c16_cells + 4 * (size_t)first, w.c16_nbr + 27 * (size_t)first);
        }
        ok = cudaStreamSynchronize(st) == cudaSuccess && ok;  // before the order goes
    }
    if (!ok || (ns && cudaMemcpyAsync(w.c16_sfirst, sfirst.data(), sfirst.size() * 4, cudaMemcpyHostToDevice, st) != cudaSuccess) ||
        cudaFuncSetAttribute(k_c16_pack<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)C16_PAGE_BYTES_MAX) != cudaSuccess ||
        cudaFuncSetAttribute(k_c16_pack<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)C16_PAGE_BYTES_MAX) != cudaSuccess ||
        !c16_solver_smem()) {
        ppe_c16_free(w);
        if (err) *err = "the compact PPE solver cannot have its shared memory";
        return MPS_ERR_CUDA;
    }
    w.c16_ready = true;
    return MPS_OK;
}

void ppe_c16_free(PpeWork& w) {
    for (void* p : {(void*)w.c16_block, (void*)w.c16_spfirst, (void*)w.c16_spent, (void*)w.c16_spside})
        if (p) cudaFree(p);
    w.c16_block = nullptr;
    w.c16_cells = w.c16_nbr = w.c16_base = w.cpos = w.clen = w.c16_off = w.c16_tile = nullptr;
    w.c16_list = w.c16_list_n = w.c16_sums = w.c16_rowcell = nullptr;
    w.c16_collist = w.c16_stats = nullptr;
    w.c16_ent = nullptr;
    w.cb64 = w.cx64 = w.cdiag64 = nullptr;
    w.cdiag32 = w.cinv_diag = w.cdsq = w.cr = w.cp = nullptr;
    w.cpub[0] = w.cpub[1] = nullptr;
    w.c16_slots = nullptr;
    w.c16_dense = w.c16_sfirst = w.c16_srow = w.c16_tb = w.c16_rowlist = w.c16_nrows = nullptr;
    w.c16_tsum = nullptr;
    w.c16_epoch = nullptr;
    w.c16_spfirst = w.c16_spent = w.c16_spside = nullptr;
    w.c16_shared = false;
    w.c16_ready = false;
    w.c16 = false;
    w.c16_learned = false;
}

// the learned S' in the tiles' codes
int ppe_c16_learned_enable(PpeWork& w, std::string* err) {
    const int e = ppe_sp_enable(w, err);
    if (e != MPS_OK) return e;
    if (w.c16_spfirst) return MPS_OK;
    const size_t cap = ppe_rows_cap(w.cap, w.nscenes);
    const size_t tiles = c16_tiles((uint32_t)cap, (uint32_t)w.sms, w.nscenes);
    const size_t ent = (cap / SP_SLICE + tiles + 1) * SP_SLICE * LP_GW;
    bool ok = c16_alloc(&w.c16_spfirst, tiles * C16_SP_SLICES);
    ok &= c16_alloc(&w.c16_spent, ent);
    ok &= c16_alloc(&w.c16_spside, ent);
    if (!ok) {
        if (err) *err = "cudaMalloc failed for the learned compact preconditioner";
        return MPS_ERR_CUDA;
    }
    return MPS_OK;
}

// the tiles' row list and count (a batch's have gaps, the others' do not)
static const uint32_t* ppe_c16_rowlist(const PpeWork& w) { return w.c16_rowlist ? w.c16_rowlist : w.rowlist; }
static const uint32_t* ppe_c16_nrows(const PpeWork& w) { return w.c16_nrows ? w.c16_nrows : w.nrows; }
static uint32_t* c16_rowlist(PpeWork& w) { return const_cast<uint32_t*>(ppe_c16_rowlist(w)); }
static uint32_t* c16_nrows(PpeWork& w) { return const_cast<uint32_t*>(ppe_c16_nrows(w)); }

// The row numbers.
static int ppe_c16_enqueue_rows(PpeWork& w, const StageArgs& a, double bthr, bool fluid, cudaStream_t st) {
    C16Flag F;
    F.fluid = fluid;
    F.pos = a.cur.pos;
    F.n = a.cur.n;
    F.id = a.cur.id;
    F.sid_of_id = a.batch.n ? a.batch.sid_of_id : nullptr;
    F.scenes = a.batch.n ? w.scenes : nullptr;
    F.bthr = bthr;
    uint32_t* counts = a.batch.n ? w.c16_dense : w.c16_base;
    uint32_t warps = w.c16_nsuper + 1, launched = 0;
    if (w.c16_list) {
        cudaMemsetAsync(w.c16_list_n, 0, sizeof(uint32_t), st);
        launch(k_c16_occupied, cblocks(w.c16_nsuper + 1, 256), 256, 0, st, w.c16_cells, w.c16_nsuper, a.cell_start,
               counts, w.c16_list, w.c16_list_n);
        warps = std::min(w.c16_nsuper, w.cap);  // an occupied cell holds a particle
        launched = 3;
    }
    launch(k_c16_count, cblocks(warps * 32u, 256), 256, 0, st, F, w.c16_cells, w.c16_nsuper, w.c16_list, w.c16_list_n,
           a.cell_start, counts, w.c16_stats);
    if (w.c16_list) launch_scan_exclusive_many(counts, w.c16_nsuper + 1, w.c16_sums, st);
    else launch_scan_exclusive(counts, w.c16_nsuper + 1, st);
    C16RowArgs A;
    A.cells = w.c16_cells;
    A.cs = a.cell_start;
    A.base = w.c16_base;
    A.nsuper = w.c16_nsuper;
    A.list = w.c16_list;
    A.list_n = w.c16_list_n;
    A.rowcell = w.c16_rowcell;
    A.dense = a.batch.n ? w.c16_dense : nullptr;
    A.cpos = w.cpos;
    A.rowlist = c16_rowlist(w);
    A.nrows = c16_nrows(w);
    A.dense_list = w.rowlist;
    A.dense_n = w.nrows;
    A.rlen = w.rlen;
    A.diag64 = w.diag64;
    if (a.batch.n)
        launch(k_c16_shift, cblocks(w.c16_nsuper + 1, 256), 256, 0, st, w.c16_dense, w.c16_nsuper, w.c16_sfirst,
               w.nscenes, w.c16_base, w.c16_srow, A.rowlist, A.rowcell, A.nrows);
    launch(k_c16_rows, cblocks(warps * 32u, 256), 256, 0, st, F, A);
    return launched + (a.batch.n ? 4 : 3);
}

static uint32_t c16_maxslices(const PpeWork& w, uint32_t cap) {
    return (ppe_rows_cap(cap, w.nscenes) + C16_ROWS - 1) / C16_ROWS;
}

static C16AsmArgs c16_asm_args(PpeWork& w, const StageArgs& a, uint32_t cap) {
    C16AsmArgs A = {};
    A.a = a;
    A.scenes = w.scenes;
    A.rowlist = c16_rowlist(w);
    A.nrows = c16_nrows(w);
    A.cpos = w.cpos;
    A.cols = w.cols;
    A.wrm = w.wrm;
    A.clen = w.clen;
    A.rlen = w.rlen;
    A.bar = w.bar;
    A.diag64 = w.diag64;
    A.cb64 = w.cb64;
    A.cx64 = w.cx64;
    A.cdiag64 = w.cdiag64;
    A.cdiag32 = w.cdiag32;
    A.cinv_diag = w.cinv_diag;
    A.cdsq = w.cdsq;
    A.width = w.c16_off;
    A.maxslices = c16_maxslices(w, cap);
    return A;
}

int ppe_c16_enqueue_assemble(PpeWork& w, const StageArgs& a, const C16Assemble& K, uint32_t cap, cudaStream_t st) {
    const int launched = ppe_c16_enqueue_rows(w, a, K.beta * K.n0, false, st);
    C16AsmArgs A = c16_asm_args(w, a, cap);
    A.K = K;
    // a.cap_solid: particles that can have rows (not dummies)
    const uint32_t blocks = cblocks(ppe_rows_cap(a.cap_solid, w.nscenes) * 32u, 256);
    const uint32_t eblocks = cblocks(C16_ROWS * (A.maxslices + 1), 256);
    if (a.batch.n) {
        if (a.exact) launch(k_c16_assemble<true, true>, blocks, 256, 0, st, A);
        else launch(k_c16_assemble<false, true>, blocks, 256, 0, st, A);
        launch(k_c16_rowend<true>, eblocks, 256, 0, st, A);
    } else {
        if (a.exact) launch(k_c16_assemble<true, false>, blocks, 256, 0, st, A);
        else launch(k_c16_assemble<false, false>, blocks, 256, 0, st, A);
        launch(k_c16_rowend<false>, eblocks, 256, 0, st, A);
    }
    return launched + 2;
}

int ppe_c16_enqueue_pack(PpeWork& w, const StageArgs& a, uint32_t cap, cudaStream_t st) {
    const uint32_t ns = w.nscenes, rows = ppe_rows_cap(cap, ns), maxslices = c16_maxslices(w, cap);
    launch_scan_exclusive(w.c16_off, maxslices + 1, st);
    if (ns) launch(k_c16_cut, 1, 32, 0, st, w.c16_off, w.c16_srow, c16_nrows(w), ns, (uint32_t)w.sms, w.c16_tb);
    C16PackArgs P;
    P.cols_rm = w.cols;
    P.w_rm = w.wrm;
    P.clen = w.clen;
    P.nrows = c16_nrows(w);
    P.ns = ns;
    P.srow = w.c16_srow;
    P.tb = w.c16_tb;
    P.off = w.c16_off;
    P.base = w.c16_base;
    P.nbr = w.c16_nbr;
    P.rowcell = w.c16_rowcell;
    P.blocks = (uint32_t)w.sms;
    P.tiles = reinterpret_cast<C16Tile*>(w.c16_tile);
    P.collist = w.c16_collist;
    P.ent = w.c16_ent;
    P.stats = w.c16_stats;
    P.rowlist = c16_rowlist(w);
    P.cpos = w.cpos;
    P.idv = a.cur.id;
    P.index_of_id = w.index_of_id;
    P.dsq = w.cdsq;
    P.s_cnt = w.lp.s_cnt;
    P.s_col = w.lp.s_col;
    P.s_val = w.lp.s_val;
    P.s_diag = w.lp.s_diag;
    P.sc = a.sc;
    P.sp_first = w.c16_spfirst;
    P.sp_ent = w.c16_spent;
    P.sp_side = w.c16_spside;
    P.sp_diag = w.sp_diag;
    const uint32_t tiles = c16_tiles(rows, (uint32_t)w.sms, ns);
    if (w.c16_learned) launch(k_c16_pack<true>, tiles, C16_PACK_THREADS, c16_page_bytes(rows), st, P);
    else launch(k_c16_pack<false>, tiles, C16_PACK_THREADS, c16_page_bytes(rows), st, P);
    return ns ? 3 : 2;
}

int ppe_c16_enqueue_solve(PpeWork& w, const StageArgs& a, const mps_options& opt, uint32_t cap, cudaStream_t st) {
    C16Args S;
    S.nrows = c16_nrows(w);
    S.ns = w.nscenes;
    S.tb = w.c16_tb;
    S.tsum = w.c16_tsum;
    S.iters = w.scene_iters;
    S.outers = w.scene_outer;
    S.srel = w.scene_relres;
    S.off = w.c16_off;
    S.ent = w.c16_ent;
    S.cols_rm = w.cols;
    S.tiles = reinterpret_cast<const C16Tile*>(w.c16_tile);
    S.collist = w.c16_collist;
    S.stats = w.c16_stats;
    S.b64 = w.cb64;
    S.diag64 = w.cdiag64;
    S.diag32 = w.cdiag32;
    S.inv_diag = w.cinv_diag;
    S.x64 = w.cx64;
    S.p = w.cp;
    S.r = w.cr;
    S.pub0 = w.cpub[0];
    S.pub1 = w.cpub[1];
    S.slots = w.c16_slots;
    S.epoch = w.c16_epoch;
    S.sc = a.sc;
    S.tol = opt.cg_tol;
    S.max_iter = opt.cg_max_iter;
    S.inner_cap = opt.cg_check_every > 0 ? opt.cg_check_every : 500;
    S.eta_min = pow(10.0, -(double)(opt.cg_inner_digits > 0 ? opt.cg_inner_digits : 4));
    S.max_outer = 40;
    // the share of the matrix kept in L2: the same byte budget as the 8-byte layout
    S.keep = w.l2_keep_entries == 0xFFFFFFFFu ? 0xFFFFFFFFu
                                               : (uint32_t)((size_t)w.l2_keep_entries * 8 / C16_CHUNK_BYTES);
    S.ahead_from = (uint32_t)((size_t)w.l2_bytes / 2 *
                            (w.c16_learned ? C16_AHEAD_FROM_SP : C16_AHEAD_FROM) / C16_CHUNK_BYTES);
    const int chunks = w.c16_smem_chunks < 0 ? 0 : (w.c16_smem_chunks > 8 ? 8 : w.c16_smem_chunks);
    S.smem_chunks = (uint32_t)chunks * 32;  // of the 32 warps an SM's share is counted in
    S.smem_bytes = (uint32_t)C16_SMEM;
    S.sp_first = w.c16_spfirst;
    S.sp_ent = w.c16_spent;
    S.sp_side = w.c16_spside;
    S.sp_diag = w.sp_diag;
    void* args[] = {&S};
    const void* fn = w.nscenes ? (w.c16_learned ? (const void*)k_ppe_solve_c16_batch<true>
                                                : (const void*)k_ppe_solve_c16_batch<false>)
                               : (w.c16_learned ? (const void*)k_ppe_solve_c16<true> : (const void*)k_ppe_solve_c16<false>);
    w.launch_err = launch_cooperative_smem(fn, w.sms, C16_THREADS, C16_SMEM, args, st);
    if (!w.write_pressure) return 1;
    launch(k_c16_finish, cblocks(cap, 256), 256, 0, st, w.cx64, w.cpos, a.cur.press, a.sc);
    return 2;
}

// One velocity component of the Crank-Nicolson viscosity: assembly, pack,
// solve, update.  The components' rows are the same: numbered with the first.
int ppe_c16_enqueue_cn(PpeWork& w, const StageArgs& a, const mps_options& opt, int c, double lambda_n0_over_dim_niu,
                       uint32_t cap, cudaStream_t st) {
    int launched = c == 0 ? ppe_c16_enqueue_rows(w, a, 0.0, true, st) : 0;
    C16CnArgs C;
    C.A = c16_asm_args(w, a, cap);
    C.c = c;
    C.moved = w.moved;
    C.lambda_n0_over_dim_niu = lambda_n0_over_dim_niu;
    const uint32_t blocks = cblocks(a.cap_fluid * 32u, 256);
    if (a.exact) launch(k_c16_cn_assemble<true>, blocks, 256, 0, st, C);
    else launch(k_c16_cn_assemble<false>, blocks, 256, 0, st, C);
    launch(k_c16_cn_rowend, cblocks(C16_ROWS * (C.A.maxslices + 1), 256), 256, 0, st, C);
    launched += 2 + ppe_c16_enqueue_pack(w, a, cap, st);
    launched += ppe_c16_enqueue_solve(w, a, opt, cap, st);
    launch(k_c16_cn_finish, cblocks(cap, 256), 256, 0, st, w.cx64, w.cpos, a.cur, c, a.sc, w.moved);
    return launched + 1;
}

int ppe_sp_enable(PpeWork& w, std::string* err) {
    if (lp_alloc_symmetric(w.lp) != MPS_OK) {
        if (err) *err = "cudaMalloc failed for the learned symmetric form";
        return MPS_ERR_CUDA;
    }
    if (w.sp_ent) return MPS_OK;
    const size_t slices = (w.cap + SP_SLICE - 1) / SP_SLICE + 2;
    w.sp_cap_chunks = slices * (LP_GW + 1);  // entries per lane position: 32-row slices of up to LP_GW + 1
    bool ok = c16_alloc(&w.sp_off, slices + 2);
    ok &= c16_alloc(&w.sp_ent, w.sp_cap_chunks * SP_SLICE);
    ok &= c16_alloc(&w.sp_diag, (size_t)ppe_rows_cap(w.cap, w.nscenes) + 8);
    ok &= c16_alloc(&w.rq[0], (size_t)w.cap + 8);
    ok &= c16_alloc(&w.rq[1], (size_t)w.cap + 8);
    if (!ok) {
        if (err) *err = "cudaMalloc failed for the learned preconditioner";
        return MPS_ERR_CUDA;
    }
    cudaMemset(w.rq[0], 0, ((size_t)w.cap + 8) * sizeof(float2));
    cudaMemset(w.rq[1], 0, ((size_t)w.cap + 8) * sizeof(float2));
    return MPS_OK;
}

int ppe_sp_enqueue_pack(PpeWork& w, const StageArgs& a, uint32_t cap, cudaStream_t st) {
    SpArgs A;
    A.rowlist = w.rowlist;
    A.nrows = w.nrows;
    A.idv = a.cur.id;
    A.index_of_id = w.index_of_id;
    A.rlen = w.rlen;
    A.diag64 = w.diag64;
    A.s_cnt = w.lp.s_cnt;
    A.s_col = w.lp.s_col;
    A.s_val = w.lp.s_val;
    A.s_diag = w.lp.s_diag;
    A.sc = a.sc;
    A.off = w.sp_off;
    A.ent = w.sp_ent;
    A.diag = w.sp_diag;
    const uint32_t maxslices = (cap + SP_SLICE - 1) / SP_SLICE;
    A.maxslices = maxslices;
    const uint32_t wb = cblocks((maxslices + 1) * SP_SLICE, 256), pb = cblocks(maxslices * SP_SLICE, 256);
    launch(k_sp_width, wb, 256, 0, st, A);
    launch_scan_exclusive(w.sp_off, maxslices + 1, st);
    launch(k_sp_pack, pb, 256, 0, st, A);
    return 3;
}

int ppe_c16_export(const PpeWork& w, uint32_t np, const uint32_t* d_row_start, uint32_t* d_cols, float* d_w,
                   cudaStream_t st) {
    const uint32_t tiles = c16_tiles(ppe_rows_cap(np, w.nscenes), (uint32_t)w.sms, w.nscenes);
    k_c16_export<<<tiles, 256, 0, st>>>(reinterpret_cast<const C16Tile*>(w.c16_tile), w.c16_collist, (uint32_t)w.sms,
                                        w.nscenes, w.clen, ppe_c16_rowlist(w), ppe_c16_nrows(w), w.c16_off, w.c16_ent, w.cols,
                                        d_row_start, d_cols, d_w);
    return MPS_OK;
}

}  // namespace mpsb
