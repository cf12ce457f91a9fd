// Dual contouring on a dense grid (sm_103a).
//
// Steps (each a C entry point; the Python layer sizes buffers between them):
//   classify   sign bitmap (mc_signs) and, per 32-cell word, the number of
//              active cells and crossings, summed per block of 1024 words.
//   intersect  crossing points (lerp, the reference's arithmetic), optional
//              normals from the cell's trilinear interpolant, active cell ids
//              and CSR offsets -- isoext's Intersection (src/its.cu:94-283).
//   solve      per active cell: QEF normal equations accumulated in the
//              reference's order (src/dc.cu:14-65), a register-resident 3x3
//              symmetric Jacobi solve in FP32 with the reference's pseudo-inverse
//              threshold (src/batched_la.cu:152-178) refined once with a
//              double-FP32 residual, clipped to the cell (src/dc.cu:82-99).
//   quads      crossed grid edges in the reference's quad order (by low
//              endpoint, then z, y, x edge; src/grid/uniform.cu:60-83), their 4
//              cells, orientation and diagonal split (src/dc.cu:101-157).
//   weld       dual vertices used by faces, merged by exact position with a
//              hash table (isoext welds by sorted position, src/utils.cu:32-59).
#include <algorithm>
#include <cstdint>

#include "common.cuh"
#define ISO_LUT_DECL static __constant__ const
#include "luts.h"
#include "dc_common.cuh"
#include "lookback.cuh"
#include "profile.cuh"
#include "weld_table.cuh"

namespace {

constexpr int DC_BLOCK = 1024;

// Sign words of a grid row (x, y), aligned to z = 0.
__device__ __forceinline__ const uint32_t* srow(const uint32_t* S, const Grid3& g, int x, int y) {
    const int NWg = (g.nz + 31) / 32;
    return S + ((long long)x * g.ny + y) * NWg;
}
__device__ __forceinline__ uint32_t word_or0(const uint32_t* row, int w, int nw) {
    return (w >= 0 && w < nw) ? row[w] : 0u;
}

// Active-cell mask of cell word (cx, cy, w): cells z in [32w, 32w+32).
__device__ __forceinline__ uint32_t cell_act(const uint32_t* S, const Grid3& g, int cx, int cy, int w,
                                             uint32_t* cw8) {
    const int NWg = (g.nz + 31) / 32;
    uint32_t and8 = ~0u, or8 = 0u;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t* r = srow(S, g, cx + (k >> 1), cy + (k & 1));
        const uint32_t a = r[w];
        const uint32_t b = __funnelshift_r(a, word_or0(r, w + 1, NWg), 1);  // bit z <- z + 1
        cw8[2 * k] = a;
        cw8[2 * k + 1] = b;
        and8 &= a & b;
        or8 |= a | b;
    }
    return (or8 & ~and8) & iso::range_mask(w, 0, g.nz - 2);  // cells z <= nz - 2
}
// Case bits of cell at bit b of a cell word, from the 8 corner words cw8
// (index 2k = dz 0, 2k+1 = dz 1 for (dx, dy) = (k >> 1, k & 1)).
__device__ __forceinline__ uint32_t case_of(const uint32_t* cw8, int b) {
    uint32_t cs = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int dx = k >> 1, dy = k & 1;
        cs |= ((cw8[2 * k] >> b) & 1u) << (4 * dx + 2 * dy);
        cs |= ((cw8[2 * k + 1] >> b) & 1u) << (4 * dx + 2 * dy + 1);
    }
    return cs;
}

// Crossings of the active cells of a cell word: the edge table's crossed
// edges are exactly the edges whose corners differ in sign, and corner j's sign
// word is cw8[j], so this is a sum of 12 popcounts.
__device__ __forceinline__ uint32_t word_crossings(const uint32_t* cw8, uint32_t act) {
    uint32_t nk = 0;
#pragma unroll
    for (int e = 0; e < 12; ++e) nk += __popc((cw8[iso_edge_corner(2 * e)] ^ cw8[iso_edge_corner(2 * e + 1)]) & act);
    return nk;
}

// Block-wide exclusive scan of two values per thread (NT threads, a multiple
// of 32).
template <int NT = DC_BLOCK>
__device__ __forceinline__ void block_scan2(uint32_t a, uint32_t b, uint32_t& ea, uint32_t& eb,
                                            uint32_t& ta, uint32_t& tb, uint32_t* sm /*66*/) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t ia = a, ib = b;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t x = __shfl_up_sync(~0u, ia, d), y = __shfl_up_sync(~0u, ib, d);
        if (lane >= d) { ia += x; ib += y; }
    }
    if (lane == 31) { sm[warp] = ia; sm[32 + warp] = ib; }
    __syncthreads();
    if (warp == 0) {
        constexpr int NWARP = NT / 32;
        uint32_t x = lane < NWARP ? sm[lane] : 0u, y = lane < NWARP ? sm[32 + lane] : 0u;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t u = __shfl_up_sync(~0u, x, d), v = __shfl_up_sync(~0u, y, d);
            if (lane >= d) { x += u; y += v; }
        }
        sm[lane] = x;
        sm[32 + lane] = y;
    }
    __syncthreads();
    ea = (warp ? sm[warp - 1] : 0u) + ia - a;
    eb = (warp ? sm[32 + warp - 1] : 0u) + ib - b;
    ta = sm[31];
    tb = sm[63];
    __syncthreads();
}

// ---------------------------------------------------------------------------
// classify: per cell word, active cells and crossings; block sums.

__global__ void __launch_bounds__(DC_BLOCK) dc_cell_count(const uint32_t* __restrict__ S, Grid3 g,
                                                          long long nwords,
                                                          unsigned long long* __restrict__ blk) {
    __shared__ uint32_t sm[66];
    const long long i = (long long)blockIdx.x * DC_BLOCK + threadIdx.x;
    uint32_t na = 0, nk = 0;
    if (i < nwords) {
        const int NWc = (g.nz - 1 + 31) / 32;
        const int w = int(i % NWc);
        const long long r = i / NWc;
        const int cy = int(r % (g.ny - 1)), cx = int(r / (g.ny - 1));
        uint32_t cw8[8];
        const uint32_t act = cell_act(S, g, cx, cy, w, cw8);
        na = __popc(act);
        nk = word_crossings(cw8, act);
    }
    uint32_t ea, ek, ta, tk;
    block_scan2(na, nk, ea, ek, ta, tk, sm);
    if (threadIdx.x == 0) {
        blk[2 * blockIdx.x] = ta;
        blk[2 * blockIdx.x + 1] = tk;
    }
}

// Exclusive scan of block sums (one CTA; pairs of u64).  A round is bound by its
// chain of loads, shuffles and one barrier, so each takes 4096 pairs: a warp
// scans four rows of 32 (14,676 pairs: 16 us, 22 at 1024 pairs a round).
constexpr int BS_ROWS = 4;

__device__ __forceinline__ void warp_scan2(unsigned long long& a, unsigned long long& b, int lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long x = __shfl_up_sync(~0u, a, d), y = __shfl_up_sync(~0u, b, d);
        if (lane >= d) { a += x; b += y; }
    }
}

__global__ void __launch_bounds__(1024) dc_block_scan(unsigned long long* blk, long long nblk,
                                                      long long* totals) {
    __shared__ unsigned long long wa[2][32], wb[2][32];
    iso::grid_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool wide = (reinterpret_cast<uintptr_t>(blk) & 15) == 0;
    unsigned long long ca = 0, cb = 0;  // the rounds before
    int buf = 0;
    for (long long base = 0; base < nblk; base += 1024 * BS_ROWS, buf ^= 1) {
        const long long i0 = base + warp * (32 * BS_ROWS) + lane;
        unsigned long long a[BS_ROWS], b[BS_ROWS], ia[BS_ROWS], ib[BS_ROWS];
#pragma unroll
        for (int r = 0; r < BS_ROWS; ++r) {
            const long long i = i0 + 32 * r;
            a[r] = b[r] = 0;
            if (i < nblk) {
                if (wide) {
                    const ulonglong2 p = reinterpret_cast<const ulonglong2*>(blk)[i];
                    a[r] = p.x;
                    b[r] = p.y;
                } else {
                    a[r] = blk[2 * i];
                    b[r] = blk[2 * i + 1];
                }
            }
        }
        unsigned long long ta = 0, tb = 0;  // the warp's rows before
#pragma unroll
        for (int r = 0; r < BS_ROWS; ++r) {
            ia[r] = a[r];
            ib[r] = b[r];
            warp_scan2(ia[r], ib[r], lane);
            const unsigned long long ra = __shfl_sync(~0u, ia[r], 31), rb = __shfl_sync(~0u, ib[r], 31);
            ia[r] += ta - a[r];
            ib[r] += tb - b[r];
            ta += ra;
            tb += rb;
        }
        if (lane == 0) { wa[buf][warp] = ta; wb[buf][warp] = tb; }
        __syncthreads();  // the buffer's last reads are two rounds back
        // every warp scans the warps' sums itself
        unsigned long long x = wa[buf][lane], y = wb[buf][lane];
        const unsigned long long ox = x, oy = y;
        warp_scan2(x, y, lane);
        const unsigned long long ea = ca + __shfl_sync(~0u, x - ox, warp), eb = cb + __shfl_sync(~0u, y - oy, warp);
        ca += __shfl_sync(~0u, x, 31);
        cb += __shfl_sync(~0u, y, 31);
#pragma unroll
        for (int r = 0; r < BS_ROWS; ++r) {
            const long long i = i0 + 32 * r;
            if (i >= nblk) continue;
            if (wide) {
                reinterpret_cast<ulonglong2*>(blk)[i] = make_ulonglong2(ea + ia[r], eb + ib[r]);
            } else {
                blk[2 * i] = ea + ia[r];
                blk[2 * i + 1] = eb + ib[r];
            }
        }
    }
    if (threadIdx.x == 0) { totals[0] = (long long)ca; totals[1] = (long long)cb; }
}

// ---------------------------------------------------------------------------
// intersect: crossing points / normals, active cells, CSR offsets; also the
// per-word active mask and exclusive active-cell prefix used by the quads.

__global__ void __launch_bounds__(DC_BLOCK) dc_intersect(const uint32_t* __restrict__ S, Grid3 g, long long nwords,
                                                         const unsigned long long* __restrict__ blk,
                                                         uint32_t* __restrict__ actm,
                                                         uint32_t* __restrict__ offA, uint32_t* cell_ids,
                                                         uint32_t* cell_off, long long A, long long K) {
    __shared__ uint32_t sm[66];
    const long long i = (long long)blockIdx.x * DC_BLOCK + threadIdx.x;
    const int NWc = (g.nz - 1 + 31) / 32;
    uint32_t act = 0, na = 0, nk = 0;
    uint32_t cw8[8];
    int cx = 0, cy = 0, w = 0;
    if (i < nwords) {
        w = int(i % NWc);
        const long long r = i / NWc;
        cy = int(r % (g.ny - 1));
        cx = int(r / (g.ny - 1));
        act = cell_act(S, g, cx, cy, w, cw8);
        na = __popc(act);
        nk = word_crossings(cw8, act);
    }
    uint32_t ea, ek, ta, tk;
    block_scan2(na, nk, ea, ek, ta, tk, sm);
    if (i >= nwords) return;
    const unsigned long long a0 = blk[2 * blockIdx.x] + ea, k0 = blk[2 * blockIdx.x + 1] + ek;
    actm[i] = act;
    offA[i] = uint32_t(a0);
    if (!act || !cell_ids) return;
    // active cells of the word: id and the offset of their crossings (values are
    // read by dc_points, one thread per active cell)
    unsigned long long a = a0, k = k0;
    if (a0 >= (unsigned long long)A) return;
    while (act) {
        const int b = __ffs(act) - 1;
        act &= act - 1;
        const int cz = 32 * w + b;
        cell_ids[a] = uint32_t(((long long)cx * (g.ny - 1) + cy) * (g.nz - 1) + cz);
        cell_off[a] = uint32_t(k);
        k += __popc(uint32_t(ISO_EDGE_STATUS[case_of(cw8, b)]));
        ++a;
    }
    if (a == (unsigned long long)A) cell_off[A] = uint32_t(K);
}

// Crossing points (lerp with the reference's arithmetic) and optional normals of
// each active cell's crossed edges, in edge order (src/its.cu:94-159, 186-268).
__global__ void __launch_bounds__(256) dc_points(const float* __restrict__ vals, Grid3 g, float level,
                                                 const uint32_t* __restrict__ cell_ids,
                                                 const uint32_t* __restrict__ cell_off, long long A,
                                                 float* __restrict__ points, float* __restrict__ normals) {
    const long long a = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= A) return;
    const uint32_t cid = cell_ids[a];
    const int cz = int(cid % uint32_t(g.nz - 1));
    const uint32_t rr = cid / uint32_t(g.nz - 1);
    const int cy = int(rr % uint32_t(g.ny - 1)), cx = int(rr / uint32_t(g.ny - 1));
    CellCorners cc;
    load_cell(vals, g, cx, cy, cz, cc);
    uint32_t cs = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) cs |= uint32_t(iso::below(cc.v[j], level)) << j;
    const uint32_t est = edge_status(cs);
    unsigned long long k = cell_off[a];
#pragma unroll 1
    for (uint32_t em = est; em; em &= em - 1) {  // this lane's crossed edges, ascending
        const int e = __ffs(em) - 1;
        float p[3];
        edge_cross(cc, level, e, p);
        points[3 * k + 0] = p[0];
        points[3 * k + 1] = p[1];
        points[3 * k + 2] = p[2];
        if (normals) {
            float n[3];
            cell_normal(cc, p, n);
            normals[3 * k + 0] = n[0];
            normals[3 * k + 1] = n[1];
            normals[3 * k + 2] = n[2];
        }
        ++k;
    }
}

// Normals of an existing intersection from the grid (isoext computes them
// when dual_contouring is given an intersection without normals).
__global__ void dc_normals(const float* __restrict__ vals, Grid3 g, const float* __restrict__ points,
                           const uint32_t* __restrict__ cell_ids, const uint32_t* __restrict__ cell_off,
                           long long A, float* normals) {
    const long long a = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= A) return;
    const uint32_t cid = cell_ids[a];
    const int cz = int(cid % uint32_t(g.nz - 1));
    const uint32_t r = cid / uint32_t(g.nz - 1);
    const int cy = int(r % uint32_t(g.ny - 1)), cx = int(r / uint32_t(g.ny - 1));
    CellCorners cc;
    load_cell(vals, g, cx, cy, cz, cc);
    for (uint32_t k = cell_off[a]; k < cell_off[a + 1]; ++k) {
        const float p[3] = {points[3 * k], points[3 * k + 1], points[3 * k + 2]};
        float n[3];
        cell_normal(cc, p, n);
        normals[3 * k] = n[0];
        normals[3 * k + 1] = n[1];
        normals[3 * k + 2] = n[2];
    }
}

// Whether faces use the dual vertex of active cell (cx, cy, cz) with crossed
// edges est: some crossed edge has all four of its cells inside the grid (then
// its quad is emitted).  Cells at least one cell away from the grid's faces
// have only such edges.
__device__ __forceinline__ bool cell_used(const Grid3& g, int cx, int cy, int cz, uint32_t est) {
    if (cx >= 1 && cx <= g.nx - 3 && cy >= 1 && cy <= g.ny - 3 && cz >= 1 && cz <= g.nz - 3) return est != 0;
    for (uint32_t em = est; em; em &= em - 1) {
        const int e = __ffs(em) - 1;
        const int ca = edge_ca(e), ax = ca ^ edge_cb(e);  // 4 x, 2 y, 1 z
        const int x = cx + (ca >> 2), y = cy + ((ca >> 1) & 1), z = cz + (ca & 1);
        const bool okx = ax == 4 || (x >= 1 && x <= g.nx - 2);
        const bool oky = ax == 2 || (y >= 1 && y <= g.ny - 2);
        const bool okz = ax == 1 || (z >= 1 && z <= g.nz - 2);
        if (okx && oky && okz) return true;
    }
    return false;
}

// Crossings, grid normals and the QEF solve of each active cell in one pass,
// when nobody asked for the intersection: the same arithmetic as dc_points
// followed by dc_solve, without writing points and normals.  F: the arithmetic
// reading (g.fma), a template argument so that each reading compiles without
// the other's code.
template <bool F>
__global__ void __launch_bounds__(256) dc_cell_solve(const float* __restrict__ vals, Grid3 g, float level,
                                                     const uint32_t* __restrict__ cell_ids, long long A, float reg,
                                                     float svd_tol, float* __restrict__ dual) {
    const long long a = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= A) return;
    const uint32_t cid = cell_ids[a];
    const int cz = int(cid % uint32_t(g.nz - 1));
    const uint32_t rr = cid / uint32_t(g.nz - 1);
    const int cy = int(rr % uint32_t(g.ny - 1)), cx = int(rr / uint32_t(g.ny - 1));
    g.fma = F;
    CellCorners cc;
    load_cell(vals, g, cx, cy, cz, cc);
    uint32_t cs = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) cs |= uint32_t(iso::below(cc.v[j], level)) << j;
    const uint32_t est = edge_status(cs);
    Qef Q;
    qef_init(Q, g.fma);
    uint32_t K = 0;
#pragma unroll 1
    for (uint32_t em = est; em; em &= em - 1) {  // this lane's crossed edges, ascending
        const int e = __ffs(em) - 1;
        float p[3], n[3];
        edge_cross(cc, level, e, p);
        cell_normal(cc, p, n);
        qef_add(Q, p[0], p[1], p[2], n[0], n[1], n[2]);
        ++K;
    }
    qef_finish(Q, K, reg, svd_tol);
#pragma unroll
    for (int q = 0; q < 3; ++q)  // clipped to the cell's box
        dual[3 * a + q] = fminf(fmaxf(float(Q.x[q]), cc.p[0][q]), cc.p[7][q]);
}

// The solve for the call's arithmetic reading.
using SolveFn = void (*)(const float*, Grid3, float, const uint32_t*, long long, float, float, float*);
SolveFn solve_kernel(const Grid3& g) { return g.fma ? dc_cell_solve<true> : dc_cell_solve<false>; }

// Lane whose inclusive prefix first exceeds j (prefixes nondecreasing, j < total).
__device__ __forceinline__ int owner_lane(uint32_t incl, uint32_t j) {
    int lo = 0;
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) {
        const uint32_t pv = __shfl_sync(~0u, incl, lo + s - 1);
        if (pv <= j) lo += s;
    }
    return lo;
}

// ---------------------------------------------------------------------------
// solve

__global__ void dc_solve(const float* __restrict__ points, const float* __restrict__ normals,
                         const uint32_t* __restrict__ cell_ids, const uint32_t* __restrict__ cell_off,
                         long long A, Grid3 g, float reg, float svd_tol, float* dual) {
    const long long a = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= A) return;
    const uint32_t k0 = cell_off[a], k1 = cell_off[a + 1];
    Qef Q;
    qef_solve(points + 3ll * k0, normals + 3ll * k0, k1 - k0, reg, svd_tol, g.fma, Q);
    const double* x = Q.x;
    // clip to the cell box (corner 0 .. corner 7)
    const uint32_t cid = cell_ids[a];
    const uint32_t cz = cid % uint32_t(g.nz - 1);
    const uint32_t rr = cid / uint32_t(g.nz - 1);
    const uint32_t cy = rr % uint32_t(g.ny - 1), cx = rr / uint32_t(g.ny - 1);
    const uint32_t ci[3] = {cx, cy, cz};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float lo = coord(g, k, ci[k]), hi = coord(g, k, ci[k] + 1);
        dual[3 * a + k] = fminf(fmaxf(float(x[k]), lo), hi);
    }
}

// ---------------------------------------------------------------------------
// quads

// Crossed edges with a complete quad, per point word (points z in [32w, 32w+32)
// of row (x, y)), as masks for the z, y and x edges leaving each point.
__device__ __forceinline__ void quad_masks(const uint32_t* S, const Grid3& g, int x, int y, int w,
                                           uint32_t& mz, uint32_t& my, uint32_t& mx) {
    const int NWg = (g.nz + 31) / 32;
    const uint32_t* r = srow(S, g, x, y);
    const uint32_t s = r[w];
    // z edge (z -> z+1): cells (x-1..x, y-1..y, z)
    mz = my = mx = 0;
    const uint32_t zin = iso::range_mask(w, 1, g.nz - 2);     // 1 <= z <= nz-2
    const uint32_t zall = iso::range_mask(w, 0, g.nz - 2);    // z <= nz-2 (edge exists)
    if (x >= 1 && x <= g.nx - 2 && y >= 1 && y <= g.ny - 2)
        mz = (s ^ __funnelshift_r(s, word_or0(r, w + 1, NWg), 1)) & zall;
    // y edge (y -> y+1): cells (x-1..x, y, z-1..z)
    if (x >= 1 && x <= g.nx - 2 && y <= g.ny - 2) my = (s ^ srow(S, g, x, y + 1)[w]) & zin;
    // x edge (x -> x+1): cells (x, y-1..y, z-1..z)
    if (x <= g.nx - 2 && y >= 1 && y <= g.ny - 2) mx = (s ^ srow(S, g, x + 1, y)[w]) & zin;
}

__global__ void __launch_bounds__(DC_BLOCK) dc_quad_count(const uint32_t* __restrict__ S, Grid3 g,
                                                          long long nwords,
                                                          unsigned long long* __restrict__ blk) {
    __shared__ uint32_t sm[66];
    const long long i = (long long)blockIdx.x * DC_BLOCK + threadIdx.x;
    uint32_t nq = 0;
    if (i < nwords) {
        const int NWg = (g.nz + 31) / 32;
        const int w = int(i % NWg);
        const long long r = i / NWg;
        const int y = int(r % g.ny), x = int(r / g.ny);
        uint32_t mz, my, mx;
        quad_masks(S, g, x, y, w, mz, my, mx);
        nq = __popc(mz) + __popc(my) + __popc(mx);
    }
    uint32_t e0, e1, t0, t1;
    block_scan2(nq, 0u, e0, e1, t0, t1, sm);
    if (threadIdx.x == 0) {
        blk[2 * blockIdx.x] = t0;
        blk[2 * blockIdx.x + 1] = 0;
    }
}

// Active index of cell (cx, cy, cz): prefix of its word + active cells below it.
__device__ __forceinline__ uint32_t active_index(const uint32_t* actm, const uint32_t* offA,
                                                 const Grid3& g, int cx, int cy, int cz) {
    const int NWc = (g.nz - 1 + 31) / 32;
    const long long wi = ((long long)cx * (g.ny - 1) + cy) * NWc + (cz >> 5);
    return offA[wi] + __popc(actm[wi] & ((1u << (cz & 31)) - 1u));
}

// The k-th quad of a point word in the reference's order: by bit (low endpoint
// z) ascending, then the bit's z, y, x edges.
__device__ __forceinline__ void kth_quad(uint32_t mz, uint32_t my, uint32_t mx, uint32_t k, int& b, int& ax) {
    int lo = 0;  // largest lo with (quads of bits < lo) <= k
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) {
        const uint32_t m = (1u << (lo + s)) - 1u;  // lo + s <= 31
        if (uint32_t(__popc(mz & m) + __popc(my & m) + __popc(mx & m)) <= k) lo += s;
    }
    b = lo;
    const uint32_t below = (1u << lo) - 1u;
    uint32_t r = k - uint32_t(__popc(mz & below) + __popc(my & below) + __popc(mx & below));
    ax = 0;
    if ((mz >> b) & 1u) {
        if (r == 0) { ax = 2; return; }
        --r;
    }
    if ((my >> b) & 1u) {
        if (r == 0) { ax = 1; return; }
    }
}

// The quads of a block of point words, handed out over the lanes of each warp
// (a word has 0 .. 96 of them): every lane emits one quad per round.
__global__ void __launch_bounds__(DC_BLOCK) dc_quad_emit(const uint32_t* __restrict__ S, Grid3 g,
                                                         long long nwords,
                                                         const unsigned long long* __restrict__ blk,
                                                         const uint32_t* __restrict__ actm,
                                                         const uint32_t* __restrict__ offA,
                                                         const float* __restrict__ dual,
                                                         int32_t* __restrict__ tri) {
    __shared__ uint32_t sm[66];
    const long long i = (long long)blockIdx.x * DC_BLOCK + threadIdx.x;
    const int NWg = (g.nz + 31) / 32;
    const int lane = threadIdx.x & 31;
    uint32_t mz = 0, my = 0, mx = 0, sw = 0;
    int x = 0, y = 0, w = 0;
    if (i < nwords) {
        w = int(i % NWg);
        const long long r = i / NWg;
        y = int(r % g.ny);
        x = int(r / g.ny);
        quad_masks(S, g, x, y, w, mz, my, mx);
        sw = srow(S, g, x, y)[w];
    }
    const uint32_t nq = __popc(mz) + __popc(my) + __popc(mx);
    uint32_t eq, e1, tq, t1;
    block_scan2(nq, 0u, eq, e1, tq, t1, sm);
    const unsigned long long qb = blk[2 * blockIdx.x];
    uint32_t incl = nq;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(~0u, incl, d);
        if (lane >= d) incl += t;
    }
    const uint32_t total = __shfl_sync(~0u, incl, 31);
    for (uint32_t rr = 0; rr < total; rr += 32) {
        const uint32_t j = rr + lane;
        const int o = owner_lane(incl, min(j, total - 1));
        const uint32_t oexcl = __shfl_sync(~0u, incl - nq, o), oeq = __shfl_sync(~0u, eq, o);
        const uint32_t omz = __shfl_sync(~0u, mz, o), omy = __shfl_sync(~0u, my, o), omx = __shfl_sync(~0u, mx, o);
        const uint32_t os = __shfl_sync(~0u, sw, o);
        const int ox = __shfl_sync(~0u, x, o), oy = __shfl_sync(~0u, y, o), ow = __shfl_sync(~0u, w, o);
        if (j >= total) continue;
        const uint32_t k = j - oexcl;
        const unsigned long long q = qb + oeq + k;
        int b, ax;
        kth_quad(omz, omy, omx, k, b, ax);
        const int z = 32 * ow + b;
        // is_out = v(p0) <= v(p1): for a crossed edge this holds exactly when
        // the low endpoint p0 is below the level
        const bool out = (os >> b) & 1u;
        // edge_neighbors_table (src/shared_luts.cu:78-81): the 4 cells are p - o_i
        int c[4][3];
        if (ax == 0) {
            const int off[4][3] = {{0, 0, 0}, {0, 1, 0}, {0, 1, 1}, {0, 0, 1}};
            for (int t = 0; t < 4; ++t) { c[t][0] = ox - off[t][0]; c[t][1] = oy - off[t][1]; c[t][2] = z - off[t][2]; }
        } else if (ax == 1) {
            const int off[4][3] = {{0, 0, 0}, {0, 0, 1}, {1, 0, 1}, {1, 0, 0}};
            for (int t = 0; t < 4; ++t) { c[t][0] = ox - off[t][0]; c[t][1] = oy - off[t][1]; c[t][2] = z - off[t][2]; }
        } else {
            const int off[4][3] = {{0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0}};
            for (int t = 0; t < 4; ++t) { c[t][0] = ox - off[t][0]; c[t][1] = oy - off[t][1]; c[t][2] = z - off[t][2]; }
        }
        int32_t qi[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) qi[t] = int32_t(active_index(actm, offA, g, c[t][0], c[t][1], c[t][2]));
        if (!out) {
            const int32_t t0 = qi[0], t1q = qi[1];
            qi[0] = qi[3]; qi[1] = qi[2]; qi[2] = t1q; qi[3] = t0;
        }
        float v[4][3];
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int a = 0; a < 3; ++a) v[t][a] = dual[3 * (long long)qi[t] + a];
        int32_t* o6 = tri + 6 * q;
        if (dist3(v[0], v[2], g.fma) > dist3(v[1], v[3], g.fma)) {
            o6[0] = qi[1]; o6[1] = qi[3]; o6[2] = qi[0];
            o6[3] = qi[3]; o6[4] = qi[1]; o6[5] = qi[2];
        } else {
            o6[0] = qi[2]; o6[1] = qi[0]; o6[2] = qi[1];
            o6[3] = qi[0]; o6[4] = qi[2]; o6[5] = qi[3];
        }
    }
}

// ---------------------------------------------------------------------------
// weld: exact-position dedup of the dual vertices faces use.

using iso::pos_bits;
using iso::pos_hash;

__global__ void dc_mark_used(const int32_t* __restrict__ tri, long long n, uint32_t* used) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) used[tri ? tri[i] : int32_t(i)] = 1u;  // tri == nullptr: triangle i is point i (a soup)
}

// Probes before an insert gives up (the table is at most half full when the
// caller's capacity holds the distinct positions; past it the status says
// overflow and the counts give a size that fits).  Once the status says
// overflow, later threads skip their probes: the call's output is discarded.
constexpr uint32_t HASH_PROBES = 512;

// Insert used vertices; a slot keeps the smallest index with its position.
__global__ void dc_hash_insert(const float* __restrict__ dual, const uint32_t* __restrict__ used,
                               long long A, uint32_t* table, uint32_t mask, int* status) {
    const long long a = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= A || !used[a]) return;
    if (status && *(volatile int*)status == int(ISO_ERR_OVERFLOW)) return;
    const uint32_t k0 = pos_bits(dual[3 * a]), k1 = pos_bits(dual[3 * a + 1]), k2 = pos_bits(dual[3 * a + 2]);
    uint32_t h = pos_hash(k0, k1, k2) & mask;
    for (uint32_t probe = 0; probe <= mask && probe < HASH_PROBES; ++probe, h = (h + 1) & mask) {
        const uint32_t cur = atomicCAS(&table[h], 0xffffffffu, uint32_t(a));
        if (cur == 0xffffffffu) return;
        const uint32_t j = cur;
        if (pos_bits(dual[3ll * j]) == k0 && pos_bits(dual[3ll * j + 1]) == k1 &&
            pos_bits(dual[3ll * j + 2]) == k2) {
            atomicMin(&table[h], uint32_t(a));
            return;
        }
    }
    if (status) atomicCAS(status, 0, int(ISO_ERR_OVERFLOW));
}

// rep[a] = smallest index with the same position (for used vertices).
__global__ void dc_hash_lookup(const float* __restrict__ dual, const uint32_t* __restrict__ used,
                               long long A, const uint32_t* __restrict__ table, uint32_t mask,
                               uint32_t* rep) {
    const long long a = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= A) return;
    if (!used[a]) { rep[a] = 0xffffffffu; return; }
    const uint32_t k0 = pos_bits(dual[3 * a]), k1 = pos_bits(dual[3 * a + 1]), k2 = pos_bits(dual[3 * a + 2]);
    uint32_t h = pos_hash(k0, k1, k2) & mask;
    for (uint32_t probe = 0; probe <= mask && probe < HASH_PROBES; ++probe, h = (h + 1) & mask) {
        const uint32_t j = table[h];
        if (j == 0xffffffffu) break;
        if (pos_bits(dual[3ll * j]) == k0 && pos_bits(dual[3ll * j + 1]) == k1 &&
            pos_bits(dual[3ll * j + 2]) == k2) {
            rep[a] = j;
            return;
        }
    }
    rep[a] = uint32_t(a);
}

// Per block of 1024 dual vertices: number of representatives (rep[a] == a).
__global__ void __launch_bounds__(DC_BLOCK) dc_rep_count(const uint32_t* __restrict__ rep, long long A,
                                                         unsigned long long* blk) {
    __shared__ uint32_t sm[66];
    const long long a = (long long)blockIdx.x * DC_BLOCK + threadIdx.x;
    const uint32_t is = (a < A && rep[a] == uint32_t(a)) ? 1u : 0u;
    uint32_t e0, e1, t0, t1;
    block_scan2(is, 0u, e0, e1, t0, t1, sm);
    if (threadIdx.x == 0) { blk[2 * blockIdx.x] = t0; blk[2 * blockIdx.x + 1] = 0; }
}

__global__ void __launch_bounds__(DC_BLOCK) dc_rep_write(const uint32_t* __restrict__ rep, long long A,
                                                         const unsigned long long* __restrict__ blk,
                                                         const float* __restrict__ dual, uint32_t* newidx,
                                                         float* vout, uint32_t* vsrc) {
    __shared__ uint32_t sm[66];
    const long long a = (long long)blockIdx.x * DC_BLOCK + threadIdx.x;
    const uint32_t is = (a < A && rep[a] == uint32_t(a)) ? 1u : 0u;
    uint32_t e0, e1, t0, t1;
    block_scan2(is, 0u, e0, e1, t0, t1, sm);
    if (!is) return;
    const unsigned long long o = blk[2 * blockIdx.x] + e0;
    newidx[a] = uint32_t(o);
    if (vsrc) vsrc[o] = uint32_t(a);
    vout[3 * o] = dual[3 * a];
    vout[3 * o + 1] = dual[3 * a + 1];
    vout[3 * o + 2] = dual[3 * a + 2];
}

__global__ void dc_remap(const int32_t* __restrict__ tri, long long n, const uint32_t* __restrict__ rep,
                         const uint32_t* __restrict__ newidx, int32_t* fout) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) fout[i] = int32_t(newidx[rep[tri ? tri[i] : int32_t(i)]]);
}

// ---------------------------------------------------------------------------
// One-call dual contouring: after the sign pass, five or six kernels chained by
// programmatic dependent launch, with the sizes kept on the device.
//
//   dc_cells (/ dc_cells_scan)
//                  the active cells, their crossings, and the quads each of them
//                  owns, per segment of point words.  A quad's owner is the cell
//                  whose lowest corner is the low endpoint of the quad's edge, so
//                  the reference's quad order (low endpoint, then z, y, x edge)
//                  is the owners' order.  The segments' sums are scanned and
//                  checked against the sizes.
//   dc_solve_cells per entry: its cell's number, the QEF solve and whether faces
//                  use the cell.
//   dc_weld_faces / dc_weld_number
//                  the exact-position weld.  A dual vertex is clipped to its
//                  cell's closed box, and the boxes of different cells meet only
//                  on shared faces, so a vertex strictly inside its box has a
//                  position of its own, and one on a face can only equal the
//                  vertices of the cells around that face, edge or corner.
//                  Representatives (smallest index of a position) are numbered
//                  in cell order.
//   dc_cell_quads  each active cell's quads with the final vertex numbers.

// Crossed edges of one cell (bit b of a cell word): the 12 corner-sign XORs.
__device__ __forceinline__ uint32_t cell_crossings(const uint32_t* cw8, int b) {
    uint32_t n = 0;
#pragma unroll
    for (int e = 0; e < 12; ++e) n += ((cw8[iso_edge_corner(2 * e)] ^ cw8[iso_edge_corner(2 * e + 1)]) >> b) & 1u;
    return n;
}

constexpr int CELLS_THREADS = 256;
constexpr int CELLS_WARPS = CELLS_THREADS / 32;
constexpr int CELLS_QUEUE = 512;      // cells a warp lays out at a time
// Point words per thread: four, or one on grids whose CTAs of four words per
// thread would leave SMs idle (256 x 256 x 128 points; the count of marching cubes
// has the same rule).
constexpr long long CELLS_FINE = 1ll << 18;
// Segments that the last CTA of dc_cells scans itself; with more, the fence and
// the atomic of every CTA cost more than the launch of dc_cells_scan.
constexpr uint32_t CELLS_SCAN = 1024;

// Geometry of the flat point-word bitmap and its segments (one CTA of dc_cells
// each).
struct PwGrid {
    int NWg;
    uint32_t syw, sxw, PW;  // row stride, plane stride, point words (< 2^32)
    bool vec;               // rows start on 16-byte boundaries
    int lgseg;              // log2 of the point words per segment
    uint32_t nseg;
};

PwGrid pw_grid(const Grid3& g) {
    PwGrid p;
    p.NWg = (g.nz + 31) / 32;
    p.syw = uint32_t(p.NWg);
    p.sxw = uint32_t(g.ny) * p.syw;
    p.PW = uint32_t(g.nx) * p.sxw;
    p.vec = (p.NWg & 3) == 0;
    p.lgseg = (long long)p.PW <= CELLS_FINE ? 8 : 10;
    p.nseg = uint32_t(((unsigned long long)p.PW + (1ull << p.lgseg) - 1) >> p.lgseg);
    return p;
}

// What dc_cells leaves for the other kernels.
struct CellIndex {
    PwGrid p;
    uint32_t* actm;             // per point word: its active cells
    uint32_t* offA;             // per word with active cells: their first's index within the segment
    uint4* seg;                 // per segment: active cells, owned quads and crossings before it
    unsigned long long* elist;  // per active cell, unordered: word | bit << 32 | quad bits << 37 | quad offset << 41
    uint32_t* klist;            // per entry: its crossings' offset within the segment (only when asked for)
};

__device__ __forceinline__ void pw_xyw(const Grid3& g, const PwGrid& p, uint32_t pw, int& x, int& y, int& w) {
    const uint32_t row = pw / p.syw;
    w = int(pw - row * p.syw);
    x = int(row / uint32_t(g.ny));
    y = int(row - uint32_t(x) * uint32_t(g.ny));
}

// Owned quad edges of a cell word's active cells: corner 0 to corner 1 (z),
// 2 (y), 4 (x); complete when the edge's other two coordinates are >= 1 (the
// upper bounds hold for every cell).
__device__ __forceinline__ void owned_quads(const Grid3& g, const uint32_t* cw8, uint32_t act, int cx, int cy, int w,
                                            uint32_t& qz, uint32_t& qy, uint32_t& qx) {
    const uint32_t zin = iso::range_mask(w, 1, g.nz - 2);
    qz = (cx >= 1 && cy >= 1) ? (cw8[0] ^ cw8[1]) & act : 0u;
    qy = cx >= 1 ? (cw8[0] ^ cw8[2]) & act & zin : 0u;
    qx = cy >= 1 ? (cw8[0] ^ cw8[4]) & act & zin : 0u;
}

// Exclusive scan of the segments' (active, quads, crossings) sums in place by
// one CTA of T threads, and the totals against the capacities.
template <int T>
__device__ void scan_cells(uint4* seg, uint32_t nseg, long long capA, long long capQ, long long capK, long long* eff,
                           long long* counts, uint32_t* __restrict__ cell_off, int* status) {
    __shared__ unsigned long long part[3][T / 32], carry[3];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < 3) carry[tid] = 0;
    __syncthreads();
    for (uint32_t base = 0; base < nseg; base += T) {
        const uint32_t i = base + tid;
        const uint4 v = i < nseg ? __ldcg(seg + i) : make_uint4(0u, 0u, 0u, 0u);
        const unsigned long long c[3] = {v.x, v.y, v.z};
        unsigned long long in[3] = {v.x, v.y, v.z};
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                const unsigned long long u = __shfl_up_sync(~0u, in[t], d);
                if (lane >= d) in[t] += u;
            }
        if (lane == 31)
#pragma unroll
            for (int t = 0; t < 3; ++t) part[t][warp] = in[t];
        __syncthreads();
        if (warp < 3) {  // warp t: inclusive sums over the warps
            unsigned long long x = lane < T / 32 ? part[warp][lane] : 0ull;
#pragma unroll
            for (int d = 1; d < T / 32; d <<= 1) {
                const unsigned long long u = __shfl_up_sync(~0u, x, d);
                if (lane >= d) x += u;
            }
            if (lane < T / 32) part[warp][lane] = x;
        }
        __syncthreads();
        if (i < nseg) {
            unsigned long long e[3];
#pragma unroll
            for (int t = 0; t < 3; ++t) e[t] = carry[t] + (warp ? part[t][warp - 1] : 0ull) + in[t] - c[t];
            // offsets past 2^32 only matter when the sizes overflow (then nothing is used)
            seg[i] = make_uint4(uint32_t(e[0]), uint32_t(e[1]), uint32_t(e[2]), 0u);
        }
        __syncthreads();
        if (tid < 3) carry[tid] += part[tid][T / 32 - 1];
        __syncthreads();
    }
    if (tid == 0) {
        const long long A = (long long)carry[0], Q = (long long)carry[1], K = (long long)carry[2];
        const bool ok = A <= capA && Q <= capQ && K <= capK && A < 0x7fffffffll && Q < 0x7fffffffll && K < 0x7fffffffll;
        if (!ok) atomicCAS(status, 0, int(ISO_ERR_OVERFLOW));
        eff[0] = ok ? A : 0;
        eff[1] = ok ? K : 0;
        eff[2] = ok ? 6 * Q : 0;
        eff[3] = capA;
        counts[0] = 0;
        counts[1] = ok ? 2 * Q : 0;
        counts[2] = A;
        counts[3] = K;
        counts[4] = Q;
        if (cell_off && ok) cell_off[A] = uint32_t(K);
    }
}

struct CellsOut {
    unsigned long long* ctr;  // [0] entries [1] CTAs done (cleared by the sign pass)
    long long capA, capQ, capK;
    long long *eff, *counts;
    uint32_t* cell_off;
    int* status;
    float* gc;  // the grid's coordinates (x, then y, then z)
    unsigned long long* zero;  // to clear for the kernels that follow (the weld's look-back states)
    long long nzero;
};

__global__ void __launch_bounds__(1024) dc_cells_scan(const CellIndex ix, const CellsOut o) {
    iso::grid_wait();
    scan_cells<1024>(ix.seg, ix.p.nseg, o.capA, o.capQ, o.capK, o.eff, o.counts, o.cell_off, o.status);
}

// The active cells of one segment of point words (whose flat order is the cells'
// id order), from the bitmap alone.  As in the count of marching cubes the CTA
// first lists its words that may hold a crossing, a thread then takes one of
// them, and the cells of a warp's words are laid out in order in shared memory
// and leave as entries in coalesced stores.  An entry finds its cell's index
// through offA and seg, so no second pass numbers the cells: the kernel that
// works on them does (the write pass that did, a lane walking up to 128 cells of
// its words, took 12 us on a 41 x 57 x 48 grid, 29 us at 256^3 and 36 at 512^3).
// KOFF: crossings' offsets are asked for.  Bound by latency.
template <int WPT, bool KOFF>
__global__ void __launch_bounds__(CELLS_THREADS, 4) dc_cells(const uint32_t* __restrict__ S, Grid3 g,
                                                             const CellIndex ix, const CellsOut o) {
    constexpr int T = CELLS_THREADS, NW = CELLS_WARPS;
    constexpr uint32_t SEG = T * WPT;
    __shared__ unsigned long long wsum[NW], base_s;
    __shared__ uint32_t bsum[NW];
    __shared__ uint16_t list[SEG];  // words that may hold a crossing
    __shared__ uint32_t queue[NW][CELLS_QUEUE];
    __shared__ uint32_t kqueue[KOFF ? NW : 1][KOFF ? CELLS_QUEUE : 1];
    __shared__ int last_s;
    iso::grid_wait();
    const PwGrid& p = ix.p;
    for (uint32_t i = blockIdx.x * T + threadIdx.x; i < uint32_t(g.nx + g.ny + g.nz); i += gridDim.x * T) {
        const int axis = i < uint32_t(g.nx) ? 0 : (i < uint32_t(g.nx + g.ny) ? 1 : 2);
        o.gc[i] = coord(g, axis, i - (axis > 0 ? uint32_t(g.nx) : 0u) - (axis > 1 ? uint32_t(g.ny) : 0u));
    }
    for (long long i = (long long)blockIdx.x * T + threadIdx.x; i < o.nzero; i += (long long)gridDim.x * T)
        o.zero[i] = 0ull;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t seg0 = blockIdx.x * SEG;
    uint32_t nbusy = 0;
    {
        const uint32_t pw0 = seg0 + threadIdx.x * WPT;
        // a word is quiet when the rows' words and the words after them are all 0 or
        // all ~0 (conservative at the grid's edges)
        uint32_t lo[WPT], hi[WPT], nlo = ~0u, nhi = 0u;
#pragma unroll
        for (int k = 0; k < WPT; ++k) { lo[k] = ~0u; hi[k] = 0u; }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t a = pw0 + (q >> 1) * p.sxw + (q & 1) * p.syw;
            uint32_t v[WPT];
            if (WPT == 4 && p.vec && pw0 + WPT <= p.PW && a + WPT <= p.PW) {
                const uint4 v4 = __ldg(reinterpret_cast<const uint4*>(S + a));
                const uint32_t t[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
                for (int k = 0; k < WPT; ++k) v[k] = t[k];
            } else {
#pragma unroll
                for (int k = 0; k < WPT; ++k) v[k] = a + k < p.PW ? __ldg(S + a + k) : 0u;
            }
            uint32_t nx = __shfl_down_sync(~0u, v[0], 1);
            if (lane == 31) nx = a + WPT < p.PW ? __ldg(S + a + WPT) : 0u;
            nlo &= nx;
            nhi |= nx;
#pragma unroll
            for (int k = 0; k < WPT; ++k) { lo[k] &= v[k]; hi[k] |= v[k]; }
        }
        uint32_t m = 0;
#pragma unroll
        for (int k = 0; k < WPT; ++k) {
            const uint32_t l = lo[k] & (k + 1 < WPT ? lo[(k + 1) % WPT] : nlo);
            const uint32_t h = hi[k] | (k + 1 < WPT ? hi[(k + 1) % WPT] : nhi);
            if (l != ~0u && h != 0u && pw0 + k < p.PW) m |= 1u << k;
        }
        // quiet words have no active cell (the weld looks neighbours up)
        if (WPT == 4 && !m && pw0 + WPT <= p.PW) {
            *reinterpret_cast<uint4*>(ix.actm + pw0) = make_uint4(0u, 0u, 0u, 0u);
        } else {
#pragma unroll
            for (int k = 0; k < WPT; ++k)
                if (!((m >> k) & 1u) && pw0 + k < p.PW) ix.actm[pw0 + k] = 0u;
        }
        const uint32_t mine = __popc(m);
        uint32_t inc = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t t = __shfl_up_sync(~0u, inc, d);
            if (lane >= d) inc += t;
        }
        if (lane == 31) bsum[warp] = inc;
        __syncthreads();
        uint32_t at = inc - mine;
#pragma unroll
        for (int q = 0; q < NW; ++q) {
            at += q < warp ? bsum[q] : 0u;
            nbusy += bsum[q];
        }
        for (; m; m &= m - 1) list[at++] = uint16_t(threadIdx.x * WPT + __ffs(m) - 1);
    }
    uint32_t sa = 0, sq = 0, sk = 0;  // active cells, quads and crossings of the rounds so far
    for (uint32_t r0 = 0; r0 < nbusy; r0 += T) {
        __syncthreads();  // the list; the shared arrays of the round before
        const uint32_t i = r0 + threadIdx.x;
        uint32_t cw8[8], act = 0, qz = 0, qy = 0, qx = 0, nk = 0, pw = 0;
        if (i < nbusy) {
            pw = seg0 + list[i];
            int x, y, w;
            pw_xyw(g, p, pw, x, y, w);
            if (x < g.nx - 1 && y < g.ny - 1) {
                const bool nxt = w + 1 < p.NWg;
                uint32_t and8 = ~0u, or8 = 0u;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t a = pw + (k >> 1) * p.sxw + (k & 1) * p.syw;
                    const uint32_t lo = __ldg(S + a), hi = nxt ? __ldg(S + a + 1) : 0u;
                    cw8[2 * k] = lo;
                    cw8[2 * k + 1] = __funnelshift_r(lo, hi, 1);  // bit z <- z + 1
                    and8 &= cw8[2 * k] & cw8[2 * k + 1];
                    or8 |= cw8[2 * k] | cw8[2 * k + 1];
                }
                act = (or8 & ~and8) & iso::range_mask(w, 0, g.nz - 2);
                owned_quads(g, cw8, act, x, y, w, qz, qy, qx);
                nk = word_crossings(cw8, act);
            }
            ix.actm[pw] = act;
        }
        const uint32_t na = __popc(act), nq = __popc(qz) + __popc(qy) + __popc(qx);
        // active cells (at most 32 T), quads (from bit 20) and crossings (from 40)
        const unsigned long long mine = (unsigned long long)na | ((unsigned long long)nq << 20) |
                                        ((unsigned long long)nk << 40);
        unsigned long long inc = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned long long t = __shfl_up_sync(~0u, inc, d);
            if (lane >= d) inc += t;
        }
        if (lane == 31) wsum[warp] = inc;
        __syncthreads();
        unsigned long long before = 0, all = 0;
#pragma unroll
        for (int q = 0; q < NW; ++q) {
            before += q < warp ? wsum[q] : 0ull;
            all += wsum[q];
        }
        const uint32_t ta = uint32_t(all) & 0xfffffu;
        if (threadIdx.x == 0) base_s = ta ? atomicAdd(o.ctr, (unsigned long long)ta) : 0ull;
        const unsigned long long ex = inc - mine;  // within the warp
        if (act) ix.offA[pw] = sa + (uint32_t(before + ex) & 0xfffffu);
        __syncthreads();  // the entries' block; from here to the next round warps go their own ways
        const uint32_t n = uint32_t(__shfl_sync(~0u, inc, 31)) & 0xfffffu, c0 = uint32_t(ex) & 0xfffffu;
        const unsigned long long base = base_s + (uint32_t(before) & 0xfffffu);
        uint32_t* q = queue[warp];
        for (uint32_t q0 = 0; q0 < n; q0 += CELLS_QUEUE) {
            if (na && c0 < q0 + CELLS_QUEUE && c0 + na > q0) {
                uint32_t j = c0 - q0;  // wraps below q0: not in this window
                uint32_t qo = sq + (uint32_t((before + ex) >> 20) & 0xfffffu), ko = sk + uint32_t((before + ex) >> 40);
                for (uint32_t m = act; m; m &= m - 1, ++j) {
                    const int b = __ffs(m) - 1;
                    const uint32_t oz = (qz >> b) & 1u, oy = (qy >> b) & 1u, ox = (qx >> b) & 1u;
                    if (j < uint32_t(CELLS_QUEUE)) {
                        // bit, lane, quad bits (edges z, y, x; the low corner's sign), quad offset
                        q[j] = uint32_t(b) | (uint32_t(lane) << 5) | (oz << 10) | (oy << 11) | (ox << 12) |
                               (((cw8[0] >> b) & 1u) << 13) | (qo << 14);
                        if (KOFF) kqueue[KOFF ? warp : 0][KOFF ? j : 0] = ko;
                    }
                    qo += oz + oy + ox;
                    if (KOFF) ko += cell_crossings(cw8, b);
                }
            }
            __syncwarp();
            for (uint32_t j = lane; j < min(uint32_t(CELLS_QUEUE), n - q0); j += 32) {
                const uint32_t it = q[j];
                const unsigned long long e = base + q0 + j;
                if ((long long)e < o.capA) {
                    ix.elist[e] = (unsigned long long)(seg0 + list[r0 + warp * 32 + ((it >> 5) & 31u)]) |
                                  ((unsigned long long)(it & 31u) << 32) | ((unsigned long long)(it >> 10) << 37);
                    if (KOFF) ix.klist[e] = kqueue[KOFF ? warp : 0][KOFF ? j : 0];
                }
            }
            __syncwarp();
        }
        sa += ta;
        sq += uint32_t(all >> 20) & 0xfffffu;
        sk += uint32_t(all >> 40);
    }
    const bool scans = p.nseg <= CELLS_SCAN;
    if (threadIdx.x == 0) {
        ix.seg[blockIdx.x] = make_uint4(sa, sq, sk, 0u);
        if (scans) {
            __threadfence();
            last_s = atomicAdd(o.ctr + 1, 1ull) == p.nseg - 1;
            __threadfence();
        }
    }
    if (!scans) return;
    __syncthreads();
    if (last_s) scan_cells<T>(ix.seg, p.nseg, o.capA, o.capQ, o.capK, o.eff, o.counts, o.cell_off, o.status);
}

// Launches dc_cells (and its scan) over the sign bitmap S.
void launch_cells(const uint32_t* S, const Grid3& g, const CellIndex& ix, const CellsOut& o, cudaStream_t st) {
    const bool fine = ix.p.lgseg == 8;
    const auto kernel = o.cell_off ? (fine ? dc_cells<1, true> : dc_cells<4, true>)
                                   : (fine ? dc_cells<1, false> : dc_cells<4, false>);
    iso::launch_pdl(kernel, ix.p.nseg, unsigned(CELLS_THREADS), st, S, g, ix, o);
    if (ix.p.nseg > CELLS_SCAN) iso::launch_pdl(dc_cells_scan, 1u, 1024u, st, ix, o);
}

// The active cell of entry e: its coordinates and index.
struct ActiveCell {
    int x, y, z;
    uint32_t a, cid, qoff, qbits, kbase;
};

__device__ __forceinline__ ActiveCell entry_cell(const CellIndex& ix, const Grid3& g, unsigned long long e) {
    ActiveCell c;
    const uint32_t pw = uint32_t(e), b = uint32_t(e >> 32) & 31u;
    const uint4 s = __ldg(ix.seg + (pw >> ix.p.lgseg));
    const uint32_t m = __ldg(ix.actm + pw), off = __ldg(ix.offA + pw);
    int w;
    pw_xyw(g, ix.p, pw, c.x, c.y, w);
    c.z = 32 * w + int(b);
    c.a = s.x + off + __popc(m & ((1u << b) - 1u));
    c.cid = (uint32_t(c.x) * uint32_t(g.ny - 1) + uint32_t(c.y)) * uint32_t(g.nz - 1) + uint32_t(c.z);
    c.qbits = uint32_t(e >> 37) & 15u;
    c.qoff = s.y + uint32_t(e >> 41);
    c.kbase = s.z;
    return c;
}

// What the solve of an active cell leaves for the weld and the quads.
struct SolveOut {
    uint32_t *cells, *qoff;
    uint8_t *qbits, *used;  // used: 0 when no face uses the cell's vertex, else 1, or 3 when it lies on a face of its box
    float* dual;
    uint32_t* cell_off;     // optional: the first crossing
    uint32_t* flist;        // the cells of used vertices on a face (FaceList)
    unsigned long long* nface;
    long long fcap;
};

// A caller's intersection (GIVEN): points and normals of the crossings (normals
// may be null: from the grid), its cells and offsets.
struct Given {
    const float *points, *normals;
    const uint32_t *cells, *off;
    long long A;
    int* status;
};

// One thread per entry of dc_cells: the cell's number and records, and its dual
// vertex: crossings, grid normals and the QEF in one pass (the arithmetic of
// dc_points followed by dc_solve, nothing of it stored), or from a caller's
// intersection.  F: the arithmetic reading (g.fma), a template argument so that
// each reading compiles without the other's code.  Bound by FP32 issue (ten IEEE
// divisions per crossing keep the normals the reference's).
template <bool F, bool GIVEN>
__global__ void __launch_bounds__(256) dc_solve_cells(const float* __restrict__ vals, Grid3 g, float level,
                                                      const CellIndex ix, float reg, float svd_tol,
                                                      const long long* __restrict__ eff,
                                                      const float* __restrict__ gc, const SolveOut out,
                                                      const Given in) {
    iso::grid_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= eff[0]) return;
    const ActiveCell c = entry_cell(ix, g, __ldg(ix.elist + i));
    const long long a = c.a;
    out.cells[a] = c.cid;
    out.qoff[a] = c.qoff;
    out.qbits[a] = uint8_t(c.qbits);
    if (out.cell_off) out.cell_off[a] = c.kbase + ix.klist[i];
    g.fma = F;
    const bool inner = c.x >= 1 && c.x <= g.nx - 3 && c.y >= 1 && c.y <= g.ny - 3 && c.z >= 1 && c.z <= g.nz - 3;
    CellCorners cc;
    uint32_t est = 1;
    if (!GIVEN || !in.normals || !inner) {
        load_cell_table(vals, g, gc, c.x, c.y, c.z, cc);
        uint32_t cs = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) cs |= uint32_t(iso::below(cc.v[j], level)) << j;
        est = edge_status(cs);
    } else {
        cc.fma = F;
        cc.p[0][0] = gc[c.x]; cc.p[7][0] = gc[c.x + 1];
        cc.p[0][1] = gc[g.nx + c.y]; cc.p[7][1] = gc[g.nx + c.y + 1];
        cc.p[0][2] = gc[g.nx + g.ny + c.z]; cc.p[7][2] = gc[g.nx + g.ny + c.z + 1];
    }
    const bool is_used = inner ? est != 0 : cell_used(g, c.x, c.y, c.z, est);
    Qef Q;
    qef_init(Q, F);
    uint32_t K = 0;
    if (GIVEN) {
        // not this grid's intersection: the result is discarded, but every record is
        // written, for the kernels that follow
        const bool mine = eff[0] == in.A && in.cells[a] == c.cid;
        if (!mine) atomicCAS(in.status, 0, int(ISO_ERR_LOOKUP));
        const uint32_t k0 = mine ? in.off[a] : 0u;
        K = mine ? in.off[a + 1] - k0 : 0u;
        const float* pt = in.points + 3ll * k0;
        for (uint32_t k = 0; k < K; ++k) {
            const float p[3] = {pt[3 * k], pt[3 * k + 1], pt[3 * k + 2]};
            float n[3];
            if (in.normals) {
#pragma unroll
                for (int q = 0; q < 3; ++q) n[q] = in.normals[3ll * (k0 + k) + q];
            } else {
                cell_normal(cc, p, n);
            }
            qef_add(Q, p[0], p[1], p[2], n[0], n[1], n[2]);
        }
    } else {
#pragma unroll 1
        for (uint32_t em = est; em; em &= em - 1) {  // this lane's crossed edges, ascending
            float p[3], n[3];
            edge_cross(cc, level, __ffs(em) - 1, p);
            cell_normal(cc, p, n);
            qef_add(Q, p[0], p[1], p[2], n[0], n[1], n[2]);
            ++K;
        }
    }
    qef_finish(Q, K, reg, svd_tol);
    bool face = false;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const float lo = cc.p[0][q], hi = cc.p[7][q];  // the cell's box
        const float x = fminf(fmaxf(float(Q.x[q]), lo), hi);
        face |= x == lo || x == hi;
        out.dual[3 * a + q] = x;
    }
    out.used[a] = is_used ? (face ? 3 : 1) : 0;
    // list the vertex for the weld: one atomic per warp
    const bool on = is_used && face;
    const uint32_t m = __ballot_sync(__activemask(), on);
    if (on) {
        const int lane = threadIdx.x & 31, lead = __ffs(m) - 1;
        unsigned long long base = 0;
        if (lane == lead) base = atomicAdd(out.nface, (unsigned long long)__popc(m));
        base = __shfl_sync(m, base, lead) + __popc(m & ((1u << lane) - 1u));
        if ((long long)base < out.fcap) out.flist[base] = uint32_t(a);
    }
}

// The crossings' points (and normals) of the entries' cells, their ids and first
// crossings: isoext's Intersection (src/its.cu:94-159, 186-268).  A warp reads 32
// entries' cells, a lane each, into shared memory, and then takes their crossings
// one per lane: these are mostly consecutive rows of the output, so the stores
// coalesce, and no lane waits for a cell with more crossings.  A lane that walked
// its own cell's crossings stored rows 12 bytes wide some 70 apart, and the
// store queue bound it: for the 99.5 M crossings of 256^3 noise 2.50 ms with normals
// and 1.14 without, where this takes 1.61 and 0.80.
constexpr int ENTRY_THREADS = 256;  // at most

__global__ void __launch_bounds__(ENTRY_THREADS) dc_entry_points(
    const float* __restrict__ vals, Grid3 g, float level, const CellIndex ix, const long long* __restrict__ eff,
    const float* __restrict__ gc, uint32_t* __restrict__ cells, uint32_t* __restrict__ cell_off,
    float* __restrict__ points, float* __restrict__ normals, const long long* __restrict__ counts,
    const int* __restrict__ status, long long* host) {
    __shared__ float cell_s[ENTRY_THREADS / 32][14][32];   // corner values, low and high corner
    __shared__ uint32_t edge_s[ENTRY_THREADS / 32][3][32];  // crossed edges, crossings up to the cell's end, first crossing
    iso::grid_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {  // the sizes and the status for the host
        for (int k = 0; k < 5; ++k) host[k] = counts[k];
        host[5] = *status;
    }
    const int lane = threadIdx.x & 31;
    if (i - lane >= eff[0]) return;
    float(*cell)[32] = cell_s[threadIdx.x >> 5];
    uint32_t(*edge)[32] = edge_s[threadIdx.x >> 5];
    uint32_t est = 0, first = 0;
    if (i < eff[0]) {
        const ActiveCell c = entry_cell(ix, g, __ldg(ix.elist + i));
        first = c.kbase + ix.klist[i];
        cells[c.a] = c.cid;
        cell_off[c.a] = first;
        CellCorners cc;
        load_cell_table(vals, g, gc, c.x, c.y, c.z, cc);
        uint32_t cs = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            cs |= uint32_t(iso::below(cc.v[j], level)) << j;
            cell[j][lane] = cc.v[j];
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            cell[8 + q][lane] = cc.p[0][q];
            cell[11 + q][lane] = cc.p[7][q];
        }
        est = edge_status(cs);
    }
    uint32_t end = __popc(est);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(~0u, end, d);
        if (lane >= d) end += t;
    }
    edge[0][lane] = est;
    edge[1][lane] = end;
    edge[2][lane] = first;
    __syncwarp();
    const uint32_t total = edge[1][31];
#pragma unroll 1
    for (uint32_t j = lane; j < total; j += 32) {
        int o = 0;  // the first cell that ends past j
#pragma unroll
        for (int s = 16; s >= 1; s >>= 1)
            if (edge[1][o + s - 1] <= j) o += s;
        uint32_t em = edge[0][o];
        const uint32_t r = j - (edge[1][o] - __popc(em));
        const unsigned long long k = edge[2][o] + r;
        for (uint32_t q = 0; q < r; ++q) em &= em - 1;
        CellCorners cc;
        cc.fma = g.fma;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            cc.v[q] = cell[q][o];
            cc.p[q][0] = cell[(q >> 2) ? 11 : 8][o];
            cc.p[q][1] = cell[((q >> 1) & 1) ? 12 : 9][o];
            cc.p[q][2] = cell[(q & 1) ? 13 : 10][o];
        }
        float p[3];
        edge_cross(cc, level, __ffs(em) - 1, p);
#pragma unroll
        for (int q = 0; q < 3; ++q) points[3 * k + q] = p[q];
        if (normals) {
            float n[3];
            cell_normal(cc, p, n);
#pragma unroll
            for (int q = 0; q < 3; ++q) normals[3 * k + q] = n[q];
        }
    }
}

// Cells along one axis whose closed interval [coord(i), coord(i + 1)] holds v, in
// cell c's: c alone, or c and the cell on the side where v is the common
// coordinate (neighbouring coordinates are distinct here).  t: the axis's
// coordinates, n of them.
__device__ __forceinline__ void cells_holding(const float* __restrict__ t, int n, int c, float v, int& i0, int& i1) {
    i0 = c - (c > 0 && __ldg(t + c) == v ? 1 : 0);
    i1 = c + (c < n - 2 && __ldg(t + c + 1) == v ? 1 : 0);
}

// Where the solve lists the cells whose vertex lies on a face of their box.
struct FaceList {
    uint32_t* cells;          // active indices, unordered
    unsigned long long* n;    // their number, past cap where the list had no room
    long long cap;
};

// Weld, eight lanes per vertex on a face of its cell's box, a lane per cell around
// that face, edge or corner (two per axis on which the vertex lies on a face):
// looks for the used ones with the same position; where coordinates may repeat it
// reads their table instead (weld_table.cuh).  When one comes before the vertex's own, vmap[a] = 0x80000000 | the
// first of them and used[a] gets bit 2.  Bound by the latency of six dependent
// gathers; the list keeps every lane at it.  A pass over all cells waited in every
// warp for its few such lanes and their cells one after another: 18 us at 512^3,
// 8 on a 41 x 57 x 48 grid.
__global__ void __launch_bounds__(128) dc_weld_faces(Grid3 g, const CellIndex ix, const float* __restrict__ gc,
                                                     const FaceList list, const uint32_t* __restrict__ cells,
                                                     uint8_t* used, const float* __restrict__ dual,
                                                     const long long* __restrict__ eff,
                                                     uint32_t* __restrict__ vmap, const WeldTable table) {
    iso::grid_wait();
    const uint32_t A = uint32_t(eff[0]);
    const bool listed = (long long)*list.n <= list.cap;  // else every cell is looked at
    const uint32_t n = listed ? min(uint32_t(*list.n), A) : A;
    const uint32_t k = threadIdx.x & 7u, group = (threadIdx.x & 31u) & ~7u;
    const uint32_t step = gridDim.x * (blockDim.x / 8);
    // a warp's four groups stay together (the shuffles name the group's lanes only)
    for (uint32_t i = blockIdx.x * (blockDim.x / 8) + threadIdx.x / 8; i < n; i += step) {
        const uint32_t a = listed ? list.cells[i] : i;
        // (bit 0 is all that is read of another cell: the bits 2 that other threads
        // set meanwhile do not matter)
        if ((used[a] & 3u) != 3u) continue;
        uint32_t rep = a;
        if (table.slot) {
            if (k == 0) rep = table_first(table, dual, a);
        } else {
            const float p[3] = {dual[3ll * a], dual[3ll * a + 1], dual[3ll * a + 2]};
            const uint32_t cid = cells[a];
            const int cz = int(cid % uint32_t(g.nz - 1));
            const uint32_t rr = cid / uint32_t(g.nz - 1);
            const int cy = int(rr % uint32_t(g.ny - 1)), cx = int(rr / uint32_t(g.ny - 1));
            int x0, x1, y0, y1, z0, z1;
            cells_holding(gc, g.nx, cx, p[0], x0, x1);
            cells_holding(gc + g.nx, g.ny, cy, p[1], y0, y1);
            cells_holding(gc + g.nx + g.ny, g.nz, cz, p[2], z0, z1);
            const uint32_t ny = uint32_t(y1 - y0 + 1), nz = uint32_t(z1 - z0 + 1),
                           count = uint32_t(x1 - x0 + 1) * ny * nz;  // at most 8
            if (k < count) {
                const uint32_t z = uint32_t(z0) + k % nz, r = k / nz;
                const uint32_t y = uint32_t(y0) + r % ny, x = uint32_t(x0) + r / ny;
                const uint32_t wi = (x * uint32_t(g.ny) + y) * uint32_t(ix.p.NWg) + (z >> 5);
                const uint32_t mw = ix.actm[wi], bit = z & 31u;
                if ((mw >> bit) & 1u) {
                    const uint32_t ib = ix.seg[wi >> ix.p.lgseg].x + ix.offA[wi] + __popc(mw & ((1u << bit) - 1u));
                    if (ib < a && (used[ib] & 1u) && same_position(dual, a, ib)) rep = ib;
                }
            }
        }
        const uint32_t lanes = 0xffu << group;
#pragma unroll
        for (int d = 4; d >= 1; d >>= 1) rep = min(rep, __shfl_xor_sync(lanes, rep, d));
        if (k == 0 && rep != a) {
            vmap[a] = 0x80000000u | rep;
            used[a] = 7;
        }
    }
}

// The used vertices that are their position's first, numbered in cell order and
// written; vmap[a] = the number, or 0xffffffff where no face uses the cell.
// Tiles of 1024 cells in ticket order, chained by look-back: the work of a tile
// is the same everywhere, so no CTA waits long (a scan between two passes took
// two more launches).
constexpr int NUM_THREADS = 256, NUM_PER = 4;
constexpr int NUM_TILE = NUM_THREADS * NUM_PER;

__global__ void __launch_bounds__(NUM_THREADS) dc_weld_number(const float* __restrict__ dual,
                                                              const long long* __restrict__ eff,
                                                              const uint8_t* __restrict__ used,
                                                              unsigned long long* state, unsigned long long* ticket,
                                                              uint32_t* __restrict__ vmap, float* __restrict__ vout,
                                                              uint32_t* __restrict__ vsrc, long long* counts,
                                                              int* status) {
    __shared__ uint32_t tile_s, wcnt[NUM_PER][NUM_THREADS / 32];
    __shared__ unsigned long long pre_s;
    iso::grid_wait();
    const uint32_t A = uint32_t(eff[0]);
    if (threadIdx.x == 0) tile_s = uint32_t(atomicAdd(ticket, 1ull));
    __syncthreads();
    const uint32_t tile = tile_s;
    if (tile * (unsigned long long)NUM_TILE >= A) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t u[NUM_PER], bal[NUM_PER];
#pragma unroll
    for (int k = 0; k < NUM_PER; ++k) {
        const uint32_t a = tile * NUM_TILE + k * NUM_THREADS + threadIdx.x;
        u[k] = a < A ? used[a] : 0u;
    }
#pragma unroll
    for (int k = 0; k < NUM_PER; ++k) {
        bal[k] = __ballot_sync(~0u, (u[k] & 5u) == 1u);
        if (lane == 0) wcnt[k][warp] = __popc(bal[k]);
    }
    __syncthreads();
    if (warp == 0) {  // the tile's 32 (round, warp) counts, one per lane, in order
        static_assert(NUM_PER * (NUM_THREADS / 32) == 32, "one count per lane");
        uint32_t& mine = wcnt[lane / (NUM_THREADS / 32)][lane % (NUM_THREADS / 32)];
        const uint32_t c = mine;
        uint32_t inc = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t t = __shfl_up_sync(~0u, inc, d);
            if (lane >= d) inc += t;
        }
        mine = inc - c;
        const uint32_t total = __shfl_sync(~0u, inc, 31);
        unsigned long long e = 0, unused = 0;
        lb_tile(state, tile, total, 0, e, unused, status);
        if (lane == 0) {
            pre_s = e;
            if ((unsigned long long)(tile + 1) * NUM_TILE >= A) counts[0] = (long long)(e + total);
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NUM_PER; ++k) {
        const uint32_t a = tile * NUM_TILE + k * NUM_THREADS + threadIdx.x;
        if (a >= A) continue;
        if (!u[k]) vmap[a] = 0xffffffffu;
        if ((u[k] & 5u) != 1u) continue;
        const unsigned long long o = pre_s + wcnt[k][warp] + __popc(bal[k] & ((1u << lane) - 1u));  // < V <= A
        vmap[a] = uint32_t(o);
        vout[3 * o] = dual[3ll * a];
        vout[3 * o + 1] = dual[3ll * a + 1];
        vout[3 * o + 2] = dual[3ll * a + 2];
        if (vsrc) vsrc[o] = a;
    }
}

// The quads active cell a owns, in the reference's order and orientation
// (src/dc.cu:101-157): the 4 cells around the edge are p - o_i with the offsets
// of edge_neighbors_table (src/shared_luts.cu:78-81), the owner being o_0 = 0.
// Bound by the latency of its gathers, so they go in two rounds: the index
// records of the four words the neighbours lie in, then the vertices and numbers
// of all neighbours that any of the quads uses.
__global__ void __launch_bounds__(256) dc_cell_quads(const uint8_t* __restrict__ qbits, Grid3 g,
                                                     const uint32_t* __restrict__ cell_ids,
                                                     const uint32_t* __restrict__ qoff, const CellIndex ix,
                                                     const float* __restrict__ dual,
                                                     const uint32_t* __restrict__ vmap,
                                                     const long long* __restrict__ eff, int32_t* __restrict__ faces,
                                                     const long long* __restrict__ counts,
                                                     const int* __restrict__ status, long long* host) {
    iso::grid_wait();
    if (host && blockIdx.x == 0 && threadIdx.x == 0) {  // the sizes and the status for the host
        for (int k = 0; k < 5; ++k) host[k] = counts[k];
        host[5] = *status;
    }
    const long long a = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= eff[0]) return;
    // owned edges (z, y, x) and the sign of the low corner
    const uint32_t qb = qbits[a];
    if (!(qb & 7u)) return;
    const uint32_t cid = cell_ids[a];
    unsigned long long q = qoff[a];
    const bool s0 = (qb >> 3) & 1u;
    const int cz = int(cid % uint32_t(g.nz - 1));
    const uint32_t rr = cid / uint32_t(g.nz - 1);
    const int cy = int(rr % uint32_t(g.ny - 1)), cx = int(rr / uint32_t(g.ny - 1));
    // cells 0 .. 6: itself, z-1, y-1, (y-1, z-1), x-1, (x-1, z-1), (x-1, y-1); those in use
    const uint32_t use = 1u | ((qb & 1u) ? 0x54u : 0u) | ((qb & 2u) ? 0x32u : 0u) | ((qb & 4u) ? 0x0eu : 0u);
    const uint32_t NWg = uint32_t(ix.p.NWg), b = uint32_t(cz & 31);
    const uint32_t w0 = (uint32_t(cx) * uint32_t(g.ny) + uint32_t(cy)) * NWg + uint32_t(cz >> 5);
    uint32_t idx[7];
    idx[0] = uint32_t(a);
    // rows (x, y), (x, y-1), (x-1, y), (x-1, y-1): the cells at z and at z - 1
    uint32_t first[4], mask[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const uint32_t here = r ? 1u << (2 * r) : 0u, low = r < 3 ? 2u << (2 * r) : 0u;  // cells 2r and 2r + 1
        first[r] = mask[r] = 0u;
        if (!(use & (here | low))) continue;
        const uint32_t wr = w0 - uint32_t(r & 1) * NWg - uint32_t(r >> 1) * uint32_t(g.ny) * NWg;
        const uint32_t wl = wr - ((!(use & here) && b == 0u) ? 1u : 0u);  // only z - 1, in the word before
        mask[r] = ix.actm[wl];
        first[r] = ix.seg[wl >> ix.p.lgseg].x + ix.offA[wl];
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const uint32_t here = r ? 1u << (2 * r) : 0u, low = r < 3 ? 2u << (2 * r) : 0u;
        if (r) idx[2 * r] = first[r] + __popc(mask[r] & ((1u << b) - 1u));
        if (r < 3) {
            if (b) {
                idx[2 * r + 1] = first[r] + __popc(mask[r] & ((1u << (b - 1)) - 1u));
            } else if (use & low) {
                // z - 1 is the last cell of the word before
                uint32_t m = mask[r], f = first[r];
                if (use & here) {
                    const uint32_t wl = w0 - uint32_t(r & 1) * NWg - uint32_t(r >> 1) * uint32_t(g.ny) * NWg - 1u;
                    m = ix.actm[wl];
                    f = ix.seg[wl >> ix.p.lgseg].x + ix.offA[wl];
                }
                idx[2 * r + 1] = f + __popc(m & 0x7fffffffu);
            }
        }
    }
    float v[7][3];
    uint32_t f[7];
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        if (!((use >> k) & 1u)) continue;
#pragma unroll
        for (int d = 0; d < 3; ++d) v[k][d] = dual[3ll * idx[k] + d];
        f[k] = vmap[idx[k]];
    }
#pragma unroll
    for (int k = 0; k < 7; ++k)
        if (((use >> k) & 1u) && f[k] != 0xffffffffu && (f[k] & 0x80000000u)) f[k] = vmap[f[k] & 0x7fffffffu];
#pragma unroll
    for (int ax = 2; ax >= 0; --ax) {
        if (!((qb >> (2 - ax)) & 1u)) continue;
        // the quad's cells 1 .. 3
        const int c1 = ax == 0 ? 2 : (ax == 1 ? 1 : 4), c2 = ax == 0 ? 3 : (ax == 1 ? 5 : 6),
                  c3 = ax == 0 ? 1 : (ax == 1 ? 4 : 2);
        // is_out = v(p0) <= v(p1): for a crossed edge, p0 below the level; else the
        // order is reversed, which swaps its ends and its middles
        const bool second = dist3(s0 ? v[0] : v[c3], s0 ? v[c2] : v[c1], g.fma) >
                            dist3(s0 ? v[c1] : v[c2], s0 ? v[c3] : v[0], g.fma);
        const int32_t f0 = int32_t(s0 ? f[0] : f[c3]), f1 = int32_t(s0 ? f[c1] : f[c2]),
                      f2 = int32_t(s0 ? f[c2] : f[c1]), f3 = int32_t(s0 ? f[c3] : f[0]);
        int32_t* o6 = faces + 6 * q;
        o6[0] = second ? f1 : f2;
        o6[1] = second ? f3 : f0;
        o6[2] = second ? f0 : f1;
        o6[3] = second ? f3 : f0;
        o6[4] = second ? f1 : f2;
        o6[5] = second ? f2 : f3;
        ++q;
    }
}

}  // namespace

// mc_signs lives in mc_dense.cu
#include "mc_dense.cuh"

// ---------------------------------------------------------------------------
// C ABI

// Exclusive scan of per-block (u64, u64) sums in place, totals -> totals[0..1]
// (used by the sparse-grid kernels).
void iso_block_scan_launch(unsigned long long* blk, long long nblk, long long* totals, cudaStream_t st) {
    iso::launch_pdl(dc_block_scan, 1u, 1024u, st, blk, nblk, totals);
}

extern "C" {

size_t iso_dc_workspace_size(int nx, int ny, int nz) {
    if (nx < 2 || ny < 2 || nz < 2) return 256;
    const long long NWg = (nz + 31) / 32, NWc = (nz - 1 + 31) / 32;
    const long long cwords = (long long)(nx - 1) * (ny - 1) * NWc;
    const long long pwords = (long long)nx * ny * NWg;
    const long long nblk = (std::max(cwords, pwords) + DC_BLOCK - 1) / DC_BLOCK;
    size_t o = 0;
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    o = al(o + size_t(pwords) * 4);       // signs
    o = al(o + size_t(std::max(cwords, pwords)) * 4);  // active masks (by cell word, or by point word)
    o = al(o + size_t(std::max(cwords, pwords)) * 4);  // active prefixes
    o = al(o + size_t(nblk) * 16);        // cell block sums
    o = al(o + size_t(nblk) * 16);        // quad block sums
    return o + 1024;
}

}  // extern "C"

namespace {
struct DcWs {
    uint32_t *S, *actm, *offA;
    unsigned long long *blkC, *blkQ;
    long long cwords, pwords, nblkC, nblkQ;
};
DcWs carve(void* ws, int nx, int ny, int nz) {
    DcWs w;
    const long long NWg = (nz + 31) / 32, NWc = (nz - 1 + 31) / 32;
    w.cwords = (long long)(nx - 1) * (ny - 1) * NWc;
    w.pwords = (long long)nx * ny * NWg;
    w.nblkC = (w.cwords + DC_BLOCK - 1) / DC_BLOCK;
    w.nblkQ = (w.pwords + DC_BLOCK - 1) / DC_BLOCK;
    const long long nblk = std::max(w.nblkC, w.nblkQ);
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    uint8_t* b = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~uintptr_t(255));
    size_t o = 0;
    w.S = reinterpret_cast<uint32_t*>(b + o);    o = al(o + size_t(w.pwords) * 4);
    const size_t nmask = size_t(std::max(w.cwords, w.pwords));
    w.actm = reinterpret_cast<uint32_t*>(b + o); o = al(o + nmask * 4);
    w.offA = reinterpret_cast<uint32_t*>(b + o); o = al(o + nmask * 4);
    w.blkC = reinterpret_cast<unsigned long long*>(b + o); o = al(o + size_t(nblk) * 16);
    w.blkQ = reinterpret_cast<unsigned long long*>(b + o);
    return w;
}
}  // namespace

extern "C" {

int iso_dc_classify(const float* values, int nx, int ny, int nz, float level, void* ws, size_t ws_bytes,
                    long long* counts, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (nx < 2 || ny < 2 || nz < 2) return cudaMemsetAsync(counts, 0, 16, st) == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
    if (ws_bytes < iso_dc_workspace_size(nx, ny, nz)) return iso::fail_code(ISO_ERR_WORKSPACE);
    DcWs w = carve(ws, nx, ny, nz);
    const float amin[3] = {0, 0, 0}, amax[3] = {1, 1, 1};
    Grid3 g = make_grid(nx, ny, nz, amin, amax);
    {
        iso::ProfScope ps("mc_signs", st);
        mc_signs_launch(values, nx, ny, nz, level, w.S, st);
    }
    iso::ProfScope ps("dc_classify", st, 2);
    dc_cell_count<<<blocks_for(w.cwords, DC_BLOCK), DC_BLOCK, 0, st>>>(w.S, g, w.cwords, w.blkC);
    dc_block_scan<<<1, 1024, 0, st>>>(w.blkC, w.nblkC, counts);
    return cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
}

int iso_dc_intersect(const float* values, int nx, int ny, int nz, const float* aabb_min,
                     const float* aabb_max, float level, void* ws, long long A, long long K, float* points,
                     float* normals, int* cell_ids, int* cell_offsets, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (nx < 2 || ny < 2 || nz < 2) return 0;
    DcWs w = carve(ws, nx, ny, nz);
    Grid3 g = make_grid(nx, ny, nz, aabb_min, aabb_max);
    iso::ProfScope ps("dc_intersect", st, A > 0 && points ? 2 : 1);
    dc_intersect<<<blocks_for(w.cwords, DC_BLOCK), DC_BLOCK, 0, st>>>(
        w.S, g, w.cwords, w.blkC, w.actm, w.offA, reinterpret_cast<uint32_t*>(cell_ids),
        reinterpret_cast<uint32_t*>(cell_offsets), A, K);
    if (A == 0 && cell_offsets) cudaMemsetAsync(cell_offsets, 0, 4, st);
    if (A > 0 && points) {
        const int bt = iso::tune_get(iso::TUNE_DC_CELL_THREADS);  // read once: another thread may set it meanwhile
        dc_points<<<blocks_for(A, bt), bt, 0, st>>>(values, g, level, reinterpret_cast<uint32_t*>(cell_ids),
                                                    reinterpret_cast<uint32_t*>(cell_offsets), A, points, normals);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
}

// Active cells, their crossing offsets and the dual vertices, without writing
// crossing points or normals (dual_contouring without a caller intersection).
int iso_dc_intersect_solve(const float* values, int nx, int ny, int nz, const float* aabb_min,
                           const float* aabb_max, float level, void* ws, long long A, long long K,
                           int* cell_ids, int* cell_offsets, float reg, float svd_tol, float* dual, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (nx < 2 || ny < 2 || nz < 2 || A <= 0) return 0;
    if (!cell_ids || !cell_offsets || !dual) return iso::fail_code(ISO_ERR_ARG);
    DcWs w = carve(ws, nx, ny, nz);
    Grid3 g = make_grid(nx, ny, nz, aabb_min, aabb_max);
    {
        iso::ProfScope ps("dc_intersect", st);
        dc_intersect<<<blocks_for(w.cwords, DC_BLOCK), DC_BLOCK, 0, st>>>(
            w.S, g, w.cwords, w.blkC, w.actm, w.offA, reinterpret_cast<uint32_t*>(cell_ids),
            reinterpret_cast<uint32_t*>(cell_offsets), A, K);
    }
    iso::ProfScope ps("dc_solve", st);
    const int bt = iso::tune_get(iso::TUNE_DC_CELL_THREADS);
    solve_kernel(g)<<<blocks_for(A, bt), bt, 0, st>>>(values, g, level, reinterpret_cast<uint32_t*>(cell_ids), A, reg,
                                                    svd_tol, dual);
    return cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
}

int iso_dc_normals(const float* values, int nx, int ny, int nz, const float* aabb_min,
                   const float* aabb_max, const float* points, const int* cell_ids,
                   const int* cell_offsets, long long A, float* normals, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (A <= 0) return 0;
    Grid3 g = make_grid(nx, ny, nz, aabb_min, aabb_max);
    iso::ProfScope ps("dc_normals", st);
    dc_normals<<<blocks_for(A, 256), 256, 0, st>>>(values, g, points,
                                                   reinterpret_cast<const uint32_t*>(cell_ids),
                                                   reinterpret_cast<const uint32_t*>(cell_offsets), A,
                                                   normals);
    return cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
}

int iso_dc_solve(int nx, int ny, int nz, const float* aabb_min, const float* aabb_max, const float* points,
                 const float* normals, const int* cell_ids, const int* cell_offsets, long long A, float reg,
                 float svd_tol, float* dual, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (A <= 0) return 0;
    Grid3 g = make_grid(nx, ny, nz, aabb_min, aabb_max);
    iso::ProfScope ps("dc_solve", st);
    const int bt = iso::tune_get(iso::TUNE_DC_CELL_THREADS);
    dc_solve<<<blocks_for(A, bt), bt, 0, st>>>(points, normals, reinterpret_cast<const uint32_t*>(cell_ids),
                                                 reinterpret_cast<const uint32_t*>(cell_offsets), A, g, reg,
                                                 svd_tol, dual);
    return cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
}

// Active masks and prefixes only (when the intersection was made earlier).
int iso_dc_cells(const float* values, int nx, int ny, int nz, float level, void* ws, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (nx < 2 || ny < 2 || nz < 2) return 0;
    DcWs w = carve(ws, nx, ny, nz);
    const float amin[3] = {0, 0, 0}, amax[3] = {1, 1, 1};
    Grid3 g = make_grid(nx, ny, nz, amin, amax);
    iso::ProfScope ps("dc_intersect", st);
    dc_intersect<<<blocks_for(w.cwords, DC_BLOCK), DC_BLOCK, 0, st>>>(
        w.S, g, w.cwords, w.blkC, w.actm, w.offA, nullptr, nullptr, -1, 0);
    return cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
}

int iso_dc_quads_count(int nx, int ny, int nz, void* ws, long long* counts, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (nx < 2 || ny < 2 || nz < 2) return cudaMemsetAsync(counts, 0, 16, st) == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
    DcWs w = carve(ws, nx, ny, nz);
    const float amin[3] = {0, 0, 0}, amax[3] = {1, 1, 1};
    Grid3 g = make_grid(nx, ny, nz, amin, amax);
    iso::ProfScope ps("dc_quads", st, 2);
    dc_quad_count<<<blocks_for(w.pwords, DC_BLOCK), DC_BLOCK, 0, st>>>(w.S, g, w.pwords, w.blkQ);
    dc_block_scan<<<1, 1024, 0, st>>>(w.blkQ, w.nblkQ, counts);
    return cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
}

int iso_dc_quads_emit(int nx, int ny, int nz, void* ws, const float* dual, int* tri, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (nx < 2 || ny < 2 || nz < 2) return 0;
    DcWs w = carve(ws, nx, ny, nz);
    const float amin[3] = {0, 0, 0}, amax[3] = {1, 1, 1};
    Grid3 g = make_grid(nx, ny, nz, amin, amax);
    iso::ProfScope ps("dc_quads", st);
    dc_quad_emit<<<blocks_for(w.pwords, DC_BLOCK), DC_BLOCK, 0, st>>>(w.S, g, w.pwords, w.blkQ, w.actm,
                                                                     w.offA, dual, tri);
    return cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
}

size_t iso_dc_weld_workspace_size(long long A) {
    uint32_t cap = 1024;
    while ((long long)cap < 2 * A + 1024) cap <<= 1;
    const long long nblk = (A + DC_BLOCK - 1) / DC_BLOCK + 1;
    return size_t(A) * 12 + size_t(cap) * 4 + size_t(nblk) * 16 + 4096;
}

// Weld step 1: used marks, hash, representatives; counts[0] <- V.
int iso_dc_weld_count(const float* dual, long long A, const int* tri, long long ntri, void* ws,
                      size_t ws_bytes, long long* counts, int* status, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (ws_bytes < iso_dc_weld_workspace_size(A)) return iso::fail_code(ISO_ERR_WORKSPACE);
    uint32_t cap = 1024;
    while ((long long)cap < 2 * A + 1024) cap <<= 1;
    uint8_t* b = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~uintptr_t(255));
    uint32_t* used = reinterpret_cast<uint32_t*>(b);
    uint32_t* rep = used + A;
    uint32_t* newidx = rep + A;
    uint32_t* table = newidx + A;
    unsigned long long* blk = reinterpret_cast<unsigned long long*>(
        (reinterpret_cast<uintptr_t>(table + cap) + 15) & ~uintptr_t(15));
    const long long nblk = (A + DC_BLOCK - 1) / DC_BLOCK;
    iso::ProfScope ps("dc_weld", st, (ntri > 0 ? 1 : 0) + (A > 0 ? 4 : 0));
    cudaMemsetAsync(used, 0, size_t(A) * 4, st);
    cudaMemsetAsync(table, 0xff, size_t(cap) * 4, st);
    if (ntri > 0) dc_mark_used<<<blocks_for(ntri, 256), 256, 0, st>>>(tri, ntri, used);
    if (A > 0) {
        dc_hash_insert<<<blocks_for(A, 256), 256, 0, st>>>(dual, used, A, table, cap - 1, status);
        dc_hash_lookup<<<blocks_for(A, 256), 256, 0, st>>>(dual, used, A, table, cap - 1, rep);
        dc_rep_count<<<unsigned(nblk), DC_BLOCK, 0, st>>>(rep, A, blk);
        dc_block_scan<<<1, 1024, 0, st>>>(blk, nblk, counts);
    } else {
        cudaMemsetAsync(counts, 0, 16, st);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
}

// Weld step 2: write vertices [V, 3] and faces [ntri / 3, 3]; vertex_source
// (optional, [V]) receives the dual vertex (active cell) each vertex came from.
int iso_dc_weld_write_src(const float* dual, long long A, const int* tri, long long ntri, void* ws,
                          float* vout, int* fout, int* vertex_source, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    uint32_t cap = 1024;
    while ((long long)cap < 2 * A + 1024) cap <<= 1;
    uint8_t* b = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~uintptr_t(255));
    uint32_t* used = reinterpret_cast<uint32_t*>(b);
    uint32_t* rep = used + A;
    uint32_t* newidx = rep + A;
    uint32_t* table = newidx + A;
    unsigned long long* blk = reinterpret_cast<unsigned long long*>(
        (reinterpret_cast<uintptr_t>(table + cap) + 15) & ~uintptr_t(15));
    const long long nblk = (A + DC_BLOCK - 1) / DC_BLOCK;
    iso::ProfScope ps("dc_weld", st, (A > 0 ? 1 : 0) + (ntri > 0 ? 1 : 0));
    if (A > 0)
        dc_rep_write<<<unsigned(nblk), DC_BLOCK, 0, st>>>(rep, A, blk, dual, newidx, vout,
                                                           reinterpret_cast<uint32_t*>(vertex_source));
    if (ntri > 0) dc_remap<<<blocks_for(ntri, 256), 256, 0, st>>>(tri, ntri, rep, newidx, fout);
    return cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
}

int iso_dc_weld_write(const float* dual, long long A, const int* tri, long long ntri, void* ws,
                      float* vout, int* fout, void* stream) {
    return iso_dc_weld_write_src(dual, A, tri, ntri, ws, vout, fout, nullptr, stream);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// One call, no host synchronisation: for stream capture and for callers that
// size their buffers once.  Capacities: vertex_capacity bounds the active cells
// (dual vertices before the weld, A >= V), face_capacity the faces (2 per quad).

namespace {
struct DcDenseWs {
    DcWs d;
    unsigned long long* zero;  // cleared by the sign pass
    long long nzero;
    long long* misc;           // [0..1] V  [2..3] dc_cells: entries, CTAs done  [4..7] eff  [8..12] counts [13] status when the caller has none  [14] numbering ticket  [15] vertices on faces
    unsigned long long* wblk;  // weld: look-back states per NUM_TILE cells (room for two words each)
    uint4* seg;                // dc_cells: a record per segment (of 256 point words at least)
    uint32_t *cells, *qoff, *vmap;
    uint8_t *used, *qbits;
    float* dual;
    float* gc;  // grid coordinates, x then y then z
    size_t total;
};

DcDenseWs carve_dense(void* ws, int nx, int ny, int nz, long long capA) {
    DcDenseWs w{};
    const size_t base = iso_dc_workspace_size(nx, ny, nz);
    uint8_t* b = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~uintptr_t(255));
    if (ws) w.d = carve(b, nx, ny, nz);
    const long long pwords = (long long)nx * ny * ((nz + 31) / 32);
    const long long n2048 = (pwords + 2047) / 2048;
    const long long ntV = (capA + NUM_TILE - 1) / NUM_TILE;
    size_t o = (base + 255) & ~size_t(255);
    auto take = [&](size_t bytes) {
        uint8_t* p = ws ? b + o : nullptr;
        o = (o + std::max<size_t>(bytes, 1) + 255) & ~size_t(255);
        return p;
    };
    w.nzero = 16;
    w.zero = reinterpret_cast<unsigned long long*>(take(size_t(w.nzero) * 8));
    w.misc = reinterpret_cast<long long*>(w.zero);
    w.wblk = reinterpret_cast<unsigned long long*>(take(size_t(ntV + 1) * 16));
    w.seg = reinterpret_cast<uint4*>(take(size_t(n2048) * 128));
    take(size_t(n2048) * 16);  // (the workspace's size is as it was)
    w.cells = reinterpret_cast<uint32_t*>(take(size_t(capA) * 4));
    w.qoff = reinterpret_cast<uint32_t*>(take(size_t(capA) * 4));
    w.vmap = reinterpret_cast<uint32_t*>(take(size_t(capA) * 4));
    w.used = take(size_t(capA));
    w.qbits = take(size_t(capA));
    w.dual = reinterpret_cast<float*>(take(size_t(capA) * 12));
    w.gc = reinterpret_cast<float*>(take(size_t(nx + ny + nz) * 4));
    w.total = o + 256;
    return w;
}

CellIndex cell_index(const DcDenseWs& w, const Grid3& g, unsigned long long* elist) {
    // the crossings' offsets of the entries live in vmap until the weld writes it
    return CellIndex{pw_grid(g), w.d.actm, w.d.offA, w.seg, elist, w.vmap};
}
}  // namespace

static int dc_dense_impl(const float* values, int nx, int ny, int nz, const float* aabb_min, const float* aabb_max,
                         float level, float reg, float svd_tol, float* vertices, long long vertex_capacity, int* faces,
                         long long face_capacity, void* workspace, size_t workspace_bytes, long long* counts,
                         int* status, int* cell_ids, int* cell_offsets, int* vertex_source, iso::HostSizes* host,
                         const Given* given, void* stream);

extern "C" {

size_t iso_dc_dense_workspace_size(int nx, int ny, int nz, long long vertex_capacity, long long face_capacity) {
    if (nx < 2 || ny < 2 || nz < 2) return 256;
    if (vertex_capacity < 0 || face_capacity < 0) return 0;
    return carve_dense(nullptr, nx, ny, nz, vertex_capacity).total;
}

int iso_dc_dense_ex(const float* values, int nx, int ny, int nz, const float* aabb_min, const float* aabb_max,
                    float level, float reg, float svd_tol, float* vertices, long long vertex_capacity, int* faces,
                    long long face_capacity, void* workspace, size_t workspace_bytes, long long* counts, int* status,
                    int* cell_ids, int* cell_offsets, int* vertex_source, void* stream) {
    return dc_dense_impl(values, nx, ny, nz, aabb_min, aabb_max, level, reg, svd_tol, vertices, vertex_capacity, faces,
                         face_capacity, workspace, workspace_bytes, counts, status, cell_ids, cell_offsets,
                         vertex_source, nullptr, nullptr, stream);
}

int iso_dc_dense_sync(const float* values, int nx, int ny, int nz, const float* aabb_min, const float* aabb_max,
                      float level, float reg, float svd_tol, float* vertices, long long vertex_capacity, int* faces,
                      long long face_capacity, void* workspace, size_t workspace_bytes, long long* sizes,
                      void* stream) {
    if (!sizes || vertex_capacity < 1) return iso::fail_code(ISO_ERR_ARG);
    iso::HostSizes host;
    const int rc = dc_dense_impl(values, nx, ny, nz, aabb_min, aabb_max, level, reg, svd_tol, vertices,
                                 vertex_capacity, faces, face_capacity, workspace, workspace_bytes, nullptr, nullptr,
                                 nullptr, nullptr, nullptr, &host, nullptr, stream);
    return host.wait(rc, 6, sizes, reinterpret_cast<cudaStream_t>(stream));
}

int iso_dc_dense_its_sync(const float* values, int nx, int ny, int nz, const float* aabb_min, const float* aabb_max,
                          float level, float reg, float svd_tol, const float* points, const float* normals,
                          const int* cell_ids, const int* cell_offsets, long long A, float* vertices, int* faces,
                          long long face_capacity, void* workspace, size_t workspace_bytes, long long* sizes,
                          void* stream) {
    if (!sizes || A < 1 || !points || !cell_ids || !cell_offsets) return iso::fail_code(ISO_ERR_ARG);
    iso::HostSizes host;
    const Given in{points, normals, reinterpret_cast<const uint32_t*>(cell_ids),
                   reinterpret_cast<const uint32_t*>(cell_offsets), A, nullptr};
    const int rc = dc_dense_impl(values, nx, ny, nz, aabb_min, aabb_max, level, reg, svd_tol, vertices, A, faces,
                                 face_capacity, workspace, workspace_bytes, nullptr, nullptr, nullptr, nullptr, nullptr,
                                 &host, &in, stream);
    return host.wait(rc, 6, sizes, reinterpret_cast<cudaStream_t>(stream));
}

int iso_dc_intersection_sync(const float* values, int nx, int ny, int nz, const float* aabb_min, const float* aabb_max,
                             float level, float* points, float* normals, long long point_capacity, int* cell_ids,
                             int* cell_offsets, long long cell_capacity, void* workspace, size_t workspace_bytes,
                             long long* sizes, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (!sizes || !aabb_min || !aabb_max || cell_capacity < 1 || point_capacity < 1 || nx < 2 || ny < 2 || nz < 2 ||
        (long long)nx * ny * nz > 0x7fffffffll || !values || !points || !cell_ids || !cell_offsets)
        return iso::fail_code(ISO_ERR_ARG);
    if (workspace_bytes < iso_dc_dense_workspace_size(nx, ny, nz, cell_capacity, 0)) return iso::fail_code(ISO_ERR_WORKSPACE);
    iso::HostSizes host;
    long long* const words = host.lease();
    if (!words) return ISO_ERR_CUDA;
    const DcDenseWs w = carve_dense(workspace, nx, ny, nz, cell_capacity);
    const Grid3 g = make_grid(nx, ny, nz, aabb_min, aabb_max);
    long long *eff = w.misc + 4, *counts = w.misc + 8;
    int* status = reinterpret_cast<int*>(w.misc + 13);
    uint32_t *cells = reinterpret_cast<uint32_t*>(cell_ids), *off = reinterpret_cast<uint32_t*>(cell_offsets);
    const CellIndex ix = cell_index(w, g, reinterpret_cast<unsigned long long*>(w.dual));
    {
        iso::ProfScope ps("mc_signs", st);
        mc_signs_launch(values, nx, ny, nz, level, w.d.S, st, w.zero, w.nzero);
    }
    {
        iso::ProfScope ps("dc_classify", st, ix.p.nseg > CELLS_SCAN ? 2 : 1);
        const CellsOut co{w.zero + 2, cell_capacity, 0x7fffffffll, point_capacity, eff, counts, off, status, w.gc,
                          nullptr, 0};
        launch_cells(w.d.S, g, ix, co, st);
    }
    {
        iso::ProfScope ps("dc_intersect", st);
        const int bt = iso::tune_get(iso::TUNE_DC_CELL_THREADS);
        iso::launch_pdl(dc_entry_points, blocks_for(cell_capacity, bt), unsigned(bt), st, values, g, level, ix,
                        static_cast<const long long*>(eff), static_cast<const float*>(w.gc), cells, off, points,
                        normals, static_cast<const long long*>(counts), static_cast<const int*>(status),
                        words);
    }
    const int rc = cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
    return host.wait(rc, 6, sizes, st);
}

int iso_dc_dense(const float* values, int nx, int ny, int nz, const float* aabb_min, const float* aabb_max,
                 float level, float reg, float svd_tol, float* vertices, long long vertex_capacity, int* faces,
                 long long face_capacity, void* workspace, size_t workspace_bytes, long long* counts, int* status,
                 void* stream) {
    return iso_dc_dense_ex(values, nx, ny, nz, aabb_min, aabb_max, level, reg, svd_tol, vertices, vertex_capacity,
                           faces, face_capacity, workspace, workspace_bytes, counts, status, nullptr, nullptr, nullptr,
                           stream);
}

}  // extern "C"

static int dc_dense_impl(const float* values, int nx, int ny, int nz, const float* aabb_min, const float* aabb_max,
                         float level, float reg, float svd_tol, float* vertices, long long vertex_capacity, int* faces,
                         long long face_capacity, void* workspace, size_t workspace_bytes, long long* counts,
                         int* status, int* cell_ids, int* cell_offsets, int* vertex_source, iso::HostSizes* host,
                         const Given* given, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (((!counts || !status) && !host) || !aabb_min || !aabb_max || vertex_capacity < 0 || face_capacity < 0) return iso::fail_code(ISO_ERR_ARG);
    if ((long long)nx * ny * nz > 0x7fffffffll) return iso::fail_code(ISO_ERR_ARG);
    if (host && (nx < 2 || ny < 2 || nz < 2)) return 0;  // the sizes are 0
    if (nx < 2 || ny < 2 || nz < 2)
        return cudaMemsetAsync(counts, 0, 5 * sizeof(long long), st) == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
    if (!values || (vertex_capacity && !vertices) || (face_capacity && !faces)) return iso::fail_code(ISO_ERR_ARG);
    // without a caller's intersection 6 Q face indices stay below 2^31
    const long long capA = vertex_capacity,
                    capQ = given ? face_capacity / 2 : std::min(face_capacity / 2, 0x7ffffffell / 6);
    if (workspace_bytes < iso_dc_dense_workspace_size(nx, ny, nz, vertex_capacity, face_capacity))
        return iso::fail_code(ISO_ERR_WORKSPACE);
    long long* const words = host ? host->lease() : nullptr;
    if (host && !words) return ISO_ERR_CUDA;
    const DcDenseWs w = carve_dense(workspace, nx, ny, nz, capA);
    const Grid3 g = make_grid(nx, ny, nz, aabb_min, aabb_max);
    long long* eff = w.misc + 4;
    if (!counts) counts = w.misc + 8;  // cleared by the sign pass
    if (!status) status = reinterpret_cast<int*>(w.misc + 13);
    uint32_t* cells = cell_ids ? reinterpret_cast<uint32_t*>(cell_ids) : w.cells;
    {
        iso::ProfScope ps("mc_signs", st);
        mc_signs_launch(values, nx, ny, nz, level, w.d.S, st, w.zero, w.nzero);
    }
    // the entries live in the vertex buffer until the weld writes it
    const CellIndex ix = cell_index(w, g, reinterpret_cast<unsigned long long*>(
                                              (reinterpret_cast<uintptr_t>(vertices) + 7) & ~uintptr_t(7)));
    const CellsOut co{w.zero + 2, capA, capQ, 0x7fffffffll, eff, counts, reinterpret_cast<uint32_t*>(cell_offsets),
                      status, w.gc, w.wblk, (capA + NUM_TILE - 1) / NUM_TILE};
    {
        iso::ProfScope ps("dc_classify", st, ix.p.nseg > CELLS_SCAN ? 2 : 1);
        launch_cells(w.d.S, g, ix, co, st);
    }
    if (capA > 0) {
        // the list of vertices on faces follows the entries: room for all cells but at most one
        const FaceList list{reinterpret_cast<uint32_t*>(ix.elist + capA), w.zero + 15,
                            (reinterpret_cast<float*>(vertices) + 3 * capA) -
                                reinterpret_cast<float*>(ix.elist + capA)};
        {
            iso::ProfScope ps("dc_solve", st);
            const int bt = iso::tune_get(iso::TUNE_DC_CELL_THREADS);
            const SolveOut so{cells, w.qoff, w.qbits, w.used, w.dual, co.cell_off, list.cells, list.n, list.cap};
            const auto kernel = given ? (g.fma ? dc_solve_cells<true, true> : dc_solve_cells<false, true>)
                                      : (g.fma ? dc_solve_cells<true, false> : dc_solve_cells<false, false>);
            Given in = given ? *given : Given{};
            in.status = status;
            iso::launch_pdl(kernel, blocks_for(capA, bt), unsigned(bt), st, values, g, level, ix, reg, svd_tol,
                            static_cast<const long long*>(eff), static_cast<const float*>(w.gc), so, in);
        }
        {
            // the table, where one is needed, takes the place of the entries, which the solve was the last to read
            const bool hash = coords_may_repeat(g);
            const WeldTable table{hash ? reinterpret_cast<uint32_t*>(ix.elist) : nullptr, weld_table_size(capA)};
            iso::ProfScope ps("dc_weld", st, hash ? 3 : 2);
            if (hash && launch_weld_table(table, w.dual, w.used, 3u, nullptr, eff, capA, st) != cudaSuccess)
                return iso::fail_code(ISO_ERR_CUDA);
            const uint32_t* cc = cells;
            // (a few percent of the vertices lie on faces)
            iso::launch_pdl(dc_weld_faces, std::min(blocks_for(capA, 16), 16u * unsigned(iso::sm_count())), 128u, st, g, ix,
                            static_cast<const float*>(w.gc), list, cc, w.used, static_cast<const float*>(w.dual),
                            static_cast<const long long*>(eff), w.vmap, table);
            iso::launch_pdl(dc_weld_number, blocks_for(capA, NUM_TILE), unsigned(NUM_THREADS), st,
                            static_cast<const float*>(w.dual), static_cast<const long long*>(eff),
                            static_cast<const uint8_t*>(w.used), w.wblk, w.zero + 14, w.vmap, vertices,
                            reinterpret_cast<uint32_t*>(vertex_source), counts, status);
        }
        {
            iso::ProfScope ps("dc_quads", st);
            iso::launch_pdl(dc_cell_quads, blocks_for(capA, 256), 256u, st, static_cast<const uint8_t*>(w.qbits), g,
                            static_cast<const uint32_t*>(cells), static_cast<const uint32_t*>(w.qoff), ix,
                            static_cast<const float*>(w.dual), static_cast<const uint32_t*>(w.vmap),
                            static_cast<const long long*>(eff), faces, static_cast<const long long*>(counts),
                            static_cast<const int*>(status), words);
        }
    }
    return cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
}
