// Sparse dual contouring in one call, sizes kept on the device (isoext's
// dual_contouring of a SparseGrid without a caller intersection:
// src/grid/sparse.cu:181-246 for the quads, src/its.cu:37-90 and 186-268 for the
// crossings and normals, src/dc.cu:14-218 for the solve, split and weld).
//
//   sd_classify   the active cells (corners on both sides of the level) compacted
//                 in id order: sparse index, lattice id and case.  The only pass
//                 over all values, tiles chained by look-back.
//   sd_solve      per active cell: crossings, grid normals and the QEF, nothing
//                 of them stored.
//   sd_quads      per active cell: the cells around its three low edges, found in
//                 the list of active cells; which of the edges have a quad, and
//                 which cells a quad uses.
//   sd_flags      which dual vertices are representatives of their position.  A
//                 vertex is clipped to its cell's box, so only one on a face of
//                 the box can equal another cell's (see dc_dense.cu).
//                 Its last CTA scans the blocks' quads and representatives.
//   sd_number     vertices in cell order.
//   sd_faces      the quads as two triangles each.
//
// A quad needs its four cells active, its owner (the cell at the low end of its
// edge) among them, so everything past the first pass works on the active cells,
// about a tenth of a band's.  The search that this replaces looked for the three
// neighbours of every cell's three edges among all ids, twice (count and emit):
// 870 us of the 1130 us of a 200^3 band (2.2 M cells), against 15.
#include <algorithm>
#include <cstdint>

#include "common.cuh"
#define ISO_LUT_DECL static __constant__ const
#include "luts.h"
#include "dc_common.cuh"
#include "lookback.cuh"
#include "profile.cuh"
#include "weld_table.cuh"

// (dc_dense.cu) exclusive scan of pairs of block sums in place, totals -> totals[0..1]
void iso_block_scan_launch(unsigned long long* blk, long long nblk, long long* totals, cudaStream_t st);

namespace {

constexpr int SD_THREADS = 256;
constexpr int SD_ROUNDS = 8;                        // cells per thread of the first pass
constexpr int SD_TILE = SD_THREADS * SD_ROUNDS;     // cells per tile
constexpr int SD_BLOCK = 512;                       // active cells per CTA (and per block sum)

__device__ __forceinline__ uint32_t case8(const float4& a, const float4& b, float level) {
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t cs = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) cs |= (iso::below(v[k], level) ? 1u : 0u) << k;
    return cs;
}

// Bound by HBM (32 bytes per cell): four rounds of two 16-byte loads in flight
// per thread.  One pass with look-back instead of a count and a second read.
__global__ void __launch_bounds__(SD_THREADS, 4) sd_classify(const int* __restrict__ ids,
                                                          const float* __restrict__ vals, uint32_t n, float level,
                                                          unsigned int* ticket, unsigned long long* state,
                                                          uint32_t* __restrict__ act, uint32_t* __restrict__ lat,
                                                          uint8_t* __restrict__ cas, uint8_t* __restrict__ used,
                                                          long long capA, long long* eff, long long* counts,
                                                          int* status) {
    __shared__ uint32_t tile_s, wcnt[SD_ROUNDS][SD_THREADS / 32], wk[SD_THREADS / 32];
    __shared__ unsigned long long pre_s;
    if (threadIdx.x == 0) tile_s = atomicAdd(ticket, 1u);
    __syncthreads();
    const uint32_t tile = tile_s, ntile = (n + SD_TILE - 1) / SD_TILE;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t c0 = tile * SD_TILE + threadIdx.x;
    uint32_t cs4[SD_ROUNDS / 4], nk = 0, on = 0;  // cases; crossings; active rounds
#pragma unroll
    for (int q = 0; q < SD_ROUNDS / 4; ++q) {
        float4 va[4], vb[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t c = c0 + (4 * q + k) * SD_THREADS;
            const float4* v4 = reinterpret_cast<const float4*>(vals) + 2ull * c;
            va[k] = c < n ? __ldg(v4) : make_float4(level, level, level, level);
            vb[k] = c < n ? __ldg(v4 + 1) : make_float4(level, level, level, level);
        }
        cs4[q] = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t cs = case8(va[k], vb[k], level);
            const bool a = cs != 0 && cs != 255;
            if (a) nk += __popc(edge_status(cs));
            cs4[q] |= cs << (8 * k);
            on |= uint32_t(a) << (4 * q + k);
        }
    }
    uint32_t mine = 0;
#pragma unroll
    for (int r = 0; r < SD_ROUNDS; ++r) {
        const uint32_t b = __ballot_sync(~0u, (on >> r) & 1u);
        if (lane == r) mine = __popc(b);
    }
    if (lane < SD_ROUNDS) wcnt[lane][warp] = mine;
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) nk += __shfl_xor_sync(~0u, nk, d);
    if (lane == 0) wk[warp] = nk;
    __syncthreads();
    if (warp == 0) {
        // the (round, warp) counts, PER per lane in order: prefixes and the tile's total
        constexpr int WARPS = SD_THREADS / 32, PER = SD_ROUNDS * WARPS / 32;
        static_assert(PER * 32 == SD_ROUNDS * WARPS && SD_ROUNDS <= 32, "every lane takes PER counts");
        uint32_t s = 0;
#pragma unroll
        for (int k = 0; k < PER; ++k) s += wcnt[(lane * PER + k) / WARPS][(lane * PER + k) % WARPS];
        uint32_t inc = s;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t t = __shfl_up_sync(~0u, inc, d);
            if (lane >= d) inc += t;
        }
        const uint32_t total = __shfl_sync(~0u, inc, 31);
        uint32_t run = inc - s;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            uint32_t& c = wcnt[(lane * PER + k) / WARPS][(lane * PER + k) % WARPS];
            const uint32_t t = c;
            c = run;
            run += t;
        }
        uint32_t ks = lane < SD_THREADS / 32 ? wk[lane] : 0u;
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) ks += __shfl_xor_sync(~0u, ks, d);
        unsigned long long ea = 0, ek = 0;
        lb_tile(state, tile, total, ks, ea, ek, status);
        if (lane == 0) {
            pre_s = ea;
            if (tile == ntile - 1) {
                const long long A = (long long)(ea + total), K = (long long)(ek + ks);
                const bool ok = A <= capA && A < 0x7fffffffll && K < 0x7fffffffll;
                if (!ok) atomicCAS(status, 0, int(ISO_ERR_OVERFLOW));
                eff[0] = ok ? A : 0;
                counts[0] = 0;
                counts[1] = 0;
                counts[2] = A;
                counts[3] = K;
                counts[4] = 0;
            }
        }
    }
    __syncthreads();
    const unsigned long long base = pre_s;
#pragma unroll
    for (int r = 0; r < SD_ROUNDS; ++r) {
        const uint32_t b = __ballot_sync(~0u, (on >> r) & 1u);
        if (!((on >> r) & 1u)) continue;
        const unsigned long long a = base + wcnt[r][warp] + __popc(b & ((1u << lane) - 1u));
        if ((long long)a >= capA) continue;
        const uint32_t c = c0 + r * SD_THREADS;
        act[a] = c;
        lat[a] = uint32_t(__ldg(ids + c));
        cas[a] = uint8_t(cs4[r >> 2] >> (8 * (r & 3)));
        used[a] = 0;
    }
}

__device__ __forceinline__ void lat_xyz(const Grid3& g, uint32_t id, int& x, int& y, int& z) {
    z = int(id % uint32_t(g.nz - 1));
    const uint32_t r = id / uint32_t(g.nz - 1);
    y = int(r % uint32_t(g.ny - 1));
    x = int(r / uint32_t(g.ny - 1));
}

// The dual vertex of each active cell, the arithmetic of the crossings, normals
// and solve steps in one thread; face: whether it lies on a face of its cell's
// box.  F: the arithmetic reading (g.fma).  Bound by FP32 issue.
template <bool F>
__global__ void __launch_bounds__(128) sd_solve(const float* __restrict__ vals, Grid3 g, float level,
                                                const uint32_t* __restrict__ act, const uint32_t* __restrict__ lat,
                                                const uint8_t* __restrict__ cas, const long long* __restrict__ eff,
                                                float reg, float svd_tol, float* __restrict__ dual,
                                                uint8_t* __restrict__ face) {
    iso::grid_wait();
    const long long a = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= eff[0]) return;
    g.fma = F;
    int x, y, z;
    lat_xyz(g, lat[a], x, y, z);
    CellCorners cc;
    cc.fma = F;
    const float4* v4 = reinterpret_cast<const float4*>(vals) + 2ull * act[a];
    const float4 v0 = __ldg(v4), v1 = __ldg(v4 + 1);
    cc.v[0] = v0.x; cc.v[1] = v0.y; cc.v[2] = v0.z; cc.v[3] = v0.w;
    cc.v[4] = v1.x; cc.v[5] = v1.y; cc.v[6] = v1.z; cc.v[7] = v1.w;
    const float x0 = coord(g, 0, x), x1 = coord(g, 0, x + 1), y0 = coord(g, 1, y), y1 = coord(g, 1, y + 1),
                z0 = coord(g, 2, z), z1 = coord(g, 2, z + 1);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        cc.p[k][0] = (k >> 2) ? x1 : x0;
        cc.p[k][1] = ((k >> 1) & 1) ? y1 : y0;
        cc.p[k][2] = (k & 1) ? z1 : z0;
    }
    Qef Q;
    qef_init(Q, F);
    uint32_t K = 0;
#pragma unroll 1
    for (uint32_t em = edge_status(cas[a]); em; em &= em - 1, ++K) {  // this lane's crossed edges, ascending
        float p[3], nn[3];
        edge_cross(cc, level, __ffs(em) - 1, p);
        cell_normal(cc, p, nn);
        qef_add(Q, p[0], p[1], p[2], nn[0], nn[1], nn[2]);
    }
    qef_finish(Q, K, reg, svd_tol);
    bool on = false;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const float lo = cc.p[0][q], hi = cc.p[7][q];
        const float v = fminf(fmaxf(float(Q.x[q]), lo), hi);
        on |= v == lo || v == hi;
        dual[3 * a + q] = v;
    }
    face[a] = on ? 1 : 0;
}

// First position in lat[lo, hi) whose id is at least key.
__device__ __forceinline__ uint32_t lower(const uint32_t* __restrict__ lat, uint32_t lo, uint32_t hi, uint32_t key) {
    while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (__ldg(lat + mid) < key) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

constexpr uint32_t NONE = 0xffffffffu;

// The active cells at key and at key - 1 (when `below`), with `at` the first
// position whose id is at least key, of `end` positions.
__device__ __forceinline__ void pair_at(const uint32_t* __restrict__ lat, uint32_t at, uint32_t end, uint32_t key,
                                        bool below, uint32_t& here, uint32_t& before) {
    here = at < end && __ldg(lat + at) == key ? at : NONE;
    before = below && at > 0 && __ldg(lat + at - 1) == key - 1u ? at - 1 : NONE;
}

// Sign of cell q's edge from corner a to corner a + step by its case: -1 not
// crossed, else 1 when the low end is below the level.
__device__ __forceinline__ int case_sign(uint32_t cs, int a, int step) {
    const uint32_t lo = (cs >> a) & 1u, hi = (cs >> (a + step)) & 1u;
    return lo == hi ? -1 : int(lo);
}

// Quads that active cell a owns, one per crossed edge at its low corner whose
// other three cells are active too.  qb: bits 0-2 the z, y, x edges with a quad,
// 3-5 their orientation.  nbr: the six cells those quads can use (y-1; y-1, z-1;
// z-1; x-1; x-1, z-1; x-1, y-1), plane by plane.  As in the reference an edge is
// crossed when any of its cells says so, and the first of them in cell order
// gives the orientation (src/grid/sparse.cu:181-246).
__global__ void __launch_bounds__(SD_BLOCK) sd_quads(Grid3 g, const uint32_t* __restrict__ lat,
                                                     const uint8_t* __restrict__ cas,
                                                     const long long* __restrict__ eff, long long capA,
                                                     uint8_t* __restrict__ used, uint8_t* __restrict__ qbits,
                                                     uint32_t* __restrict__ nbr, unsigned long long* blk) {
    __shared__ uint32_t ws[SD_BLOCK / 32];
    iso::grid_wait();
    const uint32_t A = uint32_t(eff[0]);
    const uint32_t a = blockIdx.x * SD_BLOCK + threadIdx.x;
    uint32_t qb = 0;
    if (a < A) {
        const uint32_t id = lat[a];
        int x, y, z;
        lat_xyz(g, id, x, y, z);
        if (x <= g.nx - 2) {  // (ids past the lattice's cells own no quad)
            const uint32_t nzc = uint32_t(g.nz - 1), plane = uint32_t(g.ny - 1) * nzc;
            const uint32_t zb = z > 0;
            uint32_t Y = NONE, YZ = NONE, X = NONE, XZ = NONE, XY = NONE, unused;
            const uint32_t Z = zb && a > 0 && __ldg(lat + a - 1) == id - 1u ? a - 1 : NONE;
            // at most nzc (plane) ids lie between the cell's and its y- (x-)neighbour's
            if (y > 0) pair_at(lat, lower(lat, a > nzc ? a - nzc : 0u, a, id - nzc), a, id - nzc, zb, Y, YZ);
            if (x > 0) {
                const uint32_t px = lower(lat, a > plane ? a - plane : 0u, a, id - plane);
                pair_at(lat, px, a, id - plane, zb, X, XZ);
                if (y > 0)
                    pair_at(lat, lower(lat, px > nzc ? px - nzc : 0u, px, id - plane - nzc), px, id - plane - nzc,
                            false, XY, unused);
            }
            const uint32_t c[4][3] = {{a, a, a}, {Y, Z, X}, {YZ, XZ, XY}, {Z, X, Y}};  // [cell of quad][x, y, z edge]
            // the edge's low corner within each of the four cells (4 dx + 2 dy + dz)
            const int low[4][3] = {{0, 0, 0}, {2, 1, 4}, {3, 5, 6}, {1, 4, 2}};
#pragma unroll
            for (int ax = 0; ax < 3; ++ax) {
                if (c[1][ax] == NONE || c[2][ax] == NONE || c[3][ax] == NONE) continue;
                const int step = ax == 0 ? 4 : (ax == 1 ? 2 : 1);
                uint32_t first = NONE;
                int sign = -1;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int s = case_sign(cas[c[i][ax]], low[i][ax], step);
                    if (s >= 0 && c[i][ax] < first) {
                        first = c[i][ax];
                        sign = s;
                    }
                }
                if (sign < 0) continue;
                qb |= 1u << (2 - ax);
                if (sign == 1) qb |= 8u << (2 - ax);
#pragma unroll
                for (int i = 0; i < 4; ++i) used[c[i][ax]] = 1;
            }
            if (qb & 7u) {
                const uint32_t v[6] = {Y, YZ, Z, X, XZ, XY};
#pragma unroll
                for (int k = 0; k < 6; ++k) nbr[k * capA + a] = v[k];
            }
        }
        qbits[a] = uint8_t(qb);
    }
    uint32_t s = __popc(qb & 7u);
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) s += __shfl_xor_sync(~0u, s, d);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int k = 0; k < SD_BLOCK / 32; ++k) t += ws[k];
        blk[2 * blockIdx.x] = t;
    }
}

// Cells along one axis whose closed interval holds v, in cell c's: c alone, or c
// and the cell on the side where v is the common coordinate (neighbouring
// coordinates are distinct here).
__device__ __forceinline__ void cells_holding(const Grid3& g, int axis, int c, float v, int& i0, int& i1) {
    const int n = axis == 0 ? g.nx : (axis == 1 ? g.ny : g.nz);
    i0 = c - (c > 0 && coord(g, axis, uint32_t(c)) == v ? 1 : 0);
    i1 = c + (c < n - 2 && coord(g, axis, uint32_t(c + 1)) == v ? 1 : 0);
}

// vmap[a] = NONE when no quad uses the cell, 0 when its vertex is a
// representative, else 0x80000000 | its representative, the smallest used cell
// with its position; representatives per block into blk.  Only a vertex on a face
// of its box can have one (face): a CTA lists those and takes each with four
// lanes, a lane per column (x, y) of the cells around the face, edge or corner;
// where coordinates may repeat it reads their table instead (weld_table.cuh).
// Bound by the latency of a column's binary search.  The last CTA turns blk's
// pairs into offsets (scan): 16 us with that for 0.22 M cells, where a thread per
// cell, searching its columns one after another, and the scan's launch took 16 + 5.
constexpr int SD_LANES = 4;                 // at most four columns meet at an edge
constexpr uint32_t SD_SCAN = 2 * SD_BLOCK;  // blocks the last CTA scans, two per thread

__global__ void __launch_bounds__(SD_BLOCK) sd_flags(Grid3 g, const uint32_t* __restrict__ lat,
                                                     const uint8_t* __restrict__ used,
                                                     const uint8_t* __restrict__ face,
                                                     const float* __restrict__ dual,
                                                     const long long* __restrict__ eff, uint32_t* __restrict__ vmap,
                                                     unsigned long long* blk, bool scan, unsigned int* done,
                                                     long long* tot, const WeldTable table) {
    __shared__ uint16_t list[SD_BLOCK];
    __shared__ uint32_t listed, merged;
    __shared__ bool last;
    iso::grid_wait();
    const uint32_t A = uint32_t(eff[0]);
    const uint32_t b0 = blockIdx.x * SD_BLOCK, a0 = b0 + threadIdx.x;
    if (threadIdx.x == 0) { listed = 0; merged = 0; }
    __syncthreads();
    const bool on = a0 < A && used[a0];
    if (a0 < A) vmap[a0] = on ? 0u : NONE;
    if (on && face[a0]) list[atomicAdd(&listed, 1u)] = uint16_t(threadIdx.x);  // in any order
    const uint32_t reps = uint32_t(__syncthreads_count(on));
    const uint32_t k = threadIdx.x % SD_LANES;
    const uint32_t lanes = ((1u << SD_LANES) - 1u) << (threadIdx.x & 31u & ~uint32_t(SD_LANES - 1));
    for (uint32_t i = threadIdx.x / SD_LANES; i < listed; i += SD_BLOCK / SD_LANES) {
        const uint32_t a = b0 + list[i];
        uint32_t first = a;  // cells from a on cannot come before it
        if (table.slot) {
            if (k == 0) first = table_first(table, dual, a);
        } else {
            const float p[3] = {dual[3ll * a], dual[3ll * a + 1], dual[3ll * a + 2]};
            int x, y, z, x0, x1, y0, y1, z0, z1;
            lat_xyz(g, lat[a], x, y, z);
            cells_holding(g, 0, x, p[0], x0, x1);
            cells_holding(g, 1, y, p[1], y0, y1);
            cells_holding(g, 2, z, p[2], z0, z1);
            const uint32_t cy = uint32_t(y1 - y0 + 1), columns = uint32_t(x1 - x0 + 1) * cy;  // at most SD_LANES
            if (k < columns) {
                const uint32_t key = (uint32_t(x0) + k / cy) * uint32_t(g.ny - 1) + uint32_t(y0) + k % cy;
                const uint32_t zend = key * uint32_t(g.nz - 1) + uint32_t(z1);
                for (uint32_t b = lower(lat, 0u, first, key * uint32_t(g.nz - 1) + uint32_t(z0)); b < first && lat[b] <= zend; ++b)
                    if (used[b] && same_position(dual, a, b)) first = b;
            }
        }
#pragma unroll
        for (int d = SD_LANES / 2; d >= 1; d >>= 1) first = min(first, __shfl_xor_sync(lanes, first, d));
        if (k == 0 && first != a) {
            vmap[a] = 0x80000000u | first;
            atomicAdd(&merged, 1u);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        blk[2 * blockIdx.x + 1] = (unsigned long long)(reps - merged);
        if (scan) {
            __threadfence();
            last = atomicAdd(done, 1u) == gridDim.x - 1;
        }
    }
    if (!scan) return;
    __syncthreads();
    if (!last) return;
    __threadfence();
    __shared__ unsigned long long wa[SD_BLOCK / 32], wb[SD_BLOCK / 32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, i0 = 2 * threadIdx.x;
    unsigned long long va[2], vb[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const bool in = i0 + j < gridDim.x;
        va[j] = in ? __ldcg(blk + 2 * (i0 + j)) : 0ull;
        vb[j] = in ? __ldcg(blk + 2 * (i0 + j) + 1) : 0ull;
    }
    unsigned long long ia = va[0] + va[1], ib = vb[0] + vb[1];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long ta = __shfl_up_sync(~0u, ia, d), tb = __shfl_up_sync(~0u, ib, d);
        if (lane >= uint32_t(d)) { ia += ta; ib += tb; }
    }
    if (lane == 31) { wa[warp] = ia; wb[warp] = ib; }
    __syncthreads();
    unsigned long long ea = ia - va[0] - va[1], eb = ib - vb[0] - vb[1];
#pragma unroll
    for (uint32_t q = 0; q < SD_BLOCK / 32; ++q)
        if (q < warp) { ea += wa[q]; eb += wb[q]; }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        if (i0 + j < gridDim.x) { blk[2 * (i0 + j)] = ea; blk[2 * (i0 + j) + 1] = eb; }
        ea += va[j];
        eb += vb[j];
    }
    if (threadIdx.x == SD_BLOCK - 1) { tot[0] = (long long)ea; tot[1] = (long long)eb; }
}

// Exclusive position of `mine` items of each thread within the CTA.
__device__ __forceinline__ uint32_t block_before(uint32_t mine, uint32_t* ws) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(~0u, inc, d);
        if (lane >= d) inc += t;
    }
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    uint32_t e = inc - mine;
#pragma unroll
    for (int q = 0; q < SD_BLOCK / 32; ++q) e += q < warp ? ws[q] : 0u;
    return e;
}

// Representatives numbered in cell order (offsets from the scan); the sizes.
__global__ void __launch_bounds__(SD_BLOCK) sd_number(const float* __restrict__ dual,
                                                      const long long* __restrict__ eff,
                                                      const unsigned long long* __restrict__ blk,
                                                      const long long* __restrict__ tot, long long capF,
                                                      uint32_t* __restrict__ vmap, float* __restrict__ vout,
                                                      long long* counts, int* status) {
    __shared__ uint32_t ws[SD_BLOCK / 32];
    iso::grid_wait();
    const uint32_t A = uint32_t(eff[0]);
    const uint32_t a = blockIdx.x * SD_BLOCK + threadIdx.x;
    const bool is = a < A && vmap[a] == 0u;
    const uint32_t e = block_before(is ? 1u : 0u, ws);
    if (blockIdx.x == 0 && threadIdx.x == 0 && A) {
        const long long Q = tot[0];
        if (2 * Q > capF) atomicCAS(status, 0, int(ISO_ERR_OVERFLOW));
        counts[0] = tot[1];
        counts[1] = 2 * Q;
        counts[4] = Q;
    }
    if (!is) return;
    const unsigned long long o = blk[2 * blockIdx.x + 1] + e;  // < V <= A: inside the vertex capacity
    vmap[a] = uint32_t(o);
    vout[3 * o] = dual[3ll * a];
    vout[3 * o + 1] = dual[3ll * a + 1];
    vout[3 * o + 2] = dual[3ll * a + 2];
}

__device__ __forceinline__ int32_t vertex_of(const uint32_t* vmap, uint32_t i) {
    uint32_t m = vmap[i];
    if (m & 0x80000000u) m = vmap[m & 0x7fffffffu];
    return int32_t(m);
}

// The quads in owner order, z, y, x edge within an owner, split along the shorter
// diagonal (src/dc.cu:101-157).
__global__ void __launch_bounds__(SD_BLOCK) sd_faces(Grid3 g, const uint8_t* __restrict__ qbits,
                                                     const uint32_t* __restrict__ nbr, long long capA,
                                                     const float* __restrict__ dual,
                                                     const uint32_t* __restrict__ vmap,
                                                     const long long* __restrict__ eff,
                                                     const unsigned long long* __restrict__ blk,
                                                     const long long* __restrict__ tot, long long capF,
                                                     int32_t* __restrict__ faces,
                                                     const long long* __restrict__ counts,
                                                     const int* __restrict__ status, long long* host) {
    __shared__ uint32_t ws[SD_BLOCK / 32];
    iso::grid_wait();
    if (host && blockIdx.x == 0 && threadIdx.x == 0) {  // the sizes and the status for the host
        for (int k = 0; k < 5; ++k) host[k] = counts[k];
        host[5] = *status;
    }
    const uint32_t A = uint32_t(eff[0]);
    if (2 * tot[0] > capF) return;
    const uint32_t a = blockIdx.x * SD_BLOCK + threadIdx.x;
    const uint32_t qb = a < A ? qbits[a] : 0u;
    const uint32_t e = block_before(__popc(qb & 7u), ws);
    if (!(qb & 7u)) return;
    unsigned long long q = blk[2 * blockIdx.x] + e;
    uint32_t nb[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) nb[k] = nbr[k * capA + a];
    const uint32_t Y = nb[0], YZ = nb[1], Z = nb[2], X = nb[3], XZ = nb[4], XY = nb[5];
    const uint32_t c[3][3] = {{Y, Z, X}, {YZ, XZ, XY}, {Z, X, Y}};  // [cell 1..3 of quad][x, y, z edge]
#pragma unroll
    for (int ax = 2; ax >= 0; --ax) {
        if (!((qb >> (2 - ax)) & 1u)) continue;
        uint32_t qi[4] = {a, c[0][ax], c[1][ax], c[2][ax]};
        if (!((qb >> (5 - ax)) & 1u)) {
            const uint32_t t0 = qi[0], t1 = qi[1];
            qi[0] = qi[3]; qi[1] = qi[2]; qi[2] = t1; qi[3] = t0;
        }
        float v[4][3];
        int32_t f[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
#pragma unroll
            for (int d = 0; d < 3; ++d) v[t][d] = dual[3ll * qi[t] + d];
            f[t] = vertex_of(vmap, qi[t]);
        }
        int32_t* o6 = faces + 6 * q;
        if (dist3(v[0], v[2], g.fma) > dist3(v[1], v[3], g.fma)) {
            o6[0] = f[1]; o6[1] = f[3]; o6[2] = f[0];
            o6[3] = f[3]; o6[4] = f[1]; o6[5] = f[2];
        } else {
            o6[0] = f[2]; o6[1] = f[0]; o6[2] = f[1];
            o6[3] = f[0]; o6[4] = f[2]; o6[5] = f[3];
        }
        ++q;
    }
}

struct SdWs {
    // look-back states, then [0] eff, [1..2] totals, [3] ticket and blocks done, [4..8] counts and [9] status for
    // callers without their own (zeroed together)
    unsigned long long* state;
    long long *eff, *tot, *counts;
    unsigned int* ticket;
    int* status;
    size_t zero_bytes;
    unsigned long long* blk;    // (quads, representatives) per block of active cells
    uint32_t *act, *lat, *vmap, *nbr;
    uint8_t *cas, *used, *face, *qbits;
    float* dual;
    long long nblk;
    size_t total;
};

SdWs carve_sd(void* ws, long long n, long long capA) {
    SdWs w{};
    uint8_t* b = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~uintptr_t(255));
    size_t o = 0;
    auto take = [&](size_t bytes) {
        uint8_t* p = ws ? b + o : nullptr;
        o = (o + std::max<size_t>(bytes, 1) + 255) & ~size_t(255);
        return p;
    };
    const long long ntile = (n + SD_TILE - 1) / SD_TILE;
    w.nblk = (capA + SD_BLOCK - 1) / SD_BLOCK;
    w.zero_bytes = size_t(ntile + 10) * 8;
    w.state = reinterpret_cast<unsigned long long*>(take(w.zero_bytes));
    w.eff = reinterpret_cast<long long*>(w.state) + ntile;
    w.tot = w.eff + 1;
    w.ticket = reinterpret_cast<unsigned int*>(w.eff + 3);
    w.counts = w.eff + 4;
    w.status = reinterpret_cast<int*>(w.eff + 9);
    w.blk = reinterpret_cast<unsigned long long*>(take(size_t(w.nblk + 1) * 16));
    w.act = reinterpret_cast<uint32_t*>(take(size_t(capA) * 4));
    w.lat = reinterpret_cast<uint32_t*>(take(size_t(capA) * 4));
    w.vmap = reinterpret_cast<uint32_t*>(take(size_t(capA) * 4));
    w.nbr = reinterpret_cast<uint32_t*>(take(size_t(capA) * 24));
    w.cas = take(size_t(capA));
    w.used = take(size_t(capA));
    w.face = take(size_t(capA));
    w.qbits = take(size_t(capA));
    w.dual = reinterpret_cast<float*>(take(size_t(capA) * 12));
    w.total = o + 256;
    return w;
}

size_t sd_workspace(long long n, long long capA, long long capF) {
    return n < 0 || capA < 0 || capF < 0 ? 0 : carve_sd(nullptr, n, capA).total;
}

int sd_launch(const int* ids, const float* values, long long n, int nx, int ny, int nz, const float* aabb_min,
              const float* aabb_max, float level, float reg, float svd_tol, float* vertices,
              long long vertex_capacity, int* faces, long long face_capacity, void* workspace, size_t workspace_bytes,
              long long* counts, int* status, iso::HostSizes* host, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (((!counts || !status) && !host) || !aabb_min || !aabb_max || vertex_capacity < 0 || face_capacity < 0 || n > 0x7fffffffll)
        return iso::fail_code(ISO_ERR_ARG);
    if (n <= 0 && host) return 0;  // the sizes are 0
    if (n <= 0)
        return cudaMemsetAsync(counts, 0, 5 * sizeof(long long), st) == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
    if (nx < 2 || ny < 2 || nz < 2 || !ids || !values || (reinterpret_cast<uintptr_t>(values) & 15) ||
        (vertex_capacity && !vertices) || (face_capacity && !faces))
        return iso::fail_code(ISO_ERR_ARG);
    if (workspace_bytes < sd_workspace(n, vertex_capacity, face_capacity))
        return iso::fail_code(ISO_ERR_WORKSPACE);
    long long* const words = host ? host->lease() : nullptr;
    if (host && !words) return ISO_ERR_CUDA;
    const long long capA = vertex_capacity;
    const SdWs w = carve_sd(workspace, n, capA);
    const Grid3 g = make_grid(nx, ny, nz, aabb_min, aabb_max);
    const uint32_t *act = w.act, *lat = w.lat, *vmap = w.vmap, *nbr = w.nbr;
    const uint8_t *cas = w.cas, *used = w.used, *face = w.face, *qbits = w.qbits;
    const long long *eff = w.eff, *tot = w.tot;
    const unsigned long long* blk = w.blk;
    const float* dual = w.dual;
    if (!counts) counts = w.counts;
    if (!status) status = w.status;
    {
        iso::ProfScope ps("sparse_its", st);
        if (cudaMemsetAsync(w.state, 0, w.zero_bytes, st) != cudaSuccess) return iso::fail_code(ISO_ERR_CUDA);
        sd_classify<<<unsigned((n + SD_TILE - 1) / SD_TILE), SD_THREADS, 0, st>>>(
            ids, values, uint32_t(n), level, w.ticket, w.state, w.act, w.lat, w.cas, w.used, capA, w.eff, counts,
            status);
    }
    if (capA > 0) {
        const unsigned nblk = unsigned(w.nblk);
        {
            iso::ProfScope ps("dc_solve", st);
            iso::launch_pdl(g.fma ? sd_solve<true> : sd_solve<false>, blocks_for(capA, 128), 128u, st, values, g, level,
                            act, lat, cas, eff, reg, svd_tol, w.dual, w.face);
        }
        {
            iso::ProfScope ps("sparse_quads", st);
            iso::launch_pdl(sd_quads, nblk, unsigned(SD_BLOCK), st, g, lat, cas, eff, capA, w.used, w.qbits, w.nbr,
                            w.blk);
        }
        {
            const bool scan = nblk <= SD_SCAN;
            // the table, where one is needed, lies in the vertices until sd_number writes them
            const bool hash = coords_may_repeat(g);
            const WeldTable table{hash ? reinterpret_cast<uint32_t*>(vertices) : nullptr, weld_table_size(capA)};
            iso::ProfScope ps("dc_weld", st, (scan ? 2 : 3) + (hash ? 1 : 0));
            if (hash && launch_weld_table(table, dual, used, 1u, face, eff, capA, st) != cudaSuccess)
                return iso::fail_code(ISO_ERR_CUDA);
            iso::launch_pdl(sd_flags, nblk, unsigned(SD_BLOCK), st, g, lat, used, face, dual, eff, w.vmap, w.blk, scan,
                            w.ticket + 1, w.tot, table);
            if (!scan) iso_block_scan_launch(w.blk, w.nblk, w.tot, st);
            iso::launch_pdl(sd_number, nblk, unsigned(SD_BLOCK), st, dual, eff, blk, tot, face_capacity, w.vmap,
                            vertices, counts, status);
        }
        {
            iso::ProfScope ps("sparse_quads", st);
            iso::launch_pdl(sd_faces, nblk, unsigned(SD_BLOCK), st, g, qbits, nbr, capA, dual, vmap, eff, blk, tot,
                            face_capacity, faces, static_cast<const long long*>(counts),
                            static_cast<const int*>(status), words);
        }
    }
    return cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
}

}  // namespace

extern "C" {

size_t iso_sparse_dc_workspace_size(long long n, long long vertex_capacity, long long face_capacity) {
    return sd_workspace(n, vertex_capacity, face_capacity);
}

int iso_sparse_dc(const int* ids, const float* values, long long n, int nx, int ny, int nz, const float* aabb_min,
                  const float* aabb_max, float level, float reg, float svd_tol, float* vertices,
                  long long vertex_capacity, int* faces, long long face_capacity, void* workspace,
                  size_t workspace_bytes, long long* counts, int* status, void* stream) {
    return sd_launch(ids, values, n, nx, ny, nz, aabb_min, aabb_max, level, reg, svd_tol, vertices, vertex_capacity,
                     faces, face_capacity, workspace, workspace_bytes, counts, status, nullptr, stream);
}

int iso_sparse_dc_sync(const int* ids, const float* values, long long n, int nx, int ny, int nz,
                       const float* aabb_min, const float* aabb_max, float level, float reg, float svd_tol,
                       float* vertices, long long vertex_capacity, int* faces, long long face_capacity,
                       void* workspace, size_t workspace_bytes, long long* sizes, void* stream) {
    if (!sizes || vertex_capacity < 1) return iso::fail_code(ISO_ERR_ARG);
    iso::HostSizes host;
    const int rc = sd_launch(ids, values, n, nx, ny, nz, aabb_min, aabb_max, level, reg, svd_tol, vertices,
                             vertex_capacity, faces, face_capacity, workspace, workspace_bytes, nullptr, nullptr,
                             &host, stream);
    return host.wait(rc, 6, sizes, reinterpret_cast<cudaStream_t>(stream));
}

}  // extern "C"
