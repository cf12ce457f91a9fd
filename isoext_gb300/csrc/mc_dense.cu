// Dense-grid marching cubes on sm_103a.
//
// Four launches on one stream (five on grids of more than 1024 segments), nothing
// read back by the host:
//   1. mc_signs   streams the grid once (32 coalesced 128-byte loads in flight per
//                 warp) into a sign bitmap,
//                 1 bit per point.  This is the only pass over all values.
//   2. mc_count   one CTA per segment of 128 to 1024 point words, from the bitmap
//                 alone (16.8 MB at 512^3): the words near the surface, listed;
//                 their crossed-edge masks, active cells and triangle counts,
//                 bit-parallel; vertex and cell entry lists.  On grids of few
//                 segments its last CTA scans their sums.
//   3. mc_scan    (more segments) (V, F) sums to offsets: CTAs over chunks of 1024
//                 segments chained by decoupled look-back; totals and the
//                 capacity check.
//   4. mc_emit    one thread per vertex entry (position at its slot; values are
//                 read only at crossed edges) and per cell entry (its faces, vertex
//                 indices by rank).  Vertices that can share a position with
//                 another edge's (t within tau of 0 or 1) go through a small
//                 hash that counts exact coincidences.
//   5. mc_fix     returns at once unless the emit found coinciding vertices; then
//                 merges them by exact position, drops faces that became
//                 degenerate and compacts vertices and faces in place, keeping
//                 their order.
//
// Equivalence with the reference (src/mc/mc.cu:17-68): the reference emits the
// triangles of active cells in ascending cell id, drops triangles with two equal
// vertex positions (src/mc/nagae.cu:71), and welds vertices by exact position
// (src/utils.cu:32-59).  Positions here use the reference's operation order
// and its rounding, in either reading of its arithmetic (the fused one of its
// CUDA build or the unfused one of its host build, common.cuh), so they are
// bit-identical.  Two
// distinct crossed edges give equal positions only when both vertices land on
// the same grid point (on grids whose spacing is far above float resolution;
// the host layer handles the rest), and those are the snapped vertices the
// fix-up merges.  Every crossed edge of a cell appears in its triangles (both
// tables), so without snaps the vertex set is exactly the crossed edges.
// Vertices come in edge order (the reference sorts them by position; the mesh
// is the same after relabelling).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <mutex>

#include "common.cuh"
#define ISO_LUT_DECL static __constant__ const
#include "luts.h"
#include "lookback.cuh"
#include "mc_dense.cuh"
#include "profile.cuh"

namespace {

// ---------------------------------------------------------------------------
// Geometry shared by the kernels.

// Unsigned 32-bit division by a divisor fixed for a launch, by multiply and
// shift (Granlund and Montgomery, "Division by invariant integers using
// multiplication", 1994): for 1 <= d < 2^31, l = ceil(log2 d) and
// m = floor(2^32 (2^l - d) / d) + 1, n / d = (t + ((n - t) >> 1)) >> (l - 1) with
// t = umulhi(m, n); exact for every 32-bit n.
struct FastDiv {
    uint32_t d, m, l;
};

FastDiv make_fastdiv(uint32_t d) {
    FastDiv f{d, 0u, 0u};
    while ((1ull << f.l) < d) ++f.l;
    if (d > 1) f.m = uint32_t(((1ull << 32) * ((1ull << f.l) - d)) / d + 1);
    return f;
}

__device__ __forceinline__ uint32_t fdiv(uint32_t n, const FastDiv& f) {
    if (f.d == 1) return n;
    const uint32_t t = __umulhi(f.m, n);
    return (t + ((n - t) >> 1)) >> (f.l - 1);
}

struct McGrid {
    FastDiv dNW, dNY;  // division by NW and by ny
    int nx, ny, nz, NW;
    long long PW;     // point words nx * ny * NW
    float level;
    int method;
    const float* gc;  // grid coordinates: x [nx], then y [ny], then z [nz]
    // Vertices whose edge parameter t is within tau of 0 or 1 are the only ones
    // that can share a position with a vertex of another edge (mc_snap_tau).
    float tau;
    bool fma;  // arithmetic reading (iso::arith_fma at the call)
    int lgseg; // log2 of the point words per segment (the count kernel's CTA size times WPT)
};

// Workspace carved from one buffer (offsets 256-aligned).
struct McWs {
    uint32_t* S;                // sign bitmap [PW]
    uint32_t* info;             // per word: segment-local vertex offset | popc(ex) << 20 | popc(ey) << 26
    unsigned long long* blk;    // per segment of words: (V, F) sums, then exclusive offsets
    unsigned long long* vlist;  // vertex entries [capV]: pw | axis << 32 | bit << 34 | slot << 39
    unsigned long long* clist;  // cell entries [capF]: pw | bit << 32 | the word's segment-local face offset << 37
    unsigned long long* blk2;   // blk of grids of one word per count thread, cut into more than nBlk segments
    unsigned long long* ctr;    // [0] list size [1] snaps [2] V [3] F when the caller has no counts [4] V [5] F (before the fix-up) [6] count CTAs done [7] scan ticket
                                // [8] merges [9] small hash full [10] cell entries [12] fix-up ticket
                                // [13] fix-up tiles done [14] status when the caller has none; the rest unused
    unsigned long long* state;  // look-back state per segment (follows ctr; zeroed with it)
    uint32_t* small;            // SMALL_HC entries after the states (zeroed with them)
    float* gc;                  // grid coordinates [nx + ny + nz] (x, then y, then z)
    uint32_t* snaps;            // snapped vertex slots [capV]
    uint32_t* table;            // position hash of snapped vertices [HC]
    uint32_t* moved;            // fix-up: bitmap of the merged vertices [capV / 32 + 1]
    uint32_t* newidx;           // fix-up: a merged vertex's representative, then new indices [capV]
    unsigned long long* fstate; // fix-up: look-back states of its face tiles (region of capF * 12 bytes)
    uint32_t* vbits;            // fix-up: two more bitmaps, then the look-back states of its vertex tiles
                                // (region of capV * 12 bytes)
    long long nBlk;             // segments of SEG_MIN point words: as many as four words per count thread make, at most
    uint32_t HC;
    size_t total;
};

constexpr uint32_t SMALL_HC = 1u << 15;  // merge-detection hash of emit (entries: vertex + 1, 0 = empty)
constexpr uint32_t SMALL_PROBES = 256;
constexpr int NCTR = 16;
constexpr int WPT_MAX = 4;                   // point words per count thread (1 on small grids)
constexpr int FIX_THREADS = 512;
constexpr int FIX_CTAS = 3;                  // resident fix-up CTAs per SM
constexpr int FIX_PER = 4;                   // rows per thread of a fix-up tile
constexpr int FIX_TILE = FIX_THREADS * FIX_PER;
constexpr uint32_t SEG_MIN = 128 * WPT_MAX;  // words per segment (one scan entry) of 128-thread count CTAs

inline size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

uint32_t hash_cap(long long capV) {
    uint32_t c = 1024;
    while ((long long)c < 2 * capV + 1024) c <<= 1;
    return c;
}

// Bytes cleared at the start of each call: counters, look-back states, small hash.
inline size_t zeroed_bytes(long long nBlk) { return size_t(NCTR) * 8 + size_t(nBlk) * 8 + size_t(SMALL_HC) * 4; }

McWs carve(int nx, int ny, int nz, long long capV, long long capF, uint8_t* base) {
    McWs w{};
    const long long NW = (nz + 31) / 32;
    const long long PW = (long long)nx * ny * NW;
    w.nBlk = (PW + SEG_MIN - 1) / SEG_MIN;
    w.HC = hash_cap(capV);
    size_t o = 0;
    auto take = [&](size_t bytes) {
        uint8_t* p = base ? base + o : nullptr;
        o = al256(o + std::max<size_t>(bytes, 1));
        return p;
    };
    w.S = reinterpret_cast<uint32_t*>(take(size_t(PW) * 4));
    w.info = reinterpret_cast<uint32_t*>(take(size_t(PW) * 4));
    w.blk = reinterpret_cast<unsigned long long*>(take(size_t(w.nBlk + 1) * 16));
    w.vlist = reinterpret_cast<unsigned long long*>(take(size_t(capV) * 8));
    w.clist = reinterpret_cast<unsigned long long*>(take(size_t(capF) * 8));
    w.blk2 = reinterpret_cast<unsigned long long*>(take(size_t(PW) * 4));
    w.ctr = reinterpret_cast<unsigned long long*>(take(zeroed_bytes(w.nBlk)));  // + states + small hash
    w.state = w.ctr ? w.ctr + NCTR : nullptr;
    w.small = w.ctr ? reinterpret_cast<uint32_t*>(w.state + w.nBlk) : nullptr;
    w.gc = reinterpret_cast<float*>(take(size_t(nx + ny + nz) * 4));
    w.snaps = reinterpret_cast<uint32_t*>(take(size_t(capV) * 4));
    w.table = reinterpret_cast<uint32_t*>(take(size_t(w.HC) * 4));
    w.moved = reinterpret_cast<uint32_t*>(take(size_t(capV / 32 + 1) * 4));
    w.newidx = reinterpret_cast<uint32_t*>(take(size_t(capV) * 4));
    // the fix-up needs far less of these two, whose sizes are part of the workspace's
    w.fstate = reinterpret_cast<unsigned long long*>(take(size_t(capF) * 12));
    w.vbits = reinterpret_cast<uint32_t*>(take(size_t(capV) * 12));
    w.total = o + 256;  // room to align the base
    return w;
}

// ---------------------------------------------------------------------------
// Per-word bit state.

// The 8 bitmap words around point word (x, y, w): s[dx][dy][0] = word w of row
// (x + dx, y + dy), s[..][1] = word w + 1 (0 past the row or grid).
struct Words {
    uint32_t s[2][2][2];
    int x, y, w;
    bool hasx, hasy;
};

__device__ __forceinline__ void load_words(const McGrid& g, const uint32_t* __restrict__ S, uint32_t pw, int x,
                                           int y, int w, Words& d) {
    d.x = x;
    d.y = y;
    d.w = w;
    d.hasx = x < g.nx - 1;
    d.hasy = y < g.ny - 1;
    const bool nxt = w + 1 < g.NW;
    const uint32_t sx = uint32_t(g.ny) * uint32_t(g.NW), sy = uint32_t(g.NW);
#pragma unroll
    for (int dx = 0; dx < 2; ++dx)
#pragma unroll
        for (int dy = 0; dy < 2; ++dy) {
            const bool ok = (dx == 0 || d.hasx) && (dy == 0 || d.hasy);
            const uint32_t q = pw + dx * sx + dy * sy;
            d.s[dx][dy][0] = ok ? __ldg(S + q) : 0u;
            d.s[dx][dy][1] = (ok && nxt) ? __ldg(S + q + 1) : 0u;
        }
}

// Bits of word w whose z is below nz - 1 (z edges and cells need z + 1).
__device__ __forceinline__ uint32_t zmask(const McGrid& g, int w) {
    const int n = g.nz - 1 - 32 * w;
    return n >= 32 ? ~0u : (n <= 0 ? 0u : ((1u << n) - 1u));
}

// Word shifted so that bit b holds bit b + 1 (z + 1).
__device__ __forceinline__ uint32_t up1(uint32_t lo, uint32_t hi) { return __funnelshift_r(lo, hi, 1); }

__device__ __forceinline__ uint32_t ez_of(uint32_t lo, uint32_t hi, uint32_t zm) {
    return (lo ^ up1(lo, hi)) & zm;
}

// Active cells of the word: corners straddle the level.
__device__ __forceinline__ uint32_t active_cells(const Words& d, uint32_t zm) {
    if (!d.hasx || !d.hasy) return 0u;
    uint32_t a = ~0u, o = 0u;
#pragma unroll
    for (int dx = 0; dx < 2; ++dx)
#pragma unroll
        for (int dy = 0; dy < 2; ++dy) {
            const uint32_t lo = d.s[dx][dy][0], hi = up1(lo, d.s[dx][dy][1]);
            a &= lo & hi;
            o |= lo | hi;
        }
    return (o & ~a) & zm;
}

// The 8 corner words of a word's cells: c[k] = corner k = 4dx + 2dy + dz.
__device__ __forceinline__ void corner_words(const Words& d, uint32_t* c) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        c[2 * k] = d.s[k >> 1][k & 1][0];
        c[2 * k + 1] = up1(d.s[k >> 1][k & 1][0], d.s[k >> 1][k & 1][1]);
    }
}
__device__ __forceinline__ uint32_t case_at(const uint32_t* c, int b) {
    uint32_t cs = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) cs |= ((c[k] >> b) & 1u) << k;
    return cs;
}

// Cells whose crossed edges may form more than one loop: a face whose diagonal
// corners pair up, or two opposite corners against the other six.  Every other
// active cell has one polygon, so its table has (crossed edges - 2) triangles;
// both tables hold to this (checked over all cases).
__device__ __forceinline__ uint32_t many_loops(const uint32_t* c) {
    uint32_t m = 0;
    const int f[6][4] = {{0, 1, 3, 2}, {4, 5, 7, 6}, {0, 1, 5, 4}, {2, 3, 7, 6}, {0, 2, 6, 4}, {1, 3, 7, 5}};
#pragma unroll
    for (int q = 0; q < 6; ++q)
        m |= ~(c[f[q][0]] ^ c[f[q][2]]) & ~(c[f[q][1]] ^ c[f[q][3]]) & (c[f[q][0]] ^ c[f[q][1]]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t all = ~0u, any = 0u;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (k != i && k != 7 - i) {
                all &= c[k];
                any |= c[k];
            }
        m |= (c[i] & c[7 - i] & ~any) | (~c[i] & ~c[7 - i] & all);
    }
    return m;
}

// Triangles of the active cells `cells` of a word, by popcounts: crossed edges
// minus two per cell, and the table's own number where a cell may have several
// loops.  ntri(case): the table.
template <typename Ntri>
__device__ __forceinline__ uint32_t word_faces(const uint32_t* c, uint32_t cells, const Ntri& ntri) {
    uint32_t multi = many_loops(c) & cells;
    const uint32_t one = cells & ~multi;
    uint32_t n = 0;
#pragma unroll
    for (int e = 0; e < 12; ++e) n += __popc((c[iso_edge_corner(2 * e)] ^ c[iso_edge_corner(2 * e + 1)]) & one);
    n -= 2u * __popc(one);
    for (; multi; multi &= multi - 1) n += ntri(case_at(c, __ffs(multi) - 1));
    return n;
}

// Block-wide exclusive scan of two counts; totals in ta, tb.
template <int BLOCK>
__device__ __forceinline__ void block_scan2(uint32_t a, uint32_t b, uint32_t& ea, uint32_t& eb, uint32_t& ta,
                                            uint32_t& tb, uint32_t* sm) {
    constexpr int NWARP = BLOCK / 32;
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
// 2. count: one CTA per segment of T * WPT point words (T is a launch parameter,
// "mc.count_threads"): per-word vertex offsets, vertex and cell entries, and the
// segments' (V, F) sums turned into offsets.

// Segment holding point word pw.
__device__ __forceinline__ uint32_t seg_of(const McGrid& g, uint32_t pw) { return pw >> g.lgseg; }

// (x, y, w) of point word pw.
__device__ __forceinline__ void word_xyw(const McGrid& g, uint32_t pw, int& x, int& y, int& w) {
    const uint32_t row = fdiv(pw, g.dNW);
    w = int(pw - row * uint32_t(g.NW));
    x = int(fdiv(row, g.dNY));
    y = int(row - uint32_t(x) * uint32_t(g.ny));
}

__device__ __forceinline__ uint32_t pbits(float f) { return __float_as_uint(f == 0.0f ? 0.0f : f); }
__device__ __forceinline__ uint32_t phash(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t h = a * 0x9E3779B1u ^ (b + 0x7F4A7C15u) * 0x85EBCA77u ^ (c + 0x165667B1u) * 0xC2B2AE3Du;
    h ^= h >> 15;
    h *= 0x2C1B3C6Du;
    h ^= h >> 12;
    return h;
}
// Equal positions; q is read through L2 (another CTA of the launch may have
// written it).
__device__ __forceinline__ bool same_pos(const float* p, const float* q) {
    return p[0] == __ldcg(q) && p[1] == __ldcg(q + 1) && p[2] == __ldcg(q + 2);
}

// Totals of the scan: the counts, and whether they fit.
__device__ __forceinline__ void mc_totals(unsigned long long V, unsigned long long F, unsigned long long* ctr,
                                          long long* counts, int* status, long long capV, long long capF) {
    counts[0] = (long long)V;
    counts[1] = (long long)F;
    ctr[4] = V;
    ctr[5] = F;
    if ((long long)V > capV || (long long)F > capF || V >= LB_MASK31 || F >= LB_MASK31)
        atomicCAS(status, 0, int(ISO_ERR_OVERFLOW));
}

// Segments that the last count CTA scans by itself, per thread.  Up to 4 T
// segments this saves the launch of mc_scan (4 us); the count's CTAs then each
// take a fence and an atomic on one counter before they end, which costs more
// than the launch from 2048 segments on (15 -> 22 us at 2048, 48 -> 60 us at 4096).
// Their sums fit 32 bits (1024 segments of 1024 words, each below 2^18).
constexpr int SCAN_LAST = 4;

template <int T>
__device__ void scan_segments(unsigned long long* blk, uint32_t nseg, unsigned long long* ctr, long long* counts,
                              int* status, long long capV, long long capF, uint32_t* sm) {
    const uint32_t per = (nseg + T - 1) / T;  // at most SCAN_LAST
    const uint32_t s0 = threadIdx.x * per;
    uint32_t a[SCAN_LAST], b[SCAN_LAST], sa = 0, sb = 0;
#pragma unroll
    for (int k = 0; k < SCAN_LAST; ++k) {
        const bool in = k < per && s0 + k < nseg;
        const ulonglong2 v = in ? __ldcg(reinterpret_cast<const ulonglong2*>(blk) + s0 + k) : make_ulonglong2(0, 0);
        a[k] = uint32_t(v.x);
        b[k] = uint32_t(v.y);
        sa += a[k];
        sb += b[k];
    }
    uint32_t ea, eb, ta, tb;
    block_scan2<T>(sa, sb, ea, eb, ta, tb, sm);
    if (threadIdx.x == 0) mc_totals(ta, tb, ctr, counts, status, capV, capF);
#pragma unroll
    for (int k = 0; k < SCAN_LAST; ++k) {
        if (k < per && s0 + k < nseg)
            reinterpret_cast<ulonglong2*>(blk)[s0 + k] = make_ulonglong2(ea, eb);
        ea += a[k];
        eb += b[k];
    }
}

// One CTA's segment: T threads of WPT words each.
// First every thread tells which of its words may hold a crossing: most words
// and their grid neighbours are all inside or all outside.  The others, a few
// percent, are listed in order, and from there on a thread takes one of them at
// a time: the crossed-edge masks, the active cells and the number of their
// triangles (word_faces), all bit-parallel; a block scan of the three counts; and
// the entries of the warp's crossed edges and active cells, laid out in order in
// shared memory (a lane walks its word's set bits) so that they leave in
// coalesced stores.  A cell's entry carries its word's face offset; the emit adds
// the triangles of the cells before it in the word.
// Bound by instruction issue near the surface and by latency elsewhere, not by
// bytes (the bitmap is in L2).  A lane per active cell for its case and triangle
// count, spread over the owning warp only, as before, took 48 us at 512^3 and 16 to
// 40 at 256^3 (a warp along the surface alone with its cells); this takes 39 and
// 14 to 19.  The same without the list of words (every lane its own four words'
// masks, a quarter of the lanes near the surface) took 49.
constexpr int CQ = 512;  // entries a warp lays out at a time

template <int T, int WPT>
__global__ void __launch_bounds__(T, 1280 / T) mc_count(const McGrid g, const float amin0, const float amin1,
                                                        const float amin2, const float size0, const float size1,
                                                        const float size2, const uint32_t* __restrict__ S,
                                                        uint32_t* __restrict__ info, unsigned long long* blk,
                                                        unsigned long long* __restrict__ vlist,
                                                        unsigned long long* __restrict__ clist,
                                                        unsigned long long* ctr, float* __restrict__ gc,
                                                        const uint32_t nseg, const long long capV,
                                                        const long long capF, long long* counts, int* status) {
    constexpr uint32_t SEG = T * WPT;  // words of the segment
    constexpr int NW = T / 32;
    __shared__ uint32_t sm[64];
    __shared__ unsigned long long cbase_s, vbase_s, wsum[NW];
    __shared__ uint32_t bsum[NW];
    __shared__ uint16_t list[SEG];  // words that may hold a crossing
    __shared__ uint32_t fofs[T];    // face offset of each thread's word
    __shared__ uint16_t queue[NW][CQ];
    __shared__ int last_s;
    iso::grid_wait();
    // grid coordinates (include/utils.cuh:62-80), read by the emit kernel
    const uint32_t gid = blockIdx.x * T + threadIdx.x;
    const uint32_t ncoord = uint32_t(g.nx + g.ny + g.nz);
    if (gid < ncoord) {
        if (gid < uint32_t(g.nx)) gc[gid] = iso::grid_coord(gid, g.nx, amin0, size0, g.fma);
        else if (gid < uint32_t(g.nx + g.ny)) gc[gid] = iso::grid_coord(gid - g.nx, g.ny, amin1, size1, g.fma);
        else gc[gid] = iso::grid_coord(gid - g.nx - g.ny, g.nz, amin2, size2, g.fma);
    }
    const uint32_t seg = blockIdx.x;
    if (seg >= nseg) return;  // CTAs past the segments only write coordinates
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t sxw = uint32_t(g.ny) * uint32_t(g.NW), syw = uint32_t(g.NW);
    uint32_t nbusy = 0;  // words of the segment that may hold a crossing
    {
        const bool vec = WPT == 4 && (g.NW & 3) == 0;  // rows start on 16-byte boundaries
        const uint32_t pw0 = seg * SEG + threadIdx.x * WPT;
        // a word is quiet when it, the words at the same place of the rows (x, y+1),
        // (x+1, y), (x+1, y+1) and the words after these four are all 0 or all ~0
        // (conservative: at the grid's edges the rows are not neighbours)
        uint32_t lo[WPT], hi[WPT];  // AND and OR of the four rows' words
#pragma unroll
        for (int k = 0; k < WPT; ++k) { lo[k] = ~0u; hi[k] = 0u; }
        uint32_t nlo = ~0u, nhi = 0u;  // of the words after the thread's last
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t p = pw0 + (q >> 1) * sxw + (q & 1) * syw;
            uint32_t v[WPT];
            if (vec && pw0 + WPT <= g.PW && p + WPT <= g.PW) {
                const uint4 v4 = __ldg(reinterpret_cast<const uint4*>(S + p));
                const uint32_t t[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
                for (int k = 0; k < WPT; ++k) v[k] = t[k];
            } else {
#pragma unroll
                for (int k = 0; k < WPT; ++k) v[k] = p + k < g.PW ? __ldg(S + p + k) : 0u;
            }
            uint32_t nx = __shfl_down_sync(~0u, v[0], 1);
            if (lane == 31) nx = p + WPT < g.PW ? __ldg(S + p + WPT) : 0u;
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
            if (l != ~0u && h != 0u && pw0 + k < g.PW) m |= 1u << k;
        }
        const uint32_t mine = __popc(m);
        uint32_t inc = mine;
#pragma unroll
        for (int dd = 1; dd < 32; dd <<= 1) {
            const uint32_t t = __shfl_up_sync(~0u, inc, dd);
            if (lane >= dd) inc += t;
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
    // A segment without such words has no crossed edge and no active cell: its
    // sums are 0, and no cell reads its words' vertex offsets (a cell's edges lie
    // in words with crossings).
    uint32_t tv = 0, tf = 0;  // edges and faces of the rounds so far
    for (uint32_t r0 = 0; r0 < nbusy; r0 += T) {
        __syncthreads();  // the list; the shared arrays of the round before
        uint32_t e3[3] = {0u, 0u, 0u}, act = 0, nf = 0, pw = 0;
        const uint32_t i = r0 + threadIdx.x;
        if (i < nbusy) {
            pw = seg * SEG + list[i];
            int x, y, w;
            word_xyw(g, pw, x, y, w);
            Words d;
            load_words(g, S, pw, x, y, w, d);
            const uint32_t zm = zmask(g, w);
            e3[0] = d.hasx ? (d.s[0][0][0] ^ d.s[1][0][0]) : 0u;
            e3[1] = d.hasy ? (d.s[0][0][0] ^ d.s[0][1][0]) : 0u;
            e3[2] = ez_of(d.s[0][0][0], d.s[0][0][1], zm);
            act = active_cells(d, zm);
            if (act) {
                uint32_t c[8];
                corner_words(d, c);
                nf = word_faces(c, act, [&](uint32_t cs) { return uint32_t(ISO_NTRI[g.method * 256 + cs]); });
            }
        }
        const uint32_t cx = __popc(e3[0]), cy = __popc(e3[1]);
        const uint32_t nv = cx + cy + __popc(e3[2]), na = __popc(act);
        // active cells (at most 32 T), edges (from bit 20) and faces (from 40)
        const unsigned long long mine = (unsigned long long)na | ((unsigned long long)nv << 20) |
                                        ((unsigned long long)nf << 40);
        unsigned long long inc = mine;
#pragma unroll
        for (int dd = 1; dd < 32; dd <<= 1) {
            const unsigned long long t = __shfl_up_sync(~0u, inc, dd);
            if (lane >= dd) inc += t;
        }
        if (lane == 31) wsum[warp] = inc;
        __syncthreads();
        unsigned long long before = 0, all = 0;
#pragma unroll
        for (int q = 0; q < NW; ++q) {
            before += q < warp ? wsum[q] : 0ull;
            all += wsum[q];
        }
        // the round's blocks of both lists, both atomics in flight together
        const uint32_t ta = uint32_t(all) & 0xfffffu, te = uint32_t(all >> 20) & 0xfffffu;
        if (threadIdx.x == 0) cbase_s = ta ? atomicAdd(ctr + 10, (unsigned long long)ta) : 0ull;
        else if (threadIdx.x == 32) vbase_s = te ? atomicAdd(ctr, (unsigned long long)te) : 0ull;
        const unsigned long long ex = inc - mine;  // within the warp
        if (nv) info[pw] = (tv + (uint32_t((before + ex) >> 20) & 0xfffffu)) | (cx << 20) | (cy << 26);
        fofs[threadIdx.x] = tf + uint32_t((before + ex) >> 40);
        __syncthreads();  // the list blocks; from here to the next round warps go their own ways
        const unsigned long long wtot = __shfl_sync(~0u, inc, 31);
        uint16_t* q = queue[warp];
        // active cells in cell order: lane << 5 | bit
        {
            const uint32_t n = uint32_t(wtot) & 0xfffffu, c0 = uint32_t(ex) & 0xfffffu;
            const unsigned long long base = cbase_s + (uint32_t(before) & 0xfffffu);
            for (uint32_t q0 = 0; q0 < n; q0 += CQ) {
                if (na && c0 < q0 + CQ && c0 + na > q0) {
                    uint32_t j = c0 - q0;  // wraps below q0: not in this window
                    for (uint32_t m = act; m; m &= m - 1, ++j)
                        if (j < uint32_t(CQ)) q[j] = uint16_t((lane << 5) | (__ffs(m) - 1));
                }
                __syncwarp();
                for (uint32_t j = lane; j < min(uint32_t(CQ), n - q0); j += 32) {
                    const uint32_t it = q[j], o = warp * 32 + (it >> 5);
                    const unsigned long long ci = base + q0 + j;
                    if ((long long)ci < capF)
                        clist[ci] = (unsigned long long)(seg * SEG + list[r0 + o]) |
                                    ((unsigned long long)(it & 31u) << 32) | ((unsigned long long)fofs[o] << 37);
                }
                __syncwarp();
            }
        }
        // crossed edges in slot order (x edges, then y, then z of each word):
        // lane << 7 | axis << 5 | bit
        {
            const uint32_t n = uint32_t(wtot >> 20) & 0xfffffu, v0 = uint32_t(ex >> 20) & 0xfffffu;
            const uint32_t slot0 = uint32_t(before >> 20) & 0xfffffu;
            const unsigned long long base = vbase_s + slot0;
            for (uint32_t q0 = 0; q0 < n; q0 += CQ) {
                if (nv && v0 < q0 + CQ && v0 + nv > q0) {
                    uint32_t j = v0 - q0;
#pragma unroll
                    for (int ax = 0; ax < 3; ++ax)
                        for (uint32_t m = e3[ax]; m; m &= m - 1, ++j)
                            if (j < uint32_t(CQ)) q[j] = uint16_t((lane << 7) | (ax << 5) | (__ffs(m) - 1));
                }
                __syncwarp();
                for (uint32_t j = lane; j < min(uint32_t(CQ), n - q0); j += 32) {
                    const uint32_t it = q[j];
                    const unsigned long long vb = base + q0 + j;
                    if ((long long)vb < capV)
                        vlist[vb] = (unsigned long long)(seg * SEG + list[r0 + warp * 32 + (it >> 7)]) |
                                    ((unsigned long long)((it >> 5) & 3u) << 32) |
                                    ((unsigned long long)(it & 31u) << 34) |
                                    ((unsigned long long)(tv + slot0 + q0 + j) << 39);
                }
                __syncwarp();
            }
        }
        tv += te;
        tf += uint32_t(all >> 40);
    }
    // the segment's sums; the last CTA turns them into offsets when it can
    const bool scans = nseg <= uint32_t(SCAN_LAST * T);
    if (threadIdx.x == 0) {
        reinterpret_cast<ulonglong2*>(blk)[seg] = make_ulonglong2(tv, tf);
        if (scans) {
            __threadfence();
            last_s = atomicAdd(ctr + 6, 1ull) == nseg - 1;
            __threadfence();
        }
    }
    if (!scans) return;
    __syncthreads();
    if (last_s) scan_segments<T>(blk, nseg, ctr, counts, status, capV, capF, sm);
}

// ---------------------------------------------------------------------------
// 3. scan of the per-segment (V, F) sums of mc_count into exclusive offsets,
// for grids of more segments than the last count CTA scans: CTAs take chunks of
// SCAN_THREADS segments in ticket order and chain their totals by decoupled
// look-back.  The last chunk writes the totals and checks the capacities.
constexpr int SCAN_THREADS = 1024;

__global__ void __launch_bounds__(SCAN_THREADS) mc_scan(unsigned long long* blk, uint32_t nseg,
                                                        unsigned long long* ctr, unsigned long long* state,
                                                        long long* counts, int* status, long long capV,
                                                        long long capF) {
    __shared__ uint32_t sm[64];
    __shared__ uint32_t chunk_s;
    __shared__ unsigned long long pre_s[2];
    iso::grid_wait();
    if (threadIdx.x == 0) chunk_s = uint32_t(atomicAdd(ctr + 7, 1ull));
    __syncthreads();
    const uint32_t chunk = chunk_s;
    const uint32_t nchunk = (nseg + SCAN_THREADS - 1) / SCAN_THREADS;
    const uint32_t s = chunk * SCAN_THREADS + threadIdx.x;
    const uint32_t a = s < nseg ? uint32_t(blk[2 * s]) : 0u, b = s < nseg ? uint32_t(blk[2 * s + 1]) : 0u;
    uint32_t ea, eb, ta, tb;
    block_scan2<SCAN_THREADS>(a, b, ea, eb, ta, tb, sm);
    if (threadIdx.x < 32) {
        unsigned long long pv = 0, pf = 0;
        if (chunk == 0) {
            if (threadIdx.x == 0) atomicExch(state, lb_pack(LB_INC, ta, tb));
        } else {
            if (threadIdx.x == 0) atomicExch(state + chunk, lb_pack(LB_AGG, ta, tb));
            look_back(state, chunk, pv, pf, status);
            if (threadIdx.x == 0) atomicExch(state + chunk, lb_pack(LB_INC, pv + ta, pf + tb));
        }
        if (threadIdx.x == 0) {
            pre_s[0] = pv;
            pre_s[1] = pf;
            if (chunk == nchunk - 1) mc_totals(pv + ta, pf + tb, ctr, counts, status, capV, capF);
        }
    }
    __syncthreads();
    if (s < nseg) {
        blk[2 * s] = pre_s[0] + ea;
        blk[2 * s + 1] = pre_s[1] + eb;
    }
}

// The scan's look-back for chunk `seg` over states nobody publishes: it must
// give up after `limit` polls and set the status (a test of the bounded wait).
__global__ void lookback_probe(unsigned long long* state, uint32_t seg, uint32_t limit, int* status,
                               unsigned long long* out) {
    unsigned long long ev = 0, ef = 0;
    look_back(state, seg, ev, ef, status, limit);
    if (threadIdx.x == 0) {
        out[0] = ev;
        out[1] = ef;
    }
}

// ---------------------------------------------------------------------------
// 4. emit: one thread per vertex entry, then one thread per cell entry.

__device__ __forceinline__ float gx(const McGrid& g, int x) { return g.gc[x]; }
__device__ __forceinline__ float gy(const McGrid& g, int y) { return g.gc[g.nx + y]; }
__device__ __forceinline__ float gz(const McGrid& g, int z) { return g.gc[g.nx + g.ny + z]; }

struct EmitArgs {
    const float* vals;
    const uint32_t* S;
    const uint32_t* info;
    const unsigned long long* blk;
    const unsigned long long* vlist;
    const unsigned long long* clist;
    unsigned long long* ctr;
    uint32_t* snaps;
    uint32_t* small;
    float* vout;
    int32_t* fout;
    long long* counts;
    int* status;
    long long capV, capF;
    unsigned nbv;  // CTAs with the vertex role; the rest emit faces
    McWs w;        // what the fix-up needs cleared
    long long* vedge;  // optional: each vertex's grid edge
};

// Vertex role: one thread per vertex entry; CTA `bi` of `nb`.
template <int EMIT_THREADS>
__device__ void emit_vertices(const McGrid& g, const EmitArgs& a, unsigned bi, unsigned nb) {
    const float* __restrict__ vals = a.vals;
    const unsigned long long* __restrict__ blk = a.blk;
    const unsigned long long* __restrict__ vlist = a.vlist;
    unsigned long long* ctr = a.ctr;
    uint32_t* __restrict__ snaps = a.snaps;
    uint32_t* small = a.small;
    float* vout = a.vout;
    const long long capV = a.capV;
    const unsigned long long n = min(ctr[0], (unsigned long long)capV);
    const long long sxv = (long long)g.ny * g.nz;
    for (unsigned long long i = (unsigned long long)bi * EMIT_THREADS + threadIdx.x; i < n;
         i += (unsigned long long)nb * EMIT_THREADS) {
        const unsigned long long e = vlist[i];
        const uint32_t pw = uint32_t(e);
        const int ax = int((e >> 32) & 3u), b = int((e >> 34) & 31u);
        const uint32_t vi = uint32_t(blk[2 * seg_of(g, pw)]) + uint32_t((e >> 39) & 0xfffffu);
        int x, y, w;
        word_xyw(g, pw, x, y, w);
        const int z = 32 * w + b;
        const long long ia = ((long long)x * g.ny + y) * g.nz + z;
        const long long step = ax == 0 ? sxv : (ax == 1 ? (long long)g.nz : 1ll);
        const float va = __ldg(vals + ia), vb = __ldg(vals + ia + step);
        const float t = iso::cross_t(g.level, va, vb);
        const float xa = gx(g, x), ya = gy(g, y), za = gz(g, z);
        const float xb = ax == 0 ? gx(g, x + 1) : xa;
        const float yb = ax == 1 ? gy(g, y + 1) : ya;
        const float zb = ax == 2 ? gz(g, z + 1) : za;
        const float px = iso::lerp1(t, xa, xb, g.fma), py = iso::lerp1(t, ya, yb, g.fma),
                    pz = iso::lerp1(t, za, zb, g.fma);
        float* vo = vout + 3ll * vi;
        vo[0] = px;
        vo[1] = py;
        vo[2] = pz;
        if (a.vedge) a.vedge[vi] = 3 * ia + ax;
        // (a position with a NaN equals none)
        if ((!(t >= g.tau && t <= 1.0f - g.tau) || (px == xa && py == ya && pz == za) ||
             (px == xb && py == yb && pz == zb)) &&
            px == px && py == py && pz == pz) {
            // a candidate for sharing its position: list it, and look for an
            // equal position among the candidates so far.  A slot keeps the
            // smallest vertex of its position (the fix-up's representative).
            const unsigned long long sidx = atomicAdd(ctr + 1, 1ull);
            if ((long long)sidx < capV) snaps[sidx] = vi;
            __threadfence();  // the position is visible before the hash entry
            const float pos[3] = {px, py, pz};
            uint32_t h = phash(pbits(px), pbits(py), pbits(pz)) & (SMALL_HC - 1u);
            bool placed = false;
            // past SMALL_PROBES the table counts as full: the fix-up builds its own
            for (uint32_t probe = 0; probe < SMALL_PROBES; ++probe, h = (h + 1) & (SMALL_HC - 1u)) {
                const uint32_t cur = atomicCAS(&small[h], 0u, vi + 1u);
                if (cur == 0u) { placed = true; break; }
                if (same_pos(pos, vout + 3ll * (cur - 1u))) {
                    atomicMin(&small[h], vi + 1u);
                    atomicAdd(ctr + 8, 1ull);
                    placed = true;
                    break;
                }
            }
            if (!placed) atomicOr(reinterpret_cast<unsigned int*>(ctr + 9), 1u);
        }
    }
}

// Face role: one thread per cell entry; CTA `bi` of `nb`.  Bound by the latency of
// its gathers: everything that a cell reads after its entry (the bitmap words,
// the vertex offsets of the four words its edges start in, its segment's
// offsets) is requested at once, so a cell costs two rounds of memory latency.
template <int EMIT_THREADS>
__device__ void emit_faces(const McGrid& g, const EmitArgs& a, unsigned bi, unsigned nb) {
    __shared__ unsigned long long tpk[256];  // packed triangle lists of the table
    __shared__ uint32_t vid[12][EMIT_THREADS];
    const uint32_t* __restrict__ S = a.S;
    const uint32_t* __restrict__ info = a.info;
    const unsigned long long* __restrict__ blk = a.blk;
    const unsigned long long* __restrict__ clist = a.clist;
    int32_t* __restrict__ fout = a.fout;
    for (int i = threadIdx.x; i < 256; i += EMIT_THREADS) tpk[i] = ISO_TRI_PACKED[g.method * 256 + i];
    __syncthreads();
    const unsigned long long n = min(a.ctr[10], (unsigned long long)a.capF);
    const uint32_t sxw = uint32_t(g.ny) * uint32_t(g.NW);
    const int tid = threadIdx.x;
    for (unsigned long long i = (unsigned long long)bi * EMIT_THREADS + tid; i < n;
         i += (unsigned long long)nb * EMIT_THREADS) {
        const unsigned long long e = clist[i];
        const uint32_t pw = uint32_t(e);
        const int b = int((e >> 32) & 31u);
        int x, y, w;
        word_xyw(g, pw, x, y, w);
        Words d;
        load_words(g, S, pw, x, y, w, d);
        // word w of the rows (dx, dy): vertex offset, and where its y and z edges start
        uint32_t base[4], inf[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t p = pw + uint32_t(q >> 1) * sxw + uint32_t(q & 1) * uint32_t(g.NW);
            inf[q] = info[p];
            base[q] = uint32_t(blk[2 * seg_of(g, p)]);
        }
        const unsigned long long fseg = blk[2 * seg_of(g, pw) + 1];
        const uint32_t zm = zmask(g, w);
        uint32_t c[8];
        corner_words(d, c);
        const uint32_t cs = case_at(c, b);
        const unsigned long long fo =
            fseg + (e >> 37) + word_faces(c, active_cells(d, zm) & ((1u << b) - 1u),
                                          [&](uint32_t q) { return uint32_t(tpk[q] >> 60); });
#pragma unroll
        for (int k = 0; k < 12; ++k) {
            const int ca = iso_edge_corner(2 * k), cb = iso_edge_corner(2 * k + 1);
            if (!(((cs >> ca) ^ (cs >> cb)) & 1u)) continue;
            const int ax = (cb - ca) == 4 ? 0 : ((cb - ca) == 2 ? 1 : 2);
            const int adx = ca >> 2, ady = (ca >> 1) & 1, adz = ca & 1, q = 2 * adx + ady;
            uint32_t off, m, below;
            if (adz && b == 31) {
                // the edge's low end lies in word w + 1 (at its bit 0)
                const uint32_t p = pw + uint32_t(adx) * sxw + uint32_t(ady) * uint32_t(g.NW) + 1u;
                const uint32_t in1 = info[p];
                off = uint32_t(blk[2 * seg_of(g, p)]) + (in1 & 0xfffffu);
                if (ax == 1) off += (in1 >> 20) & 63u;
                m = 0;
                below = 0;
            } else {
                off = base[q] + (inf[q] & 0xfffffu);
                if (ax >= 1) off += (inf[q] >> 20) & 63u;
                if (ax == 2) off += (inf[q] >> 26) & 63u;
                if (ax == 0) m = d.s[0][ady][0] ^ d.s[1][ady][0];
                else if (ax == 1) m = d.s[adx][0][0] ^ d.s[adx][1][0];
                else m = ez_of(d.s[adx][ady][0], d.s[adx][ady][1], zm);
                below = (1u << (b + adz)) - 1u;
            }
            vid[k][tid] = off + __popc(m & below);
        }
        unsigned long long pk = tpk[cs];
        const int ntc = int(pk >> 60);
        int32_t* f3 = fout + 3 * fo;
        for (int k = 0; k < ntc; ++k, pk >>= 12, f3 += 3) {
            f3[0] = int32_t(vid[pk & 15u][tid]);
            f3[1] = int32_t(vid[(pk >> 4) & 15u][tid]);
            f3[2] = int32_t(vid[(pk >> 8) & 15u][tid]);
        }
    }
}

// What the fix-up of V vertices and F faces keeps in the workspace.
struct FixLayout {
    uint32_t nb;        // words of a bitmap over the vertices
    uint32_t ntF, ntV;  // tiles of faces and of vertices
    uint32_t *moved, *suspect, *used;
    unsigned long long *fst, *vst;  // look-back states of the face and vertex tiles
    __device__ __forceinline__ FixLayout(const McWs& w, uint32_t V, uint32_t F) {
        nb = V / 32 + 1;
        ntF = (F + FIX_TILE - 1) / FIX_TILE;
        ntV = (V + FIX_TILE - 1) / FIX_TILE;
        moved = w.moved;
        suspect = w.vbits;
        used = w.vbits + nb;
        fst = w.fstate;
        vst = reinterpret_cast<unsigned long long*>(w.vbits + 2 * (size_t)nb);
    }
    __device__ __forceinline__ uint32_t vwords() const { return 2 * nb + 2 * ntV; }  // suspect, used, vst
};

template <int EMIT_THREADS>
__global__ void __launch_bounds__(EMIT_THREADS, 1280 / EMIT_THREADS) mc_emit(const McGrid g, const EmitArgs a) {
    iso::grid_wait();
    if (a.counts[0] > a.capV || a.counts[1] > a.capF || a.counts[0] > 0x7fffffffll) return;
    // the fix-up's bitmaps and look-back states (half a byte per vertex)
    {
        const FixLayout l(a.w, uint32_t(a.counts[0]), uint32_t(a.counts[1]));
        const uint32_t step = gridDim.x * EMIT_THREADS, i0 = blockIdx.x * EMIT_THREADS + threadIdx.x;
        for (uint32_t i = i0; i < l.nb; i += step) l.moved[i] = 0u;
        for (uint32_t i = i0; i < l.vwords(); i += step) l.suspect[i] = 0u;
        for (uint32_t i = i0; i < l.ntF; i += step) l.fst[i] = 0ull;
    }
    if (blockIdx.x < a.nbv) emit_vertices<EMIT_THREADS>(g, a, blockIdx.x, a.nbv);
    else emit_faces<EMIT_THREADS>(g, a, blockIdx.x - a.nbv, gridDim.x - a.nbv);
}

// ---------------------------------------------------------------------------
// 5. fix-up: when some vertex positions coincide (found by the emit's small
// hash; a value within FP32 rounding of the level at one grid point is enough,
// and a generic field on a fine grid has a few), merges the candidates by exact
// position (smallest index wins, as a sorted weld keeps the first), drops faces
// that became degenerate and vertices that no face uses any more, and compacts
// vertices and faces in place, keeping their order.
//
// One launch, its work cut into tiles that CTAs take by ticket, phase after
// phase; a tile waits (bounded) until the tiles of the phases before its own
// are done, so it only ever waits on tickets that running CTAs hold, and the
// launch needs no co-residency:
//   0, 1  (small hash full) clear the position table; candidates into it
//   2  each candidate's representative; `moved` bits of those that have another
//   3  faces: representatives for vertices, degenerate ones dropped (their
//      vertices become `suspect`: only those can be left without a face), the
//      rest compacted in place (look-back over tiles)
//   4  kept faces mark the suspects that they use
//   5  vertices: those neither moved nor left without a face, compacted in
//      place (look-back); their new indices
//   6  faces take the new indices
// Compaction in place: a tile's rows move to indices no higher than their own,
// and it writes only after every tile before it has published its count, for
// which that tile has read its rows.
// It is bound by latency: five dependent phases of L2 traffic, a few us each
// however small the mesh, about 100 MB for 1.6 M faces.  The fix-up by one CTA
// that it replaces was a serial chain of a block scan per 256 rows: 29.5 ms for
// a 512^3 sphere's 0.8 M vertices, against 61 us, and 3.4 ms against 31 us for
// 0.1 M.  Three CTAs per SM (one: 149 us, two: 85 us at the time), tickets taken
// ahead, and the emit clearing the bitmaps instead of a phase of their own
// (76 -> 61 us) gave the last factor of two.

struct FixArgs {
    McWs w;
    float* vout;
    int32_t* fout;
    long long* vedge;
    long long* counts;
    int* status;
    long long* host;  // optional: the sizes and the status for the host
    long long capV, capF;
};

__device__ __forceinline__ void fix_fail(int* status, volatile long long* host, int code) {
    atomicCAS(status, 0, code);
    if (host) host[2] = code;
}

__device__ __forceinline__ bool bit_of(const uint32_t* bits, uint32_t i) { return (bits[i >> 5] >> (i & 31u)) & 1u; }
__device__ __forceinline__ void set_bit(uint32_t* bits, uint32_t i) { atomicOr(&bits[i >> 5], 1u << (i & 31u)); }

// Smallest candidate at vertex v's position, or v.
__device__ __forceinline__ uint32_t fix_rep(const McWs& w, const float* vout, uint32_t v, bool big) {
    const float p[3] = {__ldcg(vout + 3ll * v), __ldcg(vout + 3ll * v + 1), __ldcg(vout + 3ll * v + 2)};
    const uint32_t mask = big ? w.HC - 1u : SMALL_HC - 1u;
    uint32_t h = phash(pbits(p[0]), pbits(p[1]), pbits(p[2])) & mask;
    for (uint32_t probe = 0; probe <= mask; ++probe, h = (h + 1) & mask) {
        const uint32_t j = big ? __ldcg(w.table + h) : __ldcg(w.small + h) - 1u;
        if (j == 0xffffffffu) break;
        if (same_pos(p, vout + 3ll * j)) return j;
    }
    return v;
}

// Candidate v into the position table; the smallest index wins.
__device__ __forceinline__ void fix_insert(const McWs& w, const float* vout, uint32_t v, int* status,
                                           volatile long long* host) {
    const float p[3] = {__ldcg(vout + 3ll * v), __ldcg(vout + 3ll * v + 1), __ldcg(vout + 3ll * v + 2)};
    const uint32_t mask = w.HC - 1u;
    uint32_t h = phash(pbits(p[0]), pbits(p[1]), pbits(p[2])) & mask;
    for (uint32_t probe = 0; probe <= mask; ++probe, h = (h + 1) & mask) {
        const uint32_t cur = atomicCAS(&w.table[h], 0xffffffffu, v);
        if (cur == 0xffffffffu) return;
        if (same_pos(p, vout + 3ll * cur)) {
            atomicMin(&w.table[h], v);
            return;
        }
    }
    fix_fail(status, host, int(ISO_ERR_OVERFLOW));
}

// Ordered compaction of a tile's kept rows (row k * FIX_THREADS + tid of the tile
// for k < FIX_PER): to[k] <- the row's index among all kept rows.  Call with
// every row read: the tile's count is published here.
__device__ __forceinline__ void fix_place(const bool* keep, unsigned long long* state, uint32_t tile, int* status,
                                          uint32_t (*wcnt)[FIX_THREADS / 32], unsigned long long* pre_s,
                                          unsigned long long* to) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t bal[FIX_PER];
#pragma unroll
    for (int k = 0; k < FIX_PER; ++k) {
        bal[k] = __ballot_sync(~0u, keep[k]);
        if (lane == 0) wcnt[k][warp] = __popc(bal[k]);
    }
    __syncthreads();
    uint32_t before[FIX_PER], run = 0;
#pragma unroll
    for (int k = 0; k < FIX_PER; ++k) {
        uint32_t mine = 0;
        for (int q = 0; q < FIX_THREADS / 32; ++q) {
            if (q == warp) mine = run;
            run += wcnt[k][q];
        }
        before[k] = mine + __popc(bal[k] & ((1u << lane) - 1u));
    }
    if (warp == 0) {
        unsigned long long e = 0, unused = 0;
        __threadfence();  // the tile's reads come before its count
        lb_tile(state, tile, run, 0, e, unused, status);
        __threadfence();
        if (lane == 0) *pre_s = e;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < FIX_PER; ++k) to[k] = *pre_s + before[k];
}

__global__ void __launch_bounds__(FIX_THREADS, FIX_CTAS) mc_fix(const FixArgs a) {
    __shared__ uint32_t wcnt[FIX_PER][FIX_THREADS / 32];
    __shared__ unsigned long long pre_s, ticket_s[2];
    __shared__ int ok_s;
    iso::grid_wait();
    const McWs& w = a.w;
    unsigned long long* ctr = w.ctr;
    const unsigned long long nsnap = min(ctr[1], (unsigned long long)a.capV);
    volatile long long* host = a.host;
    const bool first = host && blockIdx.x == 0 && threadIdx.x == 0;
    if (nsnap == 0 || (ctr[8] == 0 && ctr[9] == 0)) {
        if (first) {
            host[0] = a.counts[0];
            host[1] = a.counts[1];
            host[2] = *a.status;
        }
        return;
    }
    if (first && *a.status) host[2] = *a.status;  // the merge only ever adds a failure
    const bool big = ctr[9] != 0;
    const uint32_t V = uint32_t(ctr[4]), F = uint32_t(ctr[5]);
    const int tid = threadIdx.x;
    const FixLayout l(w, V, F);  // cleared by the emit
    uint32_t *moved = l.moved, *suspect = l.suspect, *used = l.used;
    unsigned long long *fst = l.fst, *vst = l.vst;
    const uint32_t ntF = l.ntF, ntV = l.ntV, ntS = uint32_t((nsnap + FIX_TILE - 1) / FIX_TILE);
    constexpr uint32_t CLEAR = 16 * FIX_TILE;  // words per tile of phase 0
    const unsigned long long nclear = big ? w.HC : 0u;
    // first ticket of each phase
    unsigned long long s[8];
    s[0] = 0;
    s[1] = s[0] + (nclear + CLEAR - 1) / CLEAR;
    s[2] = s[1] + (big ? ntS : 0u);
    s[3] = s[2] + ntS;
    s[4] = s[3] + ntF;
    s[5] = s[4] + ntF;
    s[6] = s[5] + ntV;
    s[7] = s[6] + (ntF ? ntF : 1u);
    // a CTA takes its next ticket while it works on one, and reports a tile done
    // while it goes on to the next: both atomics are off its critical path
    if (tid == 0) ticket_s[0] = atomicAdd(ctr + 12, 1ull);
    __syncthreads();
    unsigned long long t = ticket_s[0], met = 0;  // tiles known to be done
    for (int buf = 1;; buf ^= 1) {
        if (t >= s[7]) return;
        unsigned long long need = 0;  // tiles of the phases before this ticket's
#pragma unroll
        for (int p = 1; p < 7; ++p)
            if (t >= s[p]) need = s[p];
        if (need > met) {
            met = need;
            if (tid == 0) {
                int ok = 1;
                uint32_t spins = 0;
                while (*(volatile unsigned long long*)(ctr + 13) < need) {
                    if (++spins > ISO_SPIN_LIMIT) {
                        fix_fail(a.status, host, int(ISO_ERR_TIMEOUT));
                        ok = 0;
                        break;
                    }
                    __nanosleep(20);
                }
                __threadfence();
                ok_s = ok;
            }
            __syncthreads();
            if (!ok_s) return;
        }
        if (tid == 0) ticket_s[buf] = atomicAdd(ctr + 12, 1ull);
        if (t < s[1]) {
            for (unsigned long long i = t * CLEAR + tid; i < min(nclear, (t + 1) * CLEAR); i += FIX_THREADS)
                w.table[i] = 0xffffffffu;
        } else if (t < s[3]) {
            const bool insert = t < s[2];
            const unsigned long long b0 = (t - (insert ? s[1] : s[2])) * FIX_TILE;
            for (unsigned long long i = b0 + tid; i < min(nsnap, b0 + FIX_TILE); i += FIX_THREADS) {
                const uint32_t v = w.snaps[i];
                if (insert) {
                    fix_insert(w, a.vout, v, a.status, host);
                } else {
                    const uint32_t r = fix_rep(w, a.vout, v, big);
                    if (r != v) {
                        w.newidx[v] = r;
                        set_bit(moved, v);
                    }
                }
            }
        } else if (t < s[4]) {
            const uint32_t tile = uint32_t(t - s[3]);
            int32_t v3[FIX_PER][3];
            bool keep[FIX_PER];
#pragma unroll
            for (int k = 0; k < FIX_PER; ++k) {
                const uint32_t f = tile * FIX_TILE + k * FIX_THREADS + tid;
#pragma unroll
                for (int q = 0; q < 3; ++q) v3[k][q] = f < F ? __ldcg(a.fout + 3ull * f + q) : 0;
            }
#pragma unroll
            for (int k = 0; k < FIX_PER; ++k) {
                const uint32_t f = tile * FIX_TILE + k * FIX_THREADS + tid;
                keep[k] = false;
                if (f >= F) continue;
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    if (bit_of(moved, uint32_t(v3[k][q]))) v3[k][q] = int32_t(__ldcg(w.newidx + v3[k][q]));
                keep[k] = v3[k][0] != v3[k][1] && v3[k][0] != v3[k][2] && v3[k][1] != v3[k][2];
                if (!keep[k]) {
#pragma unroll
                    for (int q = 0; q < 3; ++q) set_bit(suspect, uint32_t(v3[k][q]));
                }
            }
            unsigned long long to[FIX_PER];
            fix_place(keep, fst, tile, a.status, wcnt, &pre_s, to);
#pragma unroll
            for (int k = 0; k < FIX_PER; ++k)
                if (keep[k]) {
                    int32_t* o = a.fout + 3 * to[k];
                    o[0] = v3[k][0]; o[1] = v3[k][1]; o[2] = v3[k][2];
                }
        } else if (t < s[5] || t >= s[6]) {
            const bool mark = t < s[5];
            const uint32_t Fk = ntF ? uint32_t((__ldcg(fst + ntF - 1) >> 31) & LB_MASK31) : 0u;  // faces kept
            const unsigned long long b0 = 3ull * FIX_TILE * (t - (mark ? s[4] : s[6]));
            uint32_t v[3 * FIX_PER];
#pragma unroll
            for (int k = 0; k < 3 * FIX_PER; ++k) {
                const unsigned long long i = b0 + k * FIX_THREADS + tid;
                v[k] = i < 3ull * Fk ? uint32_t(__ldcg(a.fout + i)) : 0u;
            }
            if (mark) {
#pragma unroll
                for (int k = 0; k < 3 * FIX_PER; ++k)
                    if (b0 + k * FIX_THREADS + tid < 3ull * Fk && bit_of(suspect, v[k]) && !bit_of(used, v[k]))
                        set_bit(used, v[k]);
            } else {
#pragma unroll
                for (int k = 0; k < 3 * FIX_PER; ++k) v[k] = __ldcg(w.newidx + v[k]);
#pragma unroll
                for (int k = 0; k < 3 * FIX_PER; ++k) {
                    const unsigned long long i = b0 + k * FIX_THREADS + tid;
                    if (i < 3ull * Fk) a.fout[i] = int32_t(v[k]);
                }
            }
            if (t == s[6] && tid == 0) {
                a.counts[0] = ntV ? (long long)((__ldcg(vst + ntV - 1) >> 31) & LB_MASK31) : 0;
                a.counts[1] = Fk;
                if (host) {
                    host[0] = a.counts[0];
                    host[1] = Fk;
                    if (*(volatile int*)a.status) host[2] = *(volatile int*)a.status;  // a look-back that gave up
                }
            }
        } else {
            const uint32_t tile = uint32_t(t - s[5]);
            float p[FIX_PER][3];
            long long e[FIX_PER];
            bool keep[FIX_PER];
#pragma unroll
            for (int k = 0; k < FIX_PER; ++k) {
                const uint32_t v = tile * FIX_TILE + k * FIX_THREADS + tid;
                keep[k] = v < V && F && !bit_of(moved, v) && !(bit_of(suspect, v) && !bit_of(used, v));
                e[k] = 0;
                if (!keep[k]) continue;
#pragma unroll
                for (int q = 0; q < 3; ++q) p[k][q] = __ldcg(a.vout + 3ull * v + q);
                if (a.vedge) e[k] = __ldcg(a.vedge + v);
            }
            unsigned long long to[FIX_PER];
            fix_place(keep, vst, tile, a.status, wcnt, &pre_s, to);
#pragma unroll
            for (int k = 0; k < FIX_PER; ++k)
                if (keep[k]) {
                    w.newidx[tile * FIX_TILE + k * FIX_THREADS + tid] = uint32_t(to[k]);
                    float* o = a.vout + 3 * to[k];
                    o[0] = p[k][0]; o[1] = p[k][1]; o[2] = p[k][2];
                    if (a.vedge) a.vedge[to[k]] = e[k];
                }
        }
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            atomicAdd(ctr + 13, 1ull);
        }
        t = ticket_s[buf];
    }
}

// ---------------------------------------------------------------------------
// 1. sign bitmap

constexpr int SIGN_BLOCK = 256;

// Bit z % 32 of word [(x * ny + y) * NW + z / 32] is (v - level < 0).  A warp has
// 32 coalesced 128-byte loads in flight before their ballots, and lane w keeps
// word w so that the words leave in one store.  Bound by HBM on large grids; a
// warp per row, as before, had only a short row's loads in flight.
// Both kernels clear `zero` (the counters, look-back states and small hash of
// the call start at zero).

// Rows that fill their words (nz a multiple of 32): 32 consecutive words are
// 1024 consecutive values.  192^3: 17.4 us before, 11.7 now; 256^3 24.7 and 16.8;
// 512^3 82.6 and 82.
__global__ void __launch_bounds__(SIGN_BLOCK) mc_signs(const float* __restrict__ vals, unsigned long long PW,
                                                       float level, uint32_t* __restrict__ out,
                                                       unsigned long long* __restrict__ zero, long long nzero) {
    iso::grid_wait();
    for (long long i = (long long)blockIdx.x * SIGN_BLOCK + threadIdx.x; i < nzero;
         i += (long long)gridDim.x * SIGN_BLOCK)
        zero[i] = 0ull;
    const uint32_t lane = threadIdx.x & 31;
    const unsigned long long step = (unsigned long long)gridDim.x * SIGN_BLOCK;  // 32 words per warp
    for (unsigned long long base = ((unsigned long long)blockIdx.x * (SIGN_BLOCK / 32) + (threadIdx.x >> 5)) * 32;
         base < PW; base += step) {
        const float* q = vals + 32 * base + lane;
        const uint32_t n = uint32_t(min(PW - base, 32ull));
        float v[32];
#pragma unroll
        for (int u = 0; u < 32; ++u) v[u] = u < n ? __ldcs(q + 32 * u) : level;  // read once: evict first
        uint32_t mine = 0;
#pragma unroll
        for (int u = 0; u < 32; ++u) {
            const uint32_t b = __ballot_sync(~0u, iso::below(v[u], level));
            if (uint32_t(u) == lane) mine = b;
        }
        if (lane < n) out[base + lane] = mine;
    }
}

// Other rows: R of them at a time, W words of each (R * W = 32, W >= NW, or W = 32
// and a row's words 32 at a time).  Carrying the place in the row from word to
// word instead would keep all loads of short rows busy, but its address arithmetic
// made it issue-bound on long ones (400 x 400 x 507: 77 us against 53).
template <int R, int W>
__global__ void __launch_bounds__(SIGN_BLOCK) mc_signs_rows(const float* __restrict__ vals, long long rows, int nz,
                                                            int NW, float level, uint32_t* __restrict__ out,
                                                            unsigned long long* __restrict__ zero, long long nzero) {
    static_assert(R * W == 32, "a word per lane");
    iso::grid_wait();
    for (long long i = (long long)blockIdx.x * SIGN_BLOCK + threadIdx.x; i < nzero;
         i += (long long)gridDim.x * SIGN_BLOCK)
        zero[i] = 0ull;
    const int lane = threadIdx.x & 31;
    const long long step = (long long)gridDim.x * (SIGN_BLOCK / 32) * R;
    for (long long row = ((long long)blockIdx.x * (SIGN_BLOCK / 32) + (threadIdx.x >> 5)) * R; row < rows;
         row += step) {
        for (int wb = 0; wb < NW; wb += W) {
            float v[32];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float* q = vals + (row + r) * nz + 32 * wb + lane;
                const int left = row + r < rows ? nz - 32 * wb - lane : 0;  // values of the row from the lane's on
#pragma unroll
                for (int w = 0; w < W; ++w) v[r * W + w] = 32 * w < left ? __ldcs(q + 32 * w) : level;
            }
            uint32_t mine = 0;
#pragma unroll
            for (int u = 0; u < 32; ++u) {
                const uint32_t b = __ballot_sync(~0u, iso::below(v[u], level));
                if (u == lane) mine = b;
            }
            const int r = lane / W, w = wb + lane % W;
            if (row + r < rows && w < NW) out[(row + r) * NW + w] = mine;
        }
    }
}

std::mutex g_mu;
int g_block = 256;

// Threads of a count CTA.
int count_threads() { return iso::tune_get(iso::TUNE_MC_COUNT_THREADS) == 128 ? 128 : 256; }

// Point words up to which a count thread takes one word instead of four: four
// times as many CTAs, for grids whose CTAs of four words per thread would not
// fill the GPU.  32^3 in one CTA of 1024 words took 21 us and takes 9 in four;
// 128^3 15 and 10.  From 2^18 words on (200 x 330 x 143 and 256^3) the scan that
// the last CTA then no longer does costs what the count gains: 13 + 4 against 16 us.
constexpr long long FINE_PW = 1ll << 18;

template <int EMIT_THREADS>
int launch_emit(const McParams& p, const McGrid& g, const McWs& w, cudaStream_t st, int sms) {
    static int per = -1;
    if (per < 0) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, mc_emit<EMIT_THREADS>, EMIT_THREADS, 0);
    // entries are a fraction of the capacities; the loops are grid-stride.  The
    // resident CTAs are split between the roles in proportion to the work
    // (a vertex costs about half a cell).
    const long long resident = (long long)sms * std::max(per, 1);
    const auto want = [&](long long cap) { return std::max<long long>(1, (cap + EMIT_THREADS - 1) / EMIT_THREADS); };
    const long long nbv = std::max<long long>(1, std::min(want(p.capV), resident / 3));
    const long long nbf = std::max<long long>(1, std::min(want(p.capF), resident - nbv));
    EmitArgs a{p.vals, w.S, w.info, w.blk, w.vlist, w.clist, w.ctr, w.snaps, w.small,
               p.vout, p.fout, p.counts, p.status, p.capV, p.capF, unsigned(nbv), w, p.vedge};
    {
        iso::ProfScope ps("mc_emit", st);
        iso::launch_pdl(mc_emit<EMIT_THREADS>, unsigned(nbv + nbf), EMIT_THREADS, st, g, a);
        if (cudaGetLastError() != cudaSuccess) return iso::fail_code(ISO_ERR_CUDA);
    }
    {
        iso::ProfScope ps("mc_fix", st);
        const FixArgs f{w, p.vout, p.fout, p.vedge, p.counts, p.status, p.host, p.capV, p.capF};
        const long long tiles = std::max<long long>(1, (std::max(p.capV, p.capF) + FIX_TILE - 1) / FIX_TILE);
        iso::launch_pdl(mc_fix, unsigned(std::min<long long>(tiles, (long long)sms * FIX_CTAS)), unsigned(FIX_THREADS), st, f);
        if (cudaGetLastError() != cudaSuccess) return iso::fail_code(ISO_ERR_CUDA);
    }
    return 0;
}

// ct: the threads of a count CTA that g.lgseg was made from.
int launch_count_emit(const McParams& p, const McGrid& g, const McWs& w, int ct, cudaStream_t st) {
    const int sms = iso::sm_count();
    const uint32_t nseg = uint32_t((g.PW + (1ll << g.lgseg) - 1) >> g.lgseg);
    {
        iso::ProfScope ps("mc_count", st);
        const bool fine = (1 << g.lgseg) == ct;  // one word per thread
        const long long ncoord = (long long)p.nx + p.ny + p.nz;
        const long long grid = std::max<long long>(nseg, (ncoord + ct - 1) / ct);
        const auto kernel = fine ? (ct == 128 ? mc_count<128, 1> : mc_count<256, 1>)
                                 : (ct == 128 ? mc_count<128, WPT_MAX> : mc_count<256, WPT_MAX>);
        iso::launch_pdl(kernel, unsigned(grid), unsigned(ct), st, g, p.amin[0], p.amin[1], p.amin[2], p.asize[0],
                        p.asize[1], p.asize[2], w.S, w.info, w.blk, w.vlist, w.clist, w.ctr, w.gc, nseg, p.capV, p.capF,
                        p.counts, p.status);
        if (cudaGetLastError() != cudaSuccess) return iso::fail_code(ISO_ERR_CUDA);
    }
    if (nseg > uint32_t(SCAN_LAST * ct)) {
        iso::ProfScope ps("mc_scan", st);
        const uint32_t nchunk = (nseg + SCAN_THREADS - 1) / SCAN_THREADS;
        iso::launch_pdl(mc_scan, nchunk, SCAN_THREADS, st, w.blk, nseg, w.ctr, w.state, p.counts, p.status, p.capV,
                   p.capF);
        if (cudaGetLastError() != cudaSuccess) return iso::fail_code(ISO_ERR_CUDA);
    }
    const int block = mc_get_block();
    return block == 128 ? launch_emit<128>(p, g, w, st, sms) : launch_emit<256>(p, g, w, st, sms);
}

}  // namespace

int mc_set_block(int threads) {
    if (threads != 128 && threads != 256) return iso::fail_code(ISO_ERR_ARG);
    std::lock_guard<std::mutex> lk(g_mu);
    g_block = threads;
    return 0;
}

int mc_get_block() {
    std::lock_guard<std::mutex> lk(g_mu);
    return g_block;
}

void mc_signs_launch(const float* vals, int nx, int ny, int nz, float level, uint32_t* out,
                     cudaStream_t st, unsigned long long* zero, long long nzero) {
    const int NW = (nz + 31) / 32;
    const long long rows = (long long)nx * ny, most = (long long)iso::sm_count() * iso::tune_get(iso::TUNE_MC_SIGN_CTAS);
    const auto ctas = [&](long long warps) {
        constexpr int per = SIGN_BLOCK / 32;
        return unsigned(std::max<long long>(1, std::min<long long>((warps + per - 1) / per, most)));
    };
    if (nz % 32 == 0) {
        const unsigned long long PW = (unsigned long long)rows * NW;
        iso::launch_pdl(mc_signs, ctas((long long)((PW + 31) / 32)), SIGN_BLOCK, st, vals, PW, level, out, zero, nzero);
        return;
    }
    const int R = NW <= 1 ? 32 : NW <= 2 ? 16 : NW <= 4 ? 8 : NW <= 8 ? 4 : NW <= 16 ? 2 : 1;
    const auto kernel = R == 32 ? mc_signs_rows<32, 1> : R == 16 ? mc_signs_rows<16, 2>
                        : R == 8 ? mc_signs_rows<8, 4> : R == 4 ? mc_signs_rows<4, 8>
                        : R == 2 ? mc_signs_rows<2, 16> : mc_signs_rows<1, 32>;
    iso::launch_pdl(kernel, ctas((rows + R - 1) / R), SIGN_BLOCK, st, vals, rows, nz, NW, level, out, zero, nzero);
}

// Bound on t for an edge vertex to land within a few ulps of an endpoint (the
// only place two edges' vertices can meet).  The lerp (1 - t) a + t b is off
// by at most ~2 ulps of max(|a|, |b|) per coordinate, so a vertex comes that
// close to an endpoint only if t * h <= 2^-22 * max|coord| (h the spacing);
// tau = 2^-20 * (1 + max|coord| / h) keeps a factor of 4 on that, and the same
// holds for 1 - t.
float snap_tau_box(int nx, int ny, int nz, const float* amin_, const float* asize) {
    const int n[3] = {nx, ny, nz};
    double r = 0;
    for (int k = 0; k < 3; ++k) {
        const double amin = amin_[k], amax = double(amin_[k]) + double(asize[k]);
        const double size = asize[k];
        const double m = std::max(std::fabs(amin), std::fabs(amax));
        if (size == 0.0 || !std::isfinite(size)) return 1.0f;
        r = std::max(r, m * double(std::max(n[k] - 1, 1)) / std::fabs(size));
    }
    const double tau = std::ldexp(1.0, -20) * (1.0 + r);
    return tau >= 0.5 ? 1.0f : float(tau);
}

float snap_tau(const McParams& p) { return snap_tau_box(p.nx, p.ny, p.nz, p.amin, p.asize); }

size_t mc_workspace_bytes(int nx, int ny, int nz, long long capV, long long capF) {
    return carve(nx, ny, nz, capV, capF, nullptr).total;
}

int mc_launch(const McParams& params, void* ws, size_t ws_bytes, cudaStream_t st) {
    McParams p = params;
    const McWs w0 = carve(p.nx, p.ny, p.nz, p.capV, p.capF, nullptr);
    if (ws_bytes < w0.total) return iso::fail_code(ISO_ERR_WORKSPACE);
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~uintptr_t(255));
    McWs w = carve(p.nx, p.ny, p.nz, p.capV, p.capF, base);
    if (!p.counts) p.counts = reinterpret_cast<long long*>(w.ctr + 2);  // cleared by the sign pass
    if (!p.status) p.status = reinterpret_cast<int*>(w.ctr + 14);
    McGrid g;
    g.nx = p.nx; g.ny = p.ny; g.nz = p.nz;
    g.NW = (p.nz + 31) / 32;
    g.dNW = make_fastdiv(uint32_t(g.NW));
    g.dNY = make_fastdiv(uint32_t(g.ny));
    g.PW = (long long)p.nx * p.ny * g.NW;
    g.level = p.level;
    g.method = p.method;
    g.tau = snap_tau(p);
    g.fma = iso::arith_fma();
    const bool fine = g.PW <= FINE_PW;
    const int ct = count_threads();  // read once: another thread may set it while this one launches
    g.lgseg = (ct == 128 ? 7 : 8) + (fine ? 0 : 2);
    if (fine) w.blk = w.blk2;
    g.gc = w.gc;
    if (g.PW > 0xffffffffll) return iso::fail_code(ISO_ERR_ARG);
    {
        iso::ProfScope ps("mc_signs", st);
        mc_signs_launch(p.vals, p.nx, p.ny, p.nz, p.level, w.S, st, w.ctr, (long long)(zeroed_bytes(w.nBlk) / 8));
        if (cudaGetLastError() != cudaSuccess) return iso::fail_code(ISO_ERR_CUDA);
    }
    const int rc = launch_count_emit(p, g, w, ct, st);
    if (rc) return rc;
    return 0;
}

// Test hook of the bounded waits (no counterpart in isoext): runs the scan's
// look-back for chunk 32 over `state` (device, >= 32 zeroed u64, never
// published) with a limit of spin_limit polls; *status (device) becomes
// ISO_ERR_TIMEOUT and the kernel returns.  spin_limit <= 2^20.
extern "C" int iso_test_wait_timeout(unsigned spin_limit, unsigned long long* state, int* status,
                                     unsigned long long* out, void* stream) {
    if (!state || !status || !out || spin_limit > (1u << 20)) return iso::fail_code(ISO_ERR_ARG);
    lookback_probe<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(state, 32u, spin_limit, status, out);
    return cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
}
