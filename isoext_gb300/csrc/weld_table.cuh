// Exact-position weld of dual vertices through a hash table, for the one-call
// dual contouring of boxes whose grid coordinates may repeat (spacing near FP32
// resolution, a box of no extent).  Elsewhere a vertex on a face of its cell's box
// can only equal the vertices of the at most eight cells around it, which the
// local searches look at (dc_weld_faces, sd_flags); where coordinates repeat those
// cells can be any number up to the whole grid for every vertex, and the table
// takes its place: work in the number of vertices whatever the coordinates.  Elsewhere
// the search is the faster one (a call of 256^3 CSG 110 us against 118 with the
// table, 512^3 sphere 281 and 289, the sparse band of 200^3 124 and 131).
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "common.cuh"
#include "dc_common.cuh"

namespace {

// Whether neighbouring grid coordinates may be equal.  A coordinate's rounding stays
// below 5 * 2^-24 of the box's magnitude m (the quotient, times an extent of at
// most 2 m, and the sum), so coordinates h > 2^-20 m apart stay distinct, on both
// readings of the arithmetic; not so for a NaN or infinite box.
bool coords_may_repeat(const Grid3& g) {
    const int n[3] = {g.nx, g.ny, g.nz};
    for (int k = 0; k < 3; ++k) {
        const double lo = g.amin[k], size = g.asize[k];
        const double m = std::max(std::fabs(lo), std::fabs(lo + size)), h = std::fabs(size) / std::max(n[k] - 1, 1);
        if (!(h > std::ldexp(m, -20) + std::ldexp(1.0, -145))) return true;
    }
    return false;
}

// Slots hold the smallest vertex of their position; twice as many as vertices, so
// an empty one always ends a probe.  slot == nullptr: the local search is used.
struct WeldTable {
    uint32_t* slot;
    uint32_t size;
};

constexpr uint32_t TABLE_EMPTY = 0xffffffffu;

__device__ __forceinline__ bool same_position(const float* dual, uint32_t a, uint32_t b) {
    return iso::pos_bits(dual[3ll * a]) == iso::pos_bits(dual[3ll * b]) &&
           iso::pos_bits(dual[3ll * a + 1]) == iso::pos_bits(dual[3ll * b + 1]) &&
           iso::pos_bits(dual[3ll * a + 2]) == iso::pos_bits(dual[3ll * b + 2]);
}

__device__ __forceinline__ uint32_t table_start(const WeldTable& t, const float* dual, uint32_t a) {
    return __umulhi(iso::pos_hash(iso::pos_bits(dual[3ll * a]), iso::pos_bits(dual[3ll * a + 1]),
                                  iso::pos_bits(dual[3ll * a + 2])),
                    t.size);
}

// The smallest vertex at vertex a's position (a itself when it was not inserted).
__device__ __forceinline__ uint32_t table_first(const WeldTable& t, const float* dual, uint32_t a) {
    uint32_t h = table_start(t, dual, a);
    for (uint32_t p = 0; p < t.size; ++p, h = h + 1 < t.size ? h + 1 : 0u) {
        const uint32_t b = t.slot[h];
        if (b == TABLE_EMPTY) break;
        if (same_position(dual, a, b)) return b;
    }
    return a;
}

// The vertices on faces into the table: those of used[a] & need == need with face[a] set
// (face may be null).
__global__ void __launch_bounds__(256) weld_table_insert(const WeldTable t, const float* __restrict__ dual,
                                                         const uint8_t* __restrict__ used, uint32_t need,
                                                         const uint8_t* __restrict__ face,
                                                         const long long* __restrict__ eff) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= eff[0] || (used[i] & need) != need || (face && !face[i])) return;
    const uint32_t a = uint32_t(i);
    uint32_t h = table_start(t, dual, a);
    for (uint32_t p = 0; p < t.size; ++p, h = h + 1 < t.size ? h + 1 : 0u) {
        const uint32_t b = atomicCAS(t.slot + h, TABLE_EMPTY, a);
        if (b == TABLE_EMPTY) return;
        if (same_position(dual, a, b)) {
            if (a < b) atomicMin(t.slot + h, a);
            return;
        }
    }
}

// Slots for up to cap vertices (8 bytes each; there are never 2^31 of them).
uint32_t weld_table_size(long long cap) { return uint32_t(2 * std::min(cap, 0x7fffffffll)); }

// Empties the table and inserts the vertices of up to cap cells.
cudaError_t launch_weld_table(const WeldTable& t, const float* dual, const uint8_t* used, uint32_t need,
                              const uint8_t* face, const long long* eff, long long cap, cudaStream_t st) {
    const cudaError_t e = cudaMemsetAsync(t.slot, 0xff, size_t(t.size) * 4, st);
    if (e != cudaSuccess) return e;
    weld_table_insert<<<blocks_for(cap, 256), 256, 0, st>>>(t, dual, used, need, face, eff);
    return cudaSuccess;
}

}  // namespace
