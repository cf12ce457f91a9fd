// Grid values of a union of spheres and boxes, evaluated in one pass.
//
// The served request stream describes each grid by such a union; evaluating it
// here writes the grid once (HBM-bound) instead of building it from a chain of
// tensor operations.  Point positions use the grid's own arithmetic
// (include/utils.cuh:62-80 of isoext, iso::grid_coord); each primitive's
// distance is the formula of isoext's sdf module (src/isoext/sdf.py:70-116):
// sphere |p - c| - r, box |max(q, 0)| + min(max(q), 0) with q = |p - c| - h.
#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "profile.cuh"

namespace {

constexpr int MAX_PRIMS = 32;

// Union distances of Z points of a row over the primitives in set: a primitive's
// parameters and everything of it that does not depend on z are taken once for
// all of them.  Every operation is rounded on its own, in the order of the
// formulas.
template <int Z>
__device__ __forceinline__ void union_points(const float (*pr)[7], uint32_t set, float px, float py, const float* pz,
                                             float* d) {
#pragma unroll
    for (int j = 0; j < Z; ++j) d[j] = 3.402823466e38f;
    for (; set; set &= set - 1) {
        const int k = __ffs(set) - 1;
        const float dx = __fsub_rn(px, pr[k][1]), dy = __fsub_rn(py, pr[k][2]), cz = pr[k][3];
        if (pr[k][0] == 0.0f) {
            const float xy = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), r = pr[k][4];
#pragma unroll
            for (int j = 0; j < Z; ++j) {
                const float dz = __fsub_rn(pz[j], cz);
                d[j] = fminf(d[j], __fsub_rn(__fsqrt_rn(__fadd_rn(xy, __fmul_rn(dz, dz))), r));
            }
        } else {
            const float qx = __fsub_rn(fabsf(dx), pr[k][4]), qy = __fsub_rn(fabsf(dy), pr[k][5]), hz = pr[k][6];
            const float ox = fmaxf(qx, 0.0f), oy = fmaxf(qy, 0.0f);
            const float xy = __fadd_rn(__fmul_rn(ox, ox), __fmul_rn(oy, oy)), qxy = fmaxf(qx, qy);
#pragma unroll
            for (int j = 0; j < Z; ++j) {
                const float qz = __fsub_rn(fabsf(__fsub_rn(pz[j], cz)), hz), oz = fmaxf(qz, 0.0f);
                const float outside = __fsqrt_rn(__fadd_rn(xy, __fmul_rn(oz, oz)));
                d[j] = fminf(d[j], __fadd_rn(outside, fminf(fmaxf(qxy, qz), 0.0f)));
            }
        }
    }
}

template <int Z>
__device__ __forceinline__ void union_run(const float (*pr)[7], uint32_t set, float px, float py, int z, int nz, float az,
                                          float sz, bool fma, float* __restrict__ orow) {
    float pz[Z], d[Z];
#pragma unroll
    for (int j = 0; j < Z; ++j) pz[j] = iso::grid_coord(uint32_t(min(z + 32 * j, nz - 1)), uint32_t(nz), az, sz, fma);
    union_points<Z>(pr, set, px, py, pz, d);
#pragma unroll
    for (int j = 0; j < Z; ++j)
        if (z + 32 * j < nz) orow[z + 32 * j] = d[j];
}

// The primitives, in shared memory; returns their number.
__device__ __forceinline__ int load_prims(const float* __restrict__ prims, float (*pr)[7], int* np) {
    if (threadIdx.x == 0) *np = min(max(int(prims[0]), 0), MAX_PRIMS);
    __syncthreads();
    for (int i = threadIdx.x; i < *np * 7; i += blockDim.x) pr[i / 7][i % 7] = prims[1 + i];
    __syncthreads();
    return *np;
}

__device__ __forceinline__ uint32_t all_prims(int np) { return np >= 32 ? ~0u : (1u << np) - 1u; }

// prims: [0] = count (as a float), then count rows of 7 floats: kind (0 sphere,
// 1 box), centre x y z, radius | half-extents x y z.
// Bound by instruction issue.  Four points per lane share a primitive's shared
// memory reads, its branch and its x and y terms: one point per lane issued some
// 45 instructions per primitive and point.  Leaving out square roots that cannot
// lower the minimum (compared squared) was slower: a warp takes the branch when
// any of its lanes does.
__global__ void __launch_bounds__(256) sdf_union_grid(const float* __restrict__ prims, int nx, int ny, int nz,
                                                      float ax, float ay, float az, float sx, float sy, float sz,
                                                      bool fma, float* __restrict__ out) {
    __shared__ float pr[MAX_PRIMS][7];
    __shared__ int np_s;
    const uint32_t set = all_prims(load_prims(prims, pr, &np_s));
    // a warp per grid row (x, y), its lanes along z: the row's coordinates once,
    // consecutive lanes store consecutive values
    const int lane = threadIdx.x & 31;
    const long long rows = (long long)nx * ny;
    const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); row < rows;
         row += nwarps) {
        const int y = int(row % ny), x = int(row / ny);
        const float px = iso::grid_coord(uint32_t(x), uint32_t(nx), ax, sx, fma);
        const float py = iso::grid_coord(uint32_t(y), uint32_t(ny), ay, sy, fma);
        float* orow = out + row * nz;
        int z0 = 0;
        for (; nz - z0 > 64; z0 += 128) union_run<4>(pr, set, px, py, z0 + lane, nz, az, sz, fma, orow);
        if (nz - z0 > 32) union_run<2>(pr, set, px, py, z0 + lane, nz, az, sz, fma, orow);
        else if (nz > z0) union_run<1>(pr, set, px, py, z0 + lane, nz, az, sz, fma, orow);
    }
}

// The primitives that can be nearest somewhere in a box, lane k looking at
// primitive k.  A primitive's distance changes by at most r between the box's
// centre c and any of its points (both formulas are 1-Lipschitz, negative radii
// and extents included), r half the box's diagonal.  One whose distance at c
// exceeds another's by more than 2 r and both roundings stays above that other
// everywhere in the box, and the minimum is the same bits without it.  The
// formulas' rounding stays below 1e-6 of the magnitudes that enter (m), and
// squares that underflow lose less than 1e-18; both are taken ten times over.
// Not finite or above 1e18, where squares overflow: neither left out nor a reason
// to leave out (every comparison with NaN fails).
__device__ __forceinline__ uint32_t near_prims(const float (*pr)[7], int np, const float* c, float r, float m) {
    const int lane = threadIdx.x & 31;
    float lo = 0.0f, hi = 3.402823466e38f;
    bool known = false;
    if (lane < np) {
        float d;
        const float zero[1] = {c[2]};
        union_points<1>(pr, 1u << lane, c[0], c[1], zero, &d);
        const float* q = pr[lane];
        m += fabsf(q[1]) + fabsf(q[2]) + fabsf(q[3]) + fabsf(q[4]);
        if (q[0] != 0.0f) m += fabsf(q[5]) + fabsf(q[6]);
        known = fabsf(d) <= 1e18f && m <= 1e18f && r <= 1e18f;
        if (known) {
            const float e = 1.001f * r + 1e-5f * m + 1e-17f;
            lo = d - e;
            hi = d + e;
        }
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) hi = fminf(hi, __shfl_xor_sync(~0u, hi, o));
    return __ballot_sync(~0u, lane < np && !(known && lo > hi));
}

// The same values for large grids: a warp takes tiles of 32 z by 4 y by 4 x (lanes
// 8 z by 4 y, four points z + 8 j each), and only the primitives that can be
// nearest in a tile: of ten random ones on 256^3 about three are left.  256^3 of 1,
// 4, 10 and 16 primitives 36, 66, 131 and 193 us by rows, 32, 46, 60 and 63 by
// tiles, a CTA per eight tiles (on a resident grid 34, 50, 66 and 69: tiles differ
// in their primitives).
constexpr int TILE_X = 4;

__global__ void __launch_bounds__(256) sdf_union_tiles(const float* __restrict__ prims, int nx, int ny, int nz,
                                                       float ax, float ay, float az, float sx, float sy, float sz,
                                                       bool fma, float* __restrict__ out) {
    __shared__ float pr[MAX_PRIMS][7];
    __shared__ int np_s;
    const int np = load_prims(prims, pr, &np_s);
    const int lane = threadIdx.x & 31, lz = lane & 7, ly = lane >> 3;
    const uint32_t tz = uint32_t(nz + 31) / 32u, ty = uint32_t(ny + 3) / 4u, tx = uint32_t(nx + TILE_X - 1) / TILE_X;
    const uint32_t tiles = tx * ty * tz;  // a few dozen points each at least (ny >= 4, nz >= 17): below 2^32 for any grid that fits
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < tiles; t += nwarps) {
        const int z0 = int(t % tz) * 32, y0 = int((t / tz) % ty) * 4, x0 = int(t / tz / ty) * TILE_X;
        float pz[4], px[TILE_X];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            pz[j] = iso::grid_coord(uint32_t(min(z0 + lz + 8 * j, nz - 1)), uint32_t(nz), az, sz, fma);
        const float py = iso::grid_coord(uint32_t(min(y0 + ly, ny - 1)), uint32_t(ny), ay, sy, fma);
#pragma unroll
        for (int i = 0; i < TILE_X; ++i) px[i] = iso::grid_coord(uint32_t(min(x0 + i, nx - 1)), uint32_t(nx), ax, sx, fma);
        // the tile's box: its first and last coordinates
        const float f[3] = {px[0], __shfl_sync(~0u, py, 0), __shfl_sync(~0u, pz[0], 0)};
        const float l[3] = {px[TILE_X - 1], __shfl_sync(~0u, py, 31), __shfl_sync(~0u, pz[3], 31)};
        float c[3], r = 0.0f, m = 0.0f;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            c[q] = 0.5f * f[q] + 0.5f * l[q];
            const float h = 0.5f * l[q] - 0.5f * f[q];
            r += h * h;
            m += fabsf(f[q]) + fabsf(l[q]);
        }
        const uint32_t set = near_prims(pr, np, c, sqrtf(r), m);
        const int y = y0 + ly;
#pragma unroll 1
        for (int i = 0; i < min(TILE_X, nx - x0); ++i) {
            float p0 = px[0];
#pragma unroll
            for (int q = 1; q < TILE_X; ++q) p0 = q == i ? px[q] : p0;
            float d[4];
            union_points<4>(pr, set, p0, py, pz, d);
            if (y >= ny) continue;
            float* o = out + ((long long)(x0 + i) * ny + y) * nz + z0 + lz;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (z0 + lz + 8 * j < nz) o[8 * j] = d[j];
        }
    }
}

}  // namespace

extern "C" {

// prims: DEVICE float [1 + 7 * count]: prims[0] = count (1 .. 32, as a float),
// then count rows of kind (0 sphere, 1 box), centre xyz, radius | half-extents
// xyz.  Reading the primitives from device memory lets a captured graph
// evaluate a new union after an upload.  out: device float [nx, ny, nz].  No
// counterpart in isoext (it builds grids with torch).
int iso_sdf_union_grid(const float* prims, int nx, int ny, int nz, const float* aabb_min, const float* aabb_max,
                       float* out, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (nx < 1 || ny < 1 || nz < 1 || !prims || !out || !aabb_min || !aabb_max) return iso::fail_code(ISO_ERR_ARG);
    iso::ProfScope ps("sdf_union_grid", st);
    // By tiles where a tile's points are grid points and the tiles fill the SMs
    // (128^3: 24 us by rows, 22 by tiles; below, rows: 97^3 10.8 against 11.4).
    if (ny >= 4 && nz >= 17 && (long long)nx * ny * nz >= (1ll << 21)) {
        const long long tiles = (long long)((nx + TILE_X - 1) / TILE_X) * ((ny + 3) / 4) * ((nz + 31) / 32);
        sdf_union_tiles<<<unsigned(std::min<long long>((tiles + 7) / 8, 1 << 24)), 256, 0, st>>>(
            prims, nx, ny, nz, aabb_min[0], aabb_min[1], aabb_min[2], aabb_max[0] - aabb_min[0],
            aabb_max[1] - aabb_min[1], aabb_max[2] - aabb_min[2], iso::arith_fma(), out);
    } else {
        const long long rows = (long long)nx * ny;  // a warp each, 8 per CTA
        const long long grid = std::max<long long>(1, std::min<long long>((rows + 7) / 8, (long long)iso::sm_count() * 8));
        sdf_union_grid<<<unsigned(grid), 256, 0, st>>>(prims, nx, ny, nz, aabb_min[0], aabb_min[1], aabb_min[2],
                                                       aabb_max[0] - aabb_min[0], aabb_max[1] - aabb_min[1],
                                                       aabb_max[2] - aabb_min[2], iso::arith_fma(), out);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
}

}  // extern "C"
