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

// Union distances of Z points of a row, z = z0 + 32 j: a primitive's parameters
// and everything of it that does not depend on z are taken once for all of them.
// Every operation is rounded on its own, in the order of the formulas.
template <int Z>
__device__ __forceinline__ void union_points(const float (*pr)[7], int np, float px, float py, const float* pz,
                                             float* d) {
#pragma unroll
    for (int j = 0; j < Z; ++j) d[j] = 3.402823466e38f;
    for (int k = 0; k < np; ++k) {
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
__device__ __forceinline__ void union_run(const float (*pr)[7], int np, float px, float py, int z, int nz, float az,
                                          float sz, bool fma, float* __restrict__ orow) {
    float pz[Z], d[Z];
#pragma unroll
    for (int j = 0; j < Z; ++j) pz[j] = iso::grid_coord(uint32_t(min(z + 32 * j, nz - 1)), uint32_t(nz), az, sz, fma);
    union_points<Z>(pr, np, px, py, pz, d);
#pragma unroll
    for (int j = 0; j < Z; ++j)
        if (z + 32 * j < nz) orow[z + 32 * j] = d[j];
}

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
    __shared__ int np;
    if (threadIdx.x == 0) np = min(max(int(prims[0]), 0), MAX_PRIMS);
    __syncthreads();
    for (int i = threadIdx.x; i < np * 7; i += blockDim.x) pr[i / 7][i % 7] = prims[1 + i];
    __syncthreads();
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
        for (; nz - z0 > 64; z0 += 128) union_run<4>(pr, np, px, py, z0 + lane, nz, az, sz, fma, orow);
        if (nz - z0 > 32) union_run<2>(pr, np, px, py, z0 + lane, nz, az, sz, fma, orow);
        else if (nz > z0) union_run<1>(pr, np, px, py, z0 + lane, nz, az, sz, fma, orow);
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
    const long long rows = (long long)nx * ny;  // a warp each, 8 per CTA
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long grid = std::max<long long>(1, std::min<long long>((rows + 7) / 8, (long long)sms * 8));
    iso::ProfScope ps("sdf_union_grid", st);
    sdf_union_grid<<<unsigned(grid), 256, 0, st>>>(prims, nx, ny, nz, aabb_min[0], aabb_min[1], aabb_min[2],
                                                   aabb_max[0] - aabb_min[0], aabb_max[1] - aabb_min[1],
                                                   aabb_max[2] - aabb_min[2], iso::arith_fma(), out);
    return cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
}

}  // extern "C"
