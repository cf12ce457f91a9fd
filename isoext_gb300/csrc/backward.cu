// Backward passes: gradients of extracted vertex positions with respect to the
// grid values (sm_103a).  Topology is integer and has no gradient: which edges
// cross, which cells are active and the faces stay fixed.  Vertex positions are
// differentiable functions of the values.
//
//   marching cubes   v = lerp(t, pa, pb), t = (level - va) / (vb - va)
//                    (src/mc/nagae.cu:52-56, include/math.cuh:77-81).  Only the
//                    edge's axis moves: dv/dt = pb - pa along it, and
//                    dt/dva = -(1 - t) / (vb - va), dt/dvb = -t / (vb - va).
//   dual contouring  x = pinv(M) r with M = sum n n^T + reg I and
//                    r = sum n (n . p) + reg mean(p) (src/dc.cu:14-65), clipped
//                    to the cell (src/dc.cu:82-99).  Implicit differentiation of
//                    M x = r gives dL/dr = lambda = pinv(M) g and
//                    dL/dM = -lambda x^T, with g zero in clipped coordinates.
//                    Per crossing this is dL/dn = lambda (n . (p - x)) + (p - x)(lambda . n)
//                    and dL/dp = n (lambda . n) + (reg / K) lambda.  Crossing
//                    points depend on the values through t, and normals taken
//                    from the grid through the cell's trilinear interpolant and
//                    its central-difference stencil (src/its.cu:170-268).
//
// Gradients are accumulated into grad_values with atomics: a grid value feeds
// several vertices.  The summation order varies between runs (FP32 rounding
// differences only).
#include <cstdint>

#include "common.cuh"
#define ISO_LUT_DECL static __constant__ const
#include "luts.h"
#include "dc_common.cuh"
#include "profile.cuh"

namespace {

__global__ void __launch_bounds__(256) mc_backward(const float* __restrict__ vals, Grid3 g, float level,
                                                   const long long* __restrict__ vedge, long long V,
                                                   const float* __restrict__ gv, float* gvals) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= V) return;
    const long long key = vedge[i];
    const long long ia = key / 3;
    const int ax = int(key - 3 * ia);
    const long long syz = (long long)g.ny * g.nz;
    const long long step = ax == 0 ? syz : (ax == 1 ? (long long)g.nz : 1ll);
    const float va = vals[ia], vb = vals[ia + step];
    const float d = __fsub_rn(vb, va);
    if (d == 0.0f) return;  // t is the constant 0 there
    const float t = iso::cross_t(level, va, vb);
    const int c = ax == 0 ? int(ia / syz) : (ax == 1 ? int((ia / g.nz) % g.ny) : int(ia % g.nz));
    const float h = coord(g, ax, uint32_t(c + 1)) - coord(g, ax, uint32_t(c));
    const float gt = gv[3 * i + ax] * h;
    atomicAdd(gvals + ia, -gt * (1.0f - t) / d);
    atomicAdd(gvals + ia + step, -gt * t / d);
}

// Gradient of the grid normal at crossing point p (cell_normal) given dL/dn:
// adds to the cell's corner values (gc) and to the point (gp).
// The interpolant f is linear along each axis, so the stencil's difference along
// axis a, (f(t + e_a) - f(t - e_a)) / width, is its derivative there whatever the
// width (the clamps change the width only), and that derivative does not depend on
// t_a.  With G_a = df/dt_a / size_a and n = G / |G|, the adjoint A_a = dL/dG_a / size_a
// gives dL/dv_j = sum_a A_a dw_j/dt_a and dL/dt_b = sum_{a != b} A_a d2f/dt_a dt_b:
// some 200 operations, where weights and their derivatives at all six samples of
// the stencil took 850.
__device__ __forceinline__ void normal_backward(const CellCorners& cc, const float* p, const float* gn, float* gp,
                                                float* gc) {
    float rsz[3], t[3], tin[3], o[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float csz = __fsub_rn(cc.p[7][a], cc.p[0][a]);
        const float r = __fdiv_rn(__fsub_rn(p[a], cc.p[0][a]), csz);
        t[a] = fmaxf(0.01f, fminf(0.99f, r));
        tin[a] = (r > 0.01f && r < 0.99f) ? 1.0f : 0.0f;
        o[a] = 1.0f - t[a];
        rsz[a] = 1.0f / csz;
    }
    const float* v = cc.v;  // corner 4x + 2y + z
    // differences along z, then along y and x of them
    const float z00 = v[1] - v[0], z01 = v[3] - v[2], z10 = v[5] - v[4], z11 = v[7] - v[6];
    const float y00 = v[2] - v[0], y01 = v[3] - v[1], y10 = v[6] - v[4], y11 = v[7] - v[5];
    const float x00 = v[4] - v[0], x01 = v[5] - v[1], x10 = v[6] - v[2], x11 = v[7] - v[3];
    const float fx = o[1] * (o[2] * x00 + t[2] * x01) + t[1] * (o[2] * x10 + t[2] * x11);
    const float fy = o[0] * (o[2] * y00 + t[2] * y01) + t[0] * (o[2] * y10 + t[2] * y11);
    const float fz = o[0] * (o[1] * z00 + t[1] * z01) + t[0] * (o[1] * z10 + t[1] * z11);
    const float fxy = o[2] * (x10 - x00) + t[2] * (x11 - x01);
    const float fxz = o[1] * (x01 - x00) + t[1] * (x11 - x10);
    const float fyz = o[0] * (y01 - y00) + t[0] * (y11 - y10);
    const float G[3] = {fx * rsz[0], fy * rsz[1], fz * rsz[2]};
    const float len = sqrtf(G[0] * G[0] + G[1] * G[1] + G[2] * G[2]);
    if (!(len > 1e-8f)) return;  // the normal is the constant (0, 0, 1) there
    const float rl = 1.0f / len;
    const float n[3] = {G[0] * rl, G[1] * rl, G[2] * rl};
    const float ng = n[0] * gn[0] + n[1] * gn[1] + n[2] * gn[2];
    float A[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) A[a] = (gn[a] - n[a] * ng) * rl * rsz[a];
    // dw_j/dt_a is the product of the other two axes' weights, signed by j's side of a
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int bx = j >> 2, by = (j >> 1) & 1, bz = j & 1;
        const float wx = bx ? t[0] : o[0], wy = by ? t[1] : o[1], wz = bz ? t[2] : o[2];
        const float ax = bx ? A[0] : -A[0], ay = by ? A[1] : -A[1], az = bz ? A[2] : -A[2];
        gc[j] += ax * (wy * wz) + ay * (wx * wz) + az * (wx * wy);
    }
    gp[0] += (A[1] * fxy + A[2] * fxz) * tin[0] * rsz[0];
    gp[1] += (A[0] * fxy + A[2] * fyz) * tin[1] * rsz[1];
    gp[2] += (A[0] * fxz + A[1] * fyz) * tin[2] * rsz[2];
}

// One thread per active cell.  The crossings, their normals and the QEF are
// recomputed in the forward's order (the same bits), then the crossings are
// walked again for the gradients; the cell's corners stay in registers (edge
// corners are selected, not indexed), and the first crossings' points and normals
// in shared memory between the two walks.  Bound by FP32 issue: spreading a
// cell's crossings over two or four lanes, which shortens its chain, made it
// slower (70 -> 105 and 98 us for 0.12 M cells before normal_backward's rewrite).
// With it 42 us at 96 registers (five CTAs per SM: 942 CTAs are a wave and a
// quarter), 35 at 72 with some spills (seven).
constexpr int DCB_THREADS = 128;
constexpr int DCB_KEEP = 6;  // crossings kept (a smooth surface's cells have three to six)

__global__ void __launch_bounds__(DCB_THREADS, 7) dc_backward(const float* __restrict__ vals, Grid3 g, float level,
                                                   const uint32_t* __restrict__ cell_ids,
                                                   const uint32_t* __restrict__ cell_off, long long A,
                                                   float reg, float svd_tol,
                                                   const float* __restrict__ user_normals,
                                                   const float* __restrict__ gdual, float* gvals,
                                                   float* gnormals) {
    __shared__ float kept[DCB_KEEP][7][DCB_THREADS];  // t, point, normal
    const long long a = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= A) return;
    const int tid = threadIdx.x;
    float gx[3] = {gdual[3 * a], gdual[3 * a + 1], gdual[3 * a + 2]};
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
    const uint32_t k0 = cell_off[a];
    // the forward again: the QEF of the crossings in edge order
    Qef Q;
    qef_init(Q, g.fma);
    uint32_t K = 0;
#pragma unroll 1
    for (uint32_t em = est; em; em &= em - 1, ++K) {
        const int e = __ffs(em) - 1;
        float p[3], n[3];
        const float t = edge_cross(cc, level, e, p);
        if (user_normals) {
#pragma unroll
            for (int q = 0; q < 3; ++q) n[q] = user_normals[3ll * (k0 + K) + q];
        } else {
            cell_normal(cc, p, n);
        }
        if (K < uint32_t(DCB_KEEP)) {
            kept[K][0][tid] = t;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                kept[K][1 + q][tid] = p[q];
                kept[K][4 + q][tid] = n[q];
            }
        }
        qef_add(Q, p[0], p[1], p[2], n[0], n[1], n[2]);
    }
    qef_finish(Q, K, reg, svd_tol);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const float lo = cc.p[0][q], hi = cc.p[7][q];  // the cell's box
        const float xf = float(Q.x[q]);
        if (xf < lo || xf > hi) gx[q] = 0.0f;  // clipped: the output does not move
    }
    if (gx[0] == 0.0f && gx[1] == 0.0f && gx[2] == 0.0f) return;
    float l[3] = {0.0f, 0.0f, 0.0f};
    apply_pinv_f(Q.w, Q.q, Q.keep, gx, l);  // lambda = pinv(M) g
    const float rk = reg / float(K);
    float gc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    uint32_t k = 0;
#pragma unroll 1
    for (uint32_t em = est; em; em &= em - 1, ++k) {
        const int e = __ffs(em) - 1;
        float t, p[3], n[3];
        if (k < uint32_t(DCB_KEEP)) {
            t = kept[k][0][tid];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                p[q] = kept[k][1 + q][tid];
                n[q] = kept[k][4 + q][tid];
            }
        } else {
            t = edge_cross(cc, level, e, p);
            if (user_normals) {
#pragma unroll
                for (int q = 0; q < 3; ++q) n[q] = user_normals[3ll * (k0 + k) + q];
            } else {
                cell_normal(cc, p, n);
            }
        }
        float u[3], gn[3], gp[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) u[q] = float(double(p[q]) - Q.x[q]);
        const float ln = l[0] * n[0] + l[1] * n[1] + l[2] * n[2];
        const float nu = n[0] * u[0] + n[1] * u[1] + n[2] * u[2];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            gn[q] = l[q] * nu + u[q] * ln;
            gp[q] = n[q] * ln + rk * l[q];
        }
        if (user_normals) {
            if (gnormals) {
#pragma unroll
                for (int q = 0; q < 3; ++q) gnormals[3ll * (k0 + k) + q] = gn[q];
            }
        } else {
            normal_backward(cc, p, gn, gp, gc);
        }
        // through the crossing's t to the edge's two corner values
        const int ca = edge_ca(e), cb = edge_cb(e);
        const float d = corner_value(cc, cb) - corner_value(cc, ca);
        if (d == 0.0f) continue;
        float pa[3], pb[3];
        corner_pos(cc, ca, pa);
        corner_pos(cc, cb, pb);
        float gt = 0.0f;
#pragma unroll
        for (int q = 0; q < 3; ++q) gt += gp[q] * (pb[q] - pa[q]);
        const float ga = -(gt * (1.0f - t) / d), gb = -(gt * t / d);
#pragma unroll
        for (int j = 0; j < 8; ++j) gc[j] += (j == ca ? ga : 0.0f) + (j == cb ? gb : 0.0f);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (gc[j] == 0.0f) continue;
        const int x = cx + (j >> 2), y = cy + ((j >> 1) & 1), z = cz + (j & 1);
        atomicAdd(gvals + ((long long)x * g.ny + y) * g.nz + z, gc[j]);
    }
}

// grad_dual[src[i]] = grad_vertices[i]: each dual vertex is the source of at
// most one welded vertex.
__global__ void dc_scatter_src(const int* __restrict__ src, long long V, const float* __restrict__ gv,
                               float* __restrict__ gdual) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= V) return;
    const long long a = src[i];
    gdual[3 * a] = gv[3 * i];
    gdual[3 * a + 1] = gv[3 * i + 1];
    gdual[3 * a + 2] = gv[3 * i + 2];
}

}  // namespace

extern "C" {

int iso_mc_backward(const float* values, int nx, int ny, int nz, const float* aabb_min, const float* aabb_max,
                    float level, const long long* vertex_edges, long long V, const float* grad_vertices,
                    float* grad_values, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (V < 0 || nx < 2 || ny < 2 || nz < 2 || !aabb_min || !aabb_max) return iso::fail_code(ISO_ERR_ARG);
    if (V == 0) return 0;
    if (!values || !vertex_edges || !grad_vertices || !grad_values) return iso::fail_code(ISO_ERR_ARG);
    const Grid3 g = make_grid(nx, ny, nz, aabb_min, aabb_max);
    iso::ProfScope ps("mc_backward", st);
    mc_backward<<<blocks_for(V, 256), 256, 0, st>>>(values, g, level, vertex_edges, V, grad_vertices, grad_values);
    return cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
}

int iso_dc_backward(const float* values, int nx, int ny, int nz, const float* aabb_min, const float* aabb_max,
                    float level, const int* cell_ids, const int* cell_offsets, long long A, float reg,
                    float svd_tol, const float* normals, const float* grad_dual, float* grad_values,
                    float* grad_normals, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (A < 0 || nx < 2 || ny < 2 || nz < 2 || !aabb_min || !aabb_max) return iso::fail_code(ISO_ERR_ARG);
    if (A == 0) return 0;
    if (!values || !cell_ids || !cell_offsets || !grad_dual || !grad_values) return iso::fail_code(ISO_ERR_ARG);
    const Grid3 g = make_grid(nx, ny, nz, aabb_min, aabb_max);
    iso::ProfScope ps("dc_backward", st);
    dc_backward<<<blocks_for(A, DCB_THREADS), DCB_THREADS, 0, st>>>(values, g, level, reinterpret_cast<const uint32_t*>(cell_ids),
                                                    reinterpret_cast<const uint32_t*>(cell_offsets), A, reg,
                                                    svd_tol, normals, grad_dual, grad_values, grad_normals);
    return cudaGetLastError() == cudaSuccess ? 0 : iso::fail_code(ISO_ERR_CUDA);
}

int iso_dc_backward_src(const float* values, int nx, int ny, int nz, const float* aabb_min, const float* aabb_max,
                        float level, const int* cell_ids, const int* cell_offsets, long long A, float reg,
                        float svd_tol, const int* vertex_source, long long V, const float* grad_vertices,
                        float* grad_dual_ws, float* grad_values, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (A < 0 || V < 0 || nx < 2 || ny < 2 || nz < 2 || !aabb_min || !aabb_max || !grad_values) return iso::fail_code(ISO_ERR_ARG);
    if (cudaMemsetAsync(grad_values, 0, size_t(nx) * ny * nz * sizeof(float), st) != cudaSuccess) return iso::fail_code(ISO_ERR_CUDA);
    if (A == 0 || V == 0) return 0;
    if (!values || !cell_ids || !cell_offsets || !vertex_source || !grad_vertices || !grad_dual_ws) return iso::fail_code(ISO_ERR_ARG);
    if (cudaMemsetAsync(grad_dual_ws, 0, size_t(A) * 3 * sizeof(float), st) != cudaSuccess) return iso::fail_code(ISO_ERR_CUDA);
    {
        iso::ProfScope ps("dc_backward", st);
        dc_scatter_src<<<blocks_for(V, 256), 256, 0, st>>>(vertex_source, V, grad_vertices, grad_dual_ws);
    }
    return iso_dc_backward(values, nx, ny, nz, aabb_min, aabb_max, level, cell_ids, cell_offsets, A, reg, svd_tol,
                           nullptr, grad_dual_ws, grad_values, nullptr, stream);
}

}  // extern "C"
