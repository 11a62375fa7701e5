// material.cu -- per-element cloth energies behind the C ABI: the reference's evaluate kernels
// with their per-element output layout (fn_evaluate_spring / fn_evaluate_stretch_face /
// fn_evaluate_bending, Solver/SimulationSolver/newton_solver.cpp:1002-1175) and the elastic
// energy of the line search (fn_calc_energy_*, Solver/SimulationSolver/solver_interface.cpp:505-728)
// summed in FP64.  The Newton loop does not go through these: it evaluates the same device
// functions (material.cuh) and adds the results straight into b, the diagonal and the material
// BSR (csrc/newton.cu), without the per-element arrays and the gather pass of the reference's
// assembly kernels (newton_solver.cpp:705-814).
#include <cuda_runtime.h>

#include "lcs_internal.h"
#include "material.cuh"

using namespace lcs;

namespace {

// The evaluators write 224 to 832 bytes per element, so they are bound by those stores.  One thread storing its own
// element spreads every store instruction of a warp over 32 half-written sectors (bending of an 88,800-vertex cloth,
// 221 MB: 212 us, 1.0 TB/s; the three evaluators and the energy: 368 us, now 88 us).  Here a warp's 32 elements are
// evaluated one per lane into shared memory (an odd number of words per element: no bank conflicts) and the warp then
// writes their output as one run of consecutive 16-byte words, each lane forming the word it stores.
constexpr int kEvalThreads = 128, kEvalWarps = kEvalThreads / 32;

__global__ void __launch_bounds__(kEvalThreads) k_eval_springs(uint32_t n, const float4* __restrict__ x,
                                                               const uint2* __restrict__ edges,
                                                               const float* __restrict__ rest_len,
                                                               const float* __restrict__ stiff, float4* grad, float4* hess)
{
    __shared__ float sh[kEvalWarps][32][13];  // gradient, Hessian block (column-major)
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    float(*sw)[13] = sh[warp];
    for (uint32_t e0 = 32u * (blockIdx.x * kEvalWarps + warp); e0 < n; e0 += 32u * kEvalWarps * gridDim.x) {
        const uint32_t e = e0 + lane, m = min(32u, n - e0);
        if (e < n) {
            const uint2 ed = edges[e];
            const v3 p0 = ld3(x, ed.x), p1 = ld3(x, ed.y);
            const v3 d = p0 - p1;
            const float l = fmx(sqrtf(dot3(d, d)), 1.19209290E-7f);
            const float k = stiff[e], L = rest_len[e];
            const float C = l - L, il = 1.0f / l, il2 = il * il;
            sw[lane][0] = k * d.x * il * C;
            sw[lane][1] = k * d.y * il * C;
            sw[lane][2] = k * d.z * il * C;
            const float a = k * il2, c = k * fmx(1.0f - L * il, 0.0f);
            const float dd[3] = {d.x, d.y, d.z};
#pragma unroll
            for (int cc = 0; cc < 3; ++cc)
#pragma unroll
                for (int r = 0; r < 3; ++r)
                    sw[lane][3 + 3 * cc + r] = a * dd[r] * dd[cc] + c * ((r == cc ? 1.0f : 0.0f) - il2 * dd[r] * dd[cc]);
        }
        __syncwarp();
        for (uint32_t i = lane; i < 2u * m; i += 32u) {  // g, -g
            const float* g = sw[i >> 1];
            const float sgn = (i & 1u) ? -1.0f : 1.0f;
            __stcs(&grad[2 * (size_t)e0 + i], make_float4(sgn * g[0], sgn * g[1], sgn * g[2], 0.0f));
        }
        for (uint32_t i = lane; i < 12u * m; i += 32u) {  // blocks (0,0) (1,1) (0,1) (1,0): H, H, -H, -H
            const uint32_t el = i / 12u, k = i - 12u * el, c = k % 3u;
            const float* H = sw[el] + 3 + 3 * c;
            const float sgn = k >= 6u ? -1.0f : 1.0f;
            __stcs(&hess[12 * (size_t)e0 + i], make_float4(sgn * H[0], sgn * H[1], sgn * H[2], 0.0f));
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(kEvalThreads) k_eval_stretch_faces(uint32_t n, const float4* __restrict__ x,
                                                                     const uint4* __restrict__ faces,
                                                                     const float4* __restrict__ dm,
                                                                     const float* __restrict__ area,
                                                                     const float2* __restrict__ mu_lambda, float4* grad,
                                                                     float4* hess)
{
    __shared__ float sh[kEvalWarps][32][63];  // 3 gradients, 6 blocks (column-major)
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    float(*sw)[63] = sh[warp];
    for (uint32_t f0 = 32u * (blockIdx.x * kEvalWarps + warp); f0 < n; f0 += 32u * kEvalWarps * gridDim.x) {
        const uint32_t f = f0 + lane, m = min(32u, n - f0);
        if (f < n) {
            const uint4 fc = faces[f];
            const float2 ml = mu_lambda[f];
            Bw98Out o;
            bw98_face(ld3(x, fc.x), ld3(x, fc.y), ld3(x, fc.z), dm[f], ml.x, ml.y, area[f], o);
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                sw[lane][3 * a] = o.g[a].x;
                sw[lane][3 * a + 1] = o.g[a].y;
                sw[lane][3 * a + 2] = o.g[a].z;
            }
#pragma unroll
            for (int k = 0; k < 6; ++k)
#pragma unroll
                for (int j = 0; j < 9; ++j) sw[lane][9 + 9 * k + j] = o.K[k][j];
        }
        __syncwarp();
        for (uint32_t i = lane; i < 3u * m; i += 32u) {
            const uint32_t el = i / 3u;
            const float* g = sw[el] + 3u * (i - 3u * el);
            __stcs(&grad[3 * (size_t)f0 + i], make_float4(g[0], g[1], g[2], 0.0f));
        }
        // blocks (0,0) (1,1) (2,2), then (0,1) (0,2) (1,0) (1,2) (2,0) (2,1) (row vertex, column vertex): the stored
        // blocks 0 1 2 3 4 3' 5 4' 5' (' transposed)
        for (uint32_t i = lane; i < 27u * m; i += 32u) {
            const uint32_t el = i / 27u, k = i - 27u * el, blk = k / 3u, c = k - 3u * blk;
            const uint32_t src = (0x545343210ull >> (4u * blk)) & 15u;
            const bool tr = (0x1A0u >> blk) & 1u;
            const float* K = sw[el] + 9 + 9 * src + (tr ? c : 3u * c);
            const uint32_t st = tr ? 3u : 1u;
            __stcs(&hess[27 * (size_t)f0 + i], make_float4(K[0], K[st], K[2 * st], 0.0f));
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(kEvalThreads) k_eval_bending(uint32_t n, const float4* __restrict__ x,
                                                               const uint4* __restrict__ st,
                                                               const float* __restrict__ rest_angle,
                                                               const float* __restrict__ hbar,
                                                               const float* __restrict__ stiffness, float scaling,
                                                               float4* grad, float4* hess)
{
    __shared__ float sh[kEvalWarps][32][15];  // dtheta/dx of the four vertices, stiffness, stiffness (theta - rest)
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    float(*sw)[15] = sh[warp];
    // 48 Hessian words per element: a run of 96 words (two elements) is three words per lane, so the lane's three
    // places (element of the two, vertices i and j, column) are the same in every run
    uint32_t pe[3], pi[3], pj[3];
#pragma unroll
    for (uint32_t q = 0; q < 3; ++q) {
        const uint32_t w = 32u * q + lane, k = w % 48u, blk = k / 3u, c = k - 3u * blk;
        pe[q] = w / 48u;
        // blocks (i, i), then (i, j), i != j, row-major
        const uint32_t o = blk - 4u, i = blk < 4u ? blk : o / 3u, jj = blk < 4u ? blk : o - 3u * i;
        const uint32_t j = blk < 4u ? blk : jj + (jj >= i ? 1u : 0u);
        pi[q] = 3u * i;
        pj[q] = 3u * j + c;
    }
    for (uint32_t s0 = 32u * (blockIdx.x * kEvalWarps + warp); s0 < n; s0 += 32u * kEvalWarps * gridDim.x) {
        const uint32_t s = s0 + lane, m = min(32u, n - s0);
        if (s < n) {
            const uint4 e = st[s];
            v3 g[4];
            const float theta = dihedral_angle_grad(ld3(x, e.x), ld3(x, e.y), ld3(x, e.z), ld3(x, e.w), g);
            const float stiff = stiffness[s] * scaling * hbar[s];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                sw[lane][3 * i] = g[i].x;
                sw[lane][3 * i + 1] = g[i].y;
                sw[lane][3 * i + 2] = g[i].z;
            }
            sw[lane][12] = stiff;
            sw[lane][13] = stiff * (theta - rest_angle[s]);
        }
        __syncwarp();
        for (uint32_t i = lane; i < 4u * m; i += 32u) {
            const float *o = sw[i >> 2], *g = o + 3u * (i & 3u);
            __stcs(&grad[4 * (size_t)s0 + i], make_float4(o[13] * g[0], o[13] * g[1], o[13] * g[2], 0.0f));
        }
        float4* h = hess + 48 * (size_t)s0 + lane;
        for (uint32_t e = 0; e < m; e += 2u, h += 96) {
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                if (e + pe[q] >= m) continue;  // the last element of an odd count
                const float *o = sw[e + pe[q]], *gi = o + pi[q];
                const float k = o[12], gj = o[pj[q]];
                __stcs(h + 32 * q, make_float4(k * (gi[0] * gj), k * (gi[1] * gj), k * (gi[2] * gj), 0.0f));
            }
        }
        __syncwarp();
    }
}

// energy terms: [0] inertia (fn_calc_energy_inertia), [1] springs, [2] stretch faces, [3] bending
// One atomic per block and term: with one per warp, about 8,300 additions to each of four addresses took most of the
// time (46 us on 88,800 vertices).
__global__ void __launch_bounds__(256) k_material_energy(lcs_cloth_elements m, const float4* __restrict__ x,
                                                         const float4* __restrict__ xt, float dt, float dirichlet,
                                                         double* out)
{
    const uint32_t n = max(max(m.n_verts, m.n_springs), max(m.n_stretch_faces, m.n_bending));
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t n_round = (n + stride - 1) / stride * stride;  // all lanes take the same trips
    double e[4] = {0.0, 0.0, 0.0, 0.0};
    const float h2inv = 1.0f / (dt * dt);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_round; i += stride) {
        if (i < m.n_verts) {
            const v3 d = ld3(x, i) - ld3(xt, i);
            float en = h2inv * dot3(d, d) * m.mass[i] / 2.0f;
            if (m.is_fixed && m.is_fixed[i]) en = dirichlet * en;
            e[0] += (double)en;
        }
        if (i < m.n_springs) {
            const uint2 ed = reinterpret_cast<const uint2*>(m.springs)[i];
            const v3 d = ld3(x, ed.y) - ld3(x, ed.x);
            const float C = sqrtf(dot3(d, d)) - m.spring_rest_len[i];
            e[1] += (double)(0.5f * m.spring_stiffness[i] * C * C);
        }
        if (i < m.n_stretch_faces) {
            const uint4 fc = reinterpret_cast<const uint4*>(m.stretch_faces)[i];
            const float4 dm = reinterpret_cast<const float4*>(m.stretch_dm_inv)[i];
            const float2 ml = reinterpret_cast<const float2*>(m.stretch_mu_lambda)[i];
            const v3 x0 = ld3(x, fc.x), e1 = ld3(x, fc.y) - x0, e2 = ld3(x, fc.z) - x0;
            const v3 Fu = mk3(__fmaf_rn(e2.x, dm.y, e1.x * dm.x), __fmaf_rn(e2.y, dm.y, e1.y * dm.x),
                              __fmaf_rn(e2.z, dm.y, e1.z * dm.x));
            const v3 Fv = mk3(__fmaf_rn(e2.x, dm.w, e1.x * dm.z), __fmaf_rn(e2.y, dm.w, e1.y * dm.z),
                              __fmaf_rn(e2.z, dm.w, e1.z * dm.z));
            const float su = sqrtf(dot3(Fu, Fu)) - 1.0f, sv = sqrtf(dot3(Fv, Fv)) - 1.0f, i6 = dot3(Fu, Fv);
            const float en = 0.5f * ml.x * (su * su + sv * sv) + 0.5f * ml.y * (i6 * i6);
            e[2] += (double)(m.stretch_area[i] * en);
        }
        if (i < m.n_bending) {
            const uint4 st = reinterpret_cast<const uint4*>(m.bending_edges)[i];
            v3 g[4];
            const float theta = dihedral_angle_grad(ld3(x, st.x), ld3(x, st.y), ld3(x, st.z), ld3(x, st.w), g);
            const float d = theta - m.bending_rest_angle[i];
            e[3] += (double)(0.5f * m.bending_stiffness[i] * m.bending_scaling * m.bending_hbar[i] * d * d);
        }
    }
    __shared__ double red[4][8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) e[k] += __shfl_xor_sync(0xFFFFFFFFu, e[k], o);
        if (lane_id() == 0) red[k][threadIdx.x >> 5] = e[k];
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) v += red[threadIdx.x][w];
        if (v != 0.0) atomicAdd(out + threadIdx.x, v);
    }
}

int launch_check(const char* what)
{
    lcs_count_launch();
    return cudaGetLastError() == cudaSuccess ? LCS_OK : lcs_fail(LCS_ERR_CUDA, what);
}

}  // namespace

extern "C" int lcs_eval_springs(const float* x, const uint32_t* edges, const float* rest_len, const float* stiffness,
                                uint32_t n, float* gradients, float* hessians, lcs_stream stream)
{
    if (n == 0) return LCS_OK;
    if (!x || !edges || !rest_len || !stiffness || !gradients || !hessians)
        return lcs_fail(LCS_ERR_INVALID, "lcs_eval_springs: null argument");
    k_eval_springs<<<grid_for(n, kEvalThreads, 16), kEvalThreads, 0, (cudaStream_t)stream>>>(
        n, reinterpret_cast<const float4*>(x), reinterpret_cast<const uint2*>(edges), rest_len, stiffness,
        reinterpret_cast<float4*>(gradients), reinterpret_cast<float4*>(hessians));
    return launch_check("lcs_eval_springs: launch failed");
}

extern "C" int lcs_eval_stretch_faces(const float* x, const uint32_t* faces, const float* dm_inv, const float* rest_area,
                                      const float* mu_lambda, uint32_t n, float* gradients, float* hessians,
                                      lcs_stream stream)
{
    if (n == 0) return LCS_OK;
    if (!x || !faces || !dm_inv || !rest_area || !mu_lambda || !gradients || !hessians)
        return lcs_fail(LCS_ERR_INVALID, "lcs_eval_stretch_faces: null argument");
    k_eval_stretch_faces<<<grid_for(n, kEvalThreads, 7), kEvalThreads, 0, (cudaStream_t)stream>>>(
        n, reinterpret_cast<const float4*>(x), reinterpret_cast<const uint4*>(faces),
        reinterpret_cast<const float4*>(dm_inv), rest_area, reinterpret_cast<const float2*>(mu_lambda),
        reinterpret_cast<float4*>(gradients), reinterpret_cast<float4*>(hessians));
    return launch_check("lcs_eval_stretch_faces: launch failed");
}

extern "C" int lcs_eval_bending(const float* x, const uint32_t* stencils, const float* rest_angle, const float* rest_hbar,
                                const float* stiffness, float scaling, uint32_t n, float* gradients, float* hessians,
                                lcs_stream stream)
{
    if (n == 0) return LCS_OK;
    if (!x || !stencils || !rest_angle || !rest_hbar || !stiffness || !gradients || !hessians)
        return lcs_fail(LCS_ERR_INVALID, "lcs_eval_bending: null argument");
    k_eval_bending<<<grid_for(n, kEvalThreads, 16), kEvalThreads, 0, (cudaStream_t)stream>>>(
        n, reinterpret_cast<const float4*>(x), reinterpret_cast<const uint4*>(stencils), rest_angle, rest_hbar,
        stiffness, scaling, reinterpret_cast<float4*>(gradients), reinterpret_cast<float4*>(hessians));
    return launch_check("lcs_eval_bending: launch failed");
}

extern "C" int lcs_material_energy(const lcs_cloth_elements* m, const float* x, const float* x_tilde, float dt,
                                   float stiffness_dirichlet, double* energy, lcs_stream stream)
{
    if (!m || !x || !energy || (m->n_verts && (!x_tilde || !m->mass)) ||
        (m->n_springs && (!m->springs || !m->spring_rest_len || !m->spring_stiffness)) ||
        (m->n_stretch_faces && (!m->stretch_faces || !m->stretch_dm_inv || !m->stretch_area || !m->stretch_mu_lambda)) ||
        (m->n_bending && (!m->bending_edges || !m->bending_rest_angle || !m->bending_hbar || !m->bending_stiffness)))
        return lcs_fail(LCS_ERR_INVALID, "lcs_material_energy: incomplete element description");
    cudaStream_t s = (cudaStream_t)stream;
    LCS_CUDA_TRY(cudaMemsetAsync(energy, 0, 4 * sizeof(double), s));
    const uint32_t n = std::max(std::max(m->n_verts, m->n_springs), std::max(m->n_stretch_faces, m->n_bending));
    if (n == 0) return LCS_OK;
    k_material_energy<<<grid_for(n, 256, 4), 256, 0, s>>>(*m, reinterpret_cast<const float4*>(x),
                                                      reinterpret_cast<const float4*>(x_tilde), dt,
                                                      stiffness_dirichlet, energy);
    return launch_check("lcs_material_energy: launch failed");
}
