// kernels_mixed.cuh -- the mixed-precision force gather and CG solve.
//
// The viscosity matrix V of a blob without Stokes drag is singular: rigid
// translations and rotations that leave every pinned node at rest produce no
// viscous stress, so V z = 0 for them (the columns of Z). The reference's FP64
// CG converges before rounding excites these directions; with V in FP32 the
// rounding of every product (~1e-7) feeds them and the 1e-10 relative
// residual becomes unreachable. This solver runs CG on
//     V~ = V + D Z G^{-1} Z^T D,     G = Z^T D Z,  D = diag(V),
// with the right-hand side projected to f^ = f - D Z G^{-1} Z^T f. V~ is
// symmetric positive definite, D^{-1} V~ maps each rigid mode to itself, and
// its solution x satisfies Z^T D x = 0 and V x = f^: exactly the solution the
// reference's Jacobi-PCG builds from x = 0 (its iterates stay in D^{-1} times
// the range of V, i.e. D-orthogonal to Z). With V~ nonsingular the whole CG
// can run in FP32: matrix, SpMV, x, r, p, q.
//
// Reductions: each node's contribution is formed in FP32, summed over the
// block and the grid as double-float pairs (two FP32 values, ~48-bit
// significand); GB300 runs FP64 at 1/64 of the FP32 rate, so no per-node work
// touches the FP64 pipe. The set-up's mode matrix is formed in FP64, and so are
// the iteration's scalars of cg_mixed_kernel and cg_batch_kernel; the owned-rows
// kernels form theirs (p.q, the mode coefficients, the stopping test) in
// double-float, step lengths in FP32 everywhere. With FP64 scalars in those too,
// every solution and iteration count of ten meshes of 343 to 166,375 nodes came
// out the same to the last digit.
//
// Z is expressed through per-node offsets d_a from a reference point: the
// k-th mode is t_k + w_k x d_a. Z^T v needs only S1 = sum v_a and
// S2 = sum d_a x v_a; D Z c at node a is D_a (tau + Omega x d_a).
#pragma once

#include "kernels.cuh"
#include "kernels_element_mixed.cuh"

namespace ffea {

constexpr int MIXED_GATHER_NP = 28;  // f.f, S1_f(3), S2_f(3), M = sum Phi^T D Phi (21)
constexpr int MIXED_A_NP = 7;        // p.q, S1(Dp)(3), S2(Dp)(3)
constexpr int MIXED_B_NP = 2;        // r.r, r.z
// partial rows: [0, A) phase A, [A, A+B) phase B, A+B the initial r.z
constexpr int MIXED_PARTIAL_ROWS = MIXED_A_NP + MIXED_B_NP + 1;
// cg_mixed_sr_kernel's one reduction per iteration: r.z, r.r, z.w, z.q, p.w, S1(Dz)(3), S2(Dz)(3)
constexpr int MIXED_SR_NP = 11;

// the six basis columns phi_j of Phi_a = [I | (.) x d]: e_x, e_y, e_z, e_x x d, e_y x d, e_z x d
__device__ __forceinline__ void phi_cols(float dx, float dy, float dz, float (&phi)[6][3]) {
    phi[0][0] = 1; phi[0][1] = 0; phi[0][2] = 0;
    phi[1][0] = 0; phi[1][1] = 1; phi[1][2] = 0;
    phi[2][0] = 0; phi[2][1] = 0; phi[2][2] = 1;
    phi[3][0] = 0; phi[3][1] = -dz; phi[3][2] = dy;
    phi[4][0] = dz; phi[4][1] = 0; phi[4][2] = -dx;
    phi[5][0] = -dy; phi[5][1] = dx; phi[5][2] = 0;
}

// mixed-path gather: f (FP64 copy) and r = f (FP32); node offsets; moments for the rigid-mode set-up. MODE is
// g.mode: 0 (one blob's CG, with the block moments), 1 (mass-lumped), 2 (batch CG); the modes without the block
// reduction carry none of its registers. NF: some node force besides the elements' (constant forces, inertial
// Stokes drag, Stokes noise, midpoint forces); without, none of their registers either, and the mass-lumped form
// is held to 32 registers (a full SM of threads; 1 % faster than 40 registers on the 64^3 step).
template <class R, int MODE, bool NF>
__global__ void __launch_bounds__(256, (MODE == 1 && !NF) ? 8 : 1) gather_mixed_kernel(GatherArgs<R> g) {
    __shared__ float2 smem[MIXED_GATHER_NP * 32];
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a == 0 && g.gb) g.gb->count = 0u;
    if constexpr (MODE == 1) {
        if (g.fin_next && a == 0 && !g.st->abort) {
            uint32_t s6[6], o6[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) s6[k] = g.nrng[k];
            mrg_apply(*g.fin_jump, s6, o6);
#pragma unroll
            for (int k = 0; k < 6; ++k) g.fin_next[k] = o6[k];
            g.st->steps_done += 1;
        }
        if (g.nchunk_state && a < g.nnchunks) {
            uint32_t s6[6], o6[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) s6[k] = g.nrng[k];
            mrg_apply(g.ncj[a], s6, o6);
#pragma unroll
            for (int k = 0; k < 6; ++k) g.nchunk_state[6 * (size_t)a + k] = o6[k];
        }
    }
    df32 acc[MIXED_GATHER_NP];
#pragma unroll
    for (int i = 0; i < MIXED_GATHER_NP; ++i) acc[i] = df32{0.f, 0.f};
    if (a < g.N && !g.st->abort) {
        float F0 = 0, F1 = 0, F2 = 0;
        if (NF && g.sn.node_ctf) {
            F0 = (float)g.sn.node_ctf[3 * (size_t)a];
            F1 = (float)g.sn.node_ctf[3 * (size_t)a + 1];
            F2 = (float)g.sn.node_ctf[3 * (size_t)a + 2];
        }
        if (g.parts) {
            // two block sums per trip, both loads ahead of the adds (the adds keep block order)
            int m = g.part_ptr[a];
            const int m1 = g.part_ptr[a + 1];
            for (; m + 2 <= m1; m += 2) {
                const float4 q = g.parts[m], q2 = g.parts[m + 1];
                F0 += q.x; F1 += q.y; F2 += q.z;
                F0 += q2.x; F1 += q2.y; F2 += q2.z;
            }
            if (m < m1) {
                const float4 q = g.parts[m];
                F0 += q.x; F1 += q.y; F2 += q.z;
            }
        } else {
            for (int m = g.inc_ptr[a]; m < g.inc_ptr[a + 1]; ++m) {
                const int es = g.inc[m];
                const R *c = g.ef + 12 * (size_t)(es >> 2) + 3 * (es & 3);
                F0 += c[0];
                F1 += c[1];
                F2 += c[2];
            }
        }
        if (NF && g.sn.vface_ptr) {
            float F[3] = {F0, F1, F2};
            surface_add<float>(g.sn, g.sn.vface_ptr, g.sn.vface, a, F);
            F0 = F[0]; F1 = F[1]; F2 = F[2];
        }
        if (NF && g.drag) {
            const double dr = g.drag[a];
            F0 -= (float)(g.vx[a] * dr);
            F1 -= (float)(g.vy[a] * dr);
            F2 -= (float)(g.vz[a] * dr);
        }
        if (NF && g.sn.on) {
            float F[3] = {F0, F1, F2};
            if (g.sn.noise) stokes_noise_sub<float>(g.sn, g.sn.node_orig[a], g.sn.node_drag[a], F);
            if (g.sn.lin_ptr) midpoint_linearise<float>(g.sn, a, F);
            F0 = F[0]; F1 = F[1]; F2 = F[2];
        }
        if (g.pinned[a]) { F0 = 0; F1 = 0; F2 = 0; }
        if (g.f32) {
            g.f32[4 * a] = F0; g.f32[4 * a + 1] = F1; g.f32[4 * a + 2] = F2;
        } else if (g.f) {
            g.f[4 * a] = F0; g.f[4 * a + 1] = F1; g.f[4 * a + 2] = F2;
        }
        if constexpr (MODE == 1) {
            const float4 di = reinterpret_cast<const float4 *>(g.dinv)[a];
            const R x0 = F0 * di.x, x1 = F1 * di.y, x2 = F2 * di.z;
            g.x[4 * a] = x0;
            g.x[4 * a + 1] = x1;
            g.x[4 * a + 2] = x2;
            if (g.fuse_euler) {
                // euler_integrate (src/Blob.cpp:3249-3279) as euler_kernel does it: v += a dt, p += v dt
                if (!(isfinite(x0) && isfinite(x1) && isfinite(x2))) atomicExch(&g.st->nonfinite, 1);
                const double a0 = (double)x0, a1 = (double)x1, a2 = (double)x2;
                const double v0 = g.uvx[a] + a0 * g.dt, v1 = g.uvy[a] + a1 * g.dt, v2 = g.uvz[a] + a2 * g.dt;
                g.uvx[a] = v0; g.uvy[a] = v1; g.uvz[a] = v2;
                const double p0 = g.upx[a] + v0 * g.dt, p1 = g.upy[a] + v1 * g.dt, p2 = g.upz[a] + v2 * g.dt;
                g.upx[a] = p0; g.upy[a] = p1; g.upz[a] = p2;
                if (g.nu) {
                    const size_t N = g.N;
                    g.nu[a] = make_float4((float)(p0 - g.nxr[a]), (float)(p1 - g.nxr[N + a]),
                                          (float)(p2 - g.nxr[2 * N + a]), 0.f);
                    g.nvf[a] = make_float4((float)v0, (float)v1, (float)v2, 0.f);
                }
            }
            return;
        }
        g.r[4 * a] = F0; g.r[4 * a + 1] = F1; g.r[4 * a + 2] = F2;
        if constexpr (MODE == 2) return;  // batch: the per-blob CG set-up forms the moments
        const float dx = (float)(g.px[a] - g.xc[0]), dy = (float)(g.py[a] - g.xc[1]), dz = (float)(g.pz[a] - g.xc[2]);
        g.dpos[a] = make_float4(dx, dy, dz, 0.f);
        acc[0] = df32{F0 * F0 + F1 * F1 + F2 * F2, 0.f};
        acc[1].hi = F0; acc[2].hi = F1; acc[3].hi = F2;
        acc[4].hi = dy * F2 - dz * F1; acc[5].hi = dz * F0 - dx * F2; acc[6].hi = dx * F1 - dy * F0;
        if (g.diag) {
            float phi[6][3];
            phi_cols(dx, dy, dz, phi);
            const float D[3] = {(float)g.diag[4 * a], (float)g.diag[4 * a + 1], (float)g.diag[4 * a + 2]};
            int k = 7;
#pragma unroll
            for (int i = 0; i < 6; ++i)
#pragma unroll
                for (int j = i; j < 6; ++j, ++k)
                    acc[k].hi = phi[i][0] * D[0] * phi[j][0] + phi[i][1] * D[1] * phi[j][1] + phi[i][2] * D[2] * phi[j][2];
        }
    }
    if constexpr (MODE != 0) return;
    df32 out[MIXED_GATHER_NP];
    block_sum_df<MIXED_GATHER_NP>(acc, smem, out);
    if (threadIdx.x == 0) {
        float2 *pp = reinterpret_cast<float2 *>(g.partials);
#pragma unroll
        for (int i = 0; i < MIXED_GATHER_NP; ++i) pp[i * g.stride + blockIdx.x] = make_float2(out[i].hi, out[i].lo);
    }
}

// The whole block, once per solve: G = Z^T D Z from the moments M, G^{-1} by Gauss-Jordan on the augmented
// [G | I] in shared memory (one thread per entry, one pivot at a time), A6 = modes^T G^{-1} modes, and
// (tau, Omega) of D Z c0 with c0 = G^{-1} Z^T f. Every thread of the block must call it; the results are
// in shared memory after it returns.
template <class A>
__device__ __noinline__ void mixed_setup(const A &g, const double *s_sc, double *s_A6, float *s_tau, float *s_Om, float *s_beta,
                            int *s_conv) {
    __shared__ double sM[36], sT[36], sAug[6][12], sF[6], sV[6], sC[6], sPiv;
    const int t = threadIdx.x, k = g.nmodes;
    if (t < 36) {
        const int i = t / 6, j = t % 6, lo = i < j ? i : j, hi = i < j ? j : i;
        // packed upper triangle: row lo starts at 7 + lo*6 - lo*(lo-1)/2
        sM[t] = s_sc[7 + lo * 6 - (lo * (lo - 1)) / 2 + (hi - lo)];
    }
    __syncthreads();
    // G = modes M modes^T and, after the inversion, A6 = modes^T G^{-1} modes, each in two products of six terms
    if (t < 36) {
        const int i = t / 6, j = t % 6;
        double sum = 0.0;
        if (j < k)
            for (int q = 0; q < 6; ++q) sum += sM[6 * i + q] * g.modes[6 * j + q];
        sT[t] = sum;
    }
    __syncthreads();
    if (t < 36) {
        const int i = t / 6, j = t % 6;
        double sum = 0.0;
        if (i < k && j < k)
            for (int p = 0; p < 6; ++p) sum += g.modes[6 * i + p] * sT[6 * p + j];
        sAug[i][j] = sum;
        sAug[i][6 + j] = (i == j) ? 1.0 : 0.0;
    }
    __syncthreads();
    for (int col = 0; col < k; ++col) {
        if (t == 0) sPiv = sAug[col][col];
        __syncthreads();
        if (t < 12) sAug[col][t] /= sPiv;
        __syncthreads();
        if (t < 6) sF[t] = sAug[t][col];
        __syncthreads();
        if (t < 72) {
            const int i = t / 12, j = t % 12;
            if (i != col && i < k) sAug[i][j] -= sF[i] * sAug[col][j];
        }
        __syncthreads();
    }
    if (t < 36) {
        const int i = t / 6, q = t % 6;
        double sum = 0.0;
        if (i < k)
            for (int j = 0; j < k; ++j) sum += sAug[i][6 + j] * g.modes[6 * j + q];
        sT[t] = sum;
    }
    __syncthreads();
    if (t < 36) {
        const int p = t / 6, q = t % 6;
        double sum = 0.0;
        for (int i = 0; i < k; ++i) sum += g.modes[6 * i + p] * sT[6 * i + q];
        s_A6[t] = sum;
    }
    if (t < 6) {
        const double *m = g.modes + 6 * t;
        sV[t] = (t < k) ? m[0] * s_sc[1] + m[1] * s_sc[2] + m[2] * s_sc[3] + m[3] * s_sc[4] + m[4] * s_sc[5] +
                              m[5] * s_sc[6]
                        : 0.0;
    }
    __syncthreads();
    if (t < 6) {
        double c = 0.0;
        for (int j = 0; j < k; ++j) c += sAug[t][6 + j] * sV[j];
        sC[t] = (t < k) ? c : 0.0;
    }
    __syncthreads();
    if (t < 6) {
        double sum = 0.0;
        for (int i = 0; i < k; ++i) sum += sC[i] * g.modes[6 * i + t];
        if (t < 3) s_tau[t] = (float)sum; else s_Om[t - 3] = (float)sum;
    }
    if (t == 0) {
        *s_beta = 0.f;
        *s_conv = 0;
    }
    __syncthreads();
}

// p at node b for this iteration: p_new = beta p_old + D^{-1} r (vec3_scale_and_add with the
// preconditioned residual, src/NoMassCGSolver.cpp:181-183), or z itself on the first iteration.
template <class A>
__device__ __forceinline__ void p_on_the_fly(const A &g, const float *pold, float beta, bool first, int b, float &p0,
                                             float &p1, float &p2) {
    const float4 di = *reinterpret_cast<const float4 *>(g.dinv + 4 * (size_t)b),
                 r = *reinterpret_cast<const float4 *>(g.r + 4 * (size_t)b);
    p0 = di.x * r.x;
    p1 = di.y * r.y;
    p2 = di.z * r.z;
    if (!first) {
        const float4 po = *reinterpret_cast<const float4 *>(pold + 4 * (size_t)b);
        p0 = fmaf(beta, po.x, p0);
        p1 = fmaf(beta, po.y, p1);
        p2 = fmaf(beta, po.z, p2);
    }
}

// spmv_row with p formed on the fly from p_old, r and D^{-1}; B3: 3x3 blocks (CG_nomass) or scalar entries. The blobs
// here have matrices far larger than L2, read past it (__ldcs), and two blocks' loads issue before either's products, in
// the same order. With one block per trip the time hung on how the compiler placed the loads around whatever else was in
// registers: ms per step at 76^3 / 80^3 / 96^3 cells 85 / 113 / 201 or 115 / 155 / 274, now 75 / 102 / 196; consistent
// mass 76^3 1.70 (1.67 to 1.91).
template <bool B3, class A>
__device__ __forceinline__ void spmv_row_fly(const A &g, const float *pold, float beta, bool first, int a, int sub,
                                             bool valid, float &q0, float &q1, float &q2) {
    q0 = 0.f; q1 = 0.f; q2 = 0.f;
    const int tpn = g.tpn;
    if (valid) {
        const int s = a >> 5, lane = a & 31;
        const int base = g.slice_ptr[s];
        const int len = g.rowlen[a];
        if constexpr (B3) {
            const float *v = g.val + 9 * (size_t)base + lane;
            int k = sub;
#pragma unroll 1
            for (; k + tpn < len; k += 2 * tpn) {
                const int ba = __ldg(g.bcol + base + 32 * k + lane), bb = __ldg(g.bcol + base + 32 * (k + tpn) + lane);
                const float *va = v + (size_t)32 * 9 * k, *vb = v + (size_t)32 * 9 * (k + tpn);
                float wa[9], wb[9];
#pragma unroll
                for (int i = 0; i < 9; ++i) {
                    wa[i] = __ldcs(va + 32 * i);
                    wb[i] = __ldcs(vb + 32 * i);
                }
                float a0, a1, a2, b0, b1, b2;
                p_on_the_fly(g, pold, beta, first, ba, a0, a1, a2);
                p_on_the_fly(g, pold, beta, first, bb, b0, b1, b2);
                q0 = fmaf(wa[0], a0, q0); q0 = fmaf(wa[1], a1, q0); q0 = fmaf(wa[2], a2, q0);
                q1 = fmaf(wa[3], a0, q1); q1 = fmaf(wa[4], a1, q1); q1 = fmaf(wa[5], a2, q1);
                q2 = fmaf(wa[6], a0, q2); q2 = fmaf(wa[7], a1, q2); q2 = fmaf(wa[8], a2, q2);
                q0 = fmaf(wb[0], b0, q0); q0 = fmaf(wb[1], b1, q0); q0 = fmaf(wb[2], b2, q0);
                q1 = fmaf(wb[3], b0, q1); q1 = fmaf(wb[4], b1, q1); q1 = fmaf(wb[5], b2, q1);
                q2 = fmaf(wb[6], b0, q2); q2 = fmaf(wb[7], b1, q2); q2 = fmaf(wb[8], b2, q2);
            }
            if (k < len) {
                const int b = __ldg(g.bcol + base + 32 * k + lane);
                const float *vk = v + (size_t)32 * 9 * k;
                float w[9], p0, p1, p2;
#pragma unroll
                for (int i = 0; i < 9; ++i) w[i] = __ldcs(vk + 32 * i);
                p_on_the_fly(g, pold, beta, first, b, p0, p1, p2);
                q0 = fmaf(w[0], p0, q0); q0 = fmaf(w[1], p1, q0); q0 = fmaf(w[2], p2, q0);
                q1 = fmaf(w[3], p0, q1); q1 = fmaf(w[4], p1, q1); q1 = fmaf(w[5], p2, q1);
                q2 = fmaf(w[6], p0, q2); q2 = fmaf(w[7], p1, q2); q2 = fmaf(w[8], p2, q2);
            }
        } else {
            const float *v = g.val + base + lane;
            for (int k = sub; k < len; k += tpn) {
                const int b = g.bcol[base + 32 * k + lane];
                const float m = v[32 * k];
                float p0, p1, p2;
                p_on_the_fly(g, pold, beta, first, b, p0, p1, p2);
                q0 = fmaf(m, p0, q0);
                q1 = fmaf(m, p1, q1);
                q2 = fmaf(m, p2, q2);
            }
        }
    }
    for (int o = 1; o < tpn; o <<= 1) {
        q0 += __shfl_xor_sync(0xffffffffu, q0, o);
        q1 += __shfl_xor_sync(0xffffffffu, q1, o);
        q2 += __shfl_xor_sync(0xffffffffu, q2, o);
    }
}

template <class R, bool B3>
__global__ void __launch_bounds__(1024, 1) cg_mixed_kernel(const __grid_constant__ CgArgs<R> g) {
    __shared__ float smemf[MIXED_A_NP * 32];
    __shared__ double s_sc[MIXED_GATHER_NP];
    __shared__ double s_A6[36];
    __shared__ float s_alpha, s_beta, s_tau[3], s_Om[3];
    __shared__ double s_delta;
    __shared__ int s_conv;
    DevStatus *st = g.st;
    if (st->abort) return;
    const bool defl = g.nmodes > 0;
    FFEA_PHASES_BEGIN(g, tm);
    float2 *partials = reinterpret_cast<float2 *>(g.partials);
    // set-up: G = Z^T D Z from the moments M, projected right-hand side
    grid_sum_df<MIXED_GATHER_NP>(reinterpret_cast<const float2 *>(g.init_partials), g.init_stride, g.n_init, s_sc);
    const double f2 = s_sc[0];
    mixed_setup(g, s_sc, s_A6, s_tau, s_Om, &s_beta, &s_conv);
    float acc0[1] = {0.f};
    FFEA_NODE_LOOP(g, a) {
        float r0 = g.r[4 * a], r1 = g.r[4 * a + 1], r2 = g.r[4 * a + 2];
        if (defl) {
            const float4 d = g.dpos[a];
            r0 -= g.diag[4 * a] * (s_tau[0] + (s_Om[1] * d.z - s_Om[2] * d.y));
            r1 -= g.diag[4 * a + 1] * (s_tau[1] + (s_Om[2] * d.x - s_Om[0] * d.z));
            r2 -= g.diag[4 * a + 2] * (s_tau[2] + (s_Om[0] * d.y - s_Om[1] * d.x));
            g.r[4 * a] = r0; g.r[4 * a + 1] = r1; g.r[4 * a + 2] = r2;
        }
        g.x[4 * a] = 0.f; g.x[4 * a + 1] = 0.f; g.x[4 * a + 2] = 0.f;
        acc0[0] += r0 * (g.dinv[4 * a] * r0) + r1 * (g.dinv[4 * a + 1] * r1) + r2 * (g.dinv[4 * a + 2] * r2);
    }
    const int row0 = MIXED_A_NP + MIXED_B_NP;
    {
        df32 o[1];
        block_reduce_f<1>(acc0, smemf, o);
        if (threadIdx.x == 0) partials[row0 * g.stride + blockIdx.x] = make_float2(o[0].hi, o[0].lo);
    }
    unsigned int bar_ep = 0;  // grid barriers passed
    bool ok = grid_sync_ep(g.gb, st, g.limit_ns, bar_ep);
    if (ok) {
        grid_sum_df<1>(partials + row0 * g.stride, 0, gridDim.x, s_sc);
        if (threadIdx.x == 0) s_delta = s_sc[0];
        __syncthreads();
    }
    float *pold = g.pbuf0, *pnew = g.pbuf1;
    FFEA_MARK(g, tm, 0);
    int it = 0;
    // a zero force (a blob exactly at rest without noise) has the solution x = 0: no iteration (the first step
    // length would be 0/0)
    if (f2 == 0.0 && threadIdx.x == 0) s_conv = 1;
    for (; ok && it < g.imax && f2 != 0.0; ++it) {
        const bool first = it == 0;
        const float beta = s_beta;
        // phase A: q = V p with p formed on the fly; p.q; moments of D p for Z^T D p
        float acc[MIXED_A_NP];
#pragma unroll
        for (int i = 0; i < MIXED_A_NP; ++i) acc[i] = 0.f;
        {
            FFEA_SPMV_LOOP(g, a, sub, valid) {
                float q0, q1, q2;
                spmv_row_fly<B3>(g, pold, beta, first, a, sub, valid, q0, q1, q2);
                if (!valid || sub != 0) continue;
                float p0, p1, p2;
                p_on_the_fly(g, pold, beta, first, a, p0, p1, p2);
                pnew[4 * a] = p0; pnew[4 * a + 1] = p1; pnew[4 * a + 2] = p2;
                g.q[4 * a] = q0; g.q[4 * a + 1] = q1; g.q[4 * a + 2] = q2;
                acc[0] += p0 * q0 + p1 * q1 + p2 * q2;
                if (defl) {
                    const float4 d = g.dpos[a];
                    const float e0 = g.diag[4 * a] * p0, e1 = g.diag[4 * a + 1] * p1, e2 = g.diag[4 * a + 2] * p2;
                    acc[1] += e0; acc[2] += e1; acc[3] += e2;
                    acc[4] += d.y * e2 - d.z * e1;
                    acc[5] += d.z * e0 - d.x * e2;
                    acc[6] += d.x * e1 - d.y * e0;
                }
            }
        }
        FFEA_MARK(g, tm, 1);
        {
            df32 o[MIXED_A_NP];
            block_reduce_f<MIXED_A_NP>(acc, smemf, o);
            if (threadIdx.x == 0)
#pragma unroll
                for (int i = 0; i < MIXED_A_NP; ++i) partials[i * g.stride + blockIdx.x] = make_float2(o[i].hi, o[i].lo);
        }
        FFEA_MARK(g, tm, 2);
        if (!(ok = grid_sync_ep(g.gb, st, g.limit_ns, bar_ep))) break;
        FFEA_MARK(g, tm, 3);
        grid_sum_df<MIXED_A_NP>(partials, g.stride, gridDim.x, s_sc);
        // (tau, Omega) = A6 S over six lanes of warp 0; p.V~p = p.q + S . (tau, Omega); alpha = delta / p.V~p
        if (threadIdx.x < 32) {
            const int l = threadIdx.x;
            double tO = 0.0;
            if (defl && l < 6) {
#pragma unroll
                for (int q = 0; q < 6; ++q) tO += s_A6[6 * l + q] * s_sc[1 + q];
            }
            double prod = (l < 6) ? tO * s_sc[1 + l] : 0.0;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) prod += __shfl_xor_sync(0xffffffffu, prod, o);
            if (l < 6) {
                if (l < 3) s_tau[l] = (float)tO; else s_Om[l - 3] = (float)tO;
            }
            if (l == 0) s_alpha = (float)s_delta / (float)(s_sc[0] + prod);
        }
        __syncthreads();
        FFEA_MARK(g, tm, 4);
        const float alpha = s_alpha;
        const float t0 = s_tau[0], t1 = s_tau[1], t2 = s_tau[2], O0 = s_Om[0], O1 = s_Om[1], O2 = s_Om[2];
        // phase B: x += alpha p ; r -= alpha (q + D (tau + Omega x d)) ; r.r ; r.z
        float acc2[MIXED_B_NP] = {0.f, 0.f};
        FFEA_NODE_LOOP(g, a) {
#pragma unroll
            for (int c = 0; c < 3; ++c) g.x[4 * a + c] += alpha * pnew[4 * a + c];
            float q0 = g.q[4 * a], q1 = g.q[4 * a + 1], q2 = g.q[4 * a + 2];
            if (defl) {
                const float4 d = g.dpos[a];
                q0 += g.diag[4 * a] * (t0 + (O1 * d.z - O2 * d.y));
                q1 += g.diag[4 * a + 1] * (t1 + (O2 * d.x - O0 * d.z));
                q2 += g.diag[4 * a + 2] * (t2 + (O0 * d.y - O1 * d.x));
            }
            const float r0 = g.r[4 * a] - alpha * q0, r1 = g.r[4 * a + 1] - alpha * q1, r2 = g.r[4 * a + 2] - alpha * q2;
            g.r[4 * a] = r0; g.r[4 * a + 1] = r1; g.r[4 * a + 2] = r2;
            acc2[0] += r0 * r0 + r1 * r1 + r2 * r2;
            acc2[1] += r0 * (g.dinv[4 * a] * r0) + r1 * (g.dinv[4 * a + 1] * r1) + r2 * (g.dinv[4 * a + 2] * r2);
        }
        FFEA_MARK(g, tm, 5);
        {
            df32 o[MIXED_B_NP];
            block_reduce_f<MIXED_B_NP>(acc2, smemf, o);
            if (threadIdx.x == 0)
                for (int i = 0; i < MIXED_B_NP; ++i)
                    partials[(MIXED_A_NP + i) * g.stride + blockIdx.x] = make_float2(o[i].hi, o[i].lo);
        }
        FFEA_MARK(g, tm, 6);
        if (!(ok = grid_sync_ep(g.gb, st, g.limit_ns, bar_ep))) break;
        FFEA_MARK(g, tm, 7);
        grid_sum_df<MIXED_B_NP>(partials + MIXED_A_NP * g.stride, g.stride, gridDim.x, s_sc);
        if (threadIdx.x == 0) {
            // |r|^2/|f|^2 < epsilon2 tested as |r|^2 < epsilon2 |f|^2 (f2 == 0 counts as converged)
            s_conv = (g.check_last || it + 1 < g.imax) && (f2 == 0.0 || s_sc[0] < g.eps2 * f2);
            if (blockIdx.x == 0 && it < g.hist_cap) g.history[it] = (f2 == 0.0) ? 0.0 : s_sc[0] / f2;
            const double delta_old = s_delta;
            s_delta = s_sc[1];
            s_beta = (float)s_delta / (float)delta_old;
        }
        __syncthreads();
        FFEA_MARK(g, tm, 8);
        if (s_conv) {
            ++it;
            break;
        }
        float *t = pold; pold = pnew; pnew = t;
    }
    FFEA_PHASES_END(g);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (!ok) {
            st->abort = 1;
        } else if (!s_conv) {
            st->cg_fail = 1;
            st->abort = 1;
            st->last_iters = g.imax;
            st->total_iters += g.imax;
        } else {
            st->last_iters = it;
            st->total_iters += it;
        }
    }
}

// Block reduction of NV FP32 per-thread values straight into the per-block partial rows: FP32 within
// each warp, then warp w sums values w, w + (warps), ... over the warps in double-float and its lane 0
// stores the pairs. The caller must pass a __syncthreads() before smem is written again.
template <int NV>
__device__ __forceinline__ void block_reduce_store(const float (&v)[NV], float *smem, float2 *partials, int stride,
                                                   int row0) {
    const int lane = threadIdx.x & 31, wid = warp_index(), nw = blockDim.x >> 5;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const float w = warp_sum_f(v[i]);
        if (lane == 0) smem[i * 32 + wid] = w;
    }
    __syncthreads();
    for (int i = wid; i < NV; i += nw) {
        df32 t = {lane < nw ? smem[i * 32 + lane] : 0.f, 0.f};
        t = warp_sum_df(t);
        if (lane == 0) partials[(row0 + i) * stride + blockIdx.x] = make_float2(t.hi, t.lo);
    }
}

// grid_sum_df with each lane's loads issued eight at a time before their sums: the same fixed order, the
// partials' L2 latency paid once per 256 blocks.
__device__ __forceinline__ void put_sum(double *s, df32 t) { *s = (double)t.hi + (double)t.lo; }
__device__ __forceinline__ void put_sum(df32 *s, df32 t) { *s = t; }

template <int NV, class T>
__device__ __forceinline__ void grid_sum_df8(const float2 *partials, int stride, int nb, T *s_out) {
    const int lane = threadIdx.x & 31, wid = warp_index(), nw = blockDim.x >> 5;
    for (int i = wid; i < NV; i += nw) {
        df32 t = {0.f, 0.f};
        for (int b0 = 0; b0 < nb; b0 += 256) {
            float2 q[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int b = b0 + lane + 32 * j;
                q[j] = (b < nb) ? __ldcg(partials + i * stride + b) : make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) t = df_add(t, df32{q[j].x, q[j].y});
        }
        t = warp_sum_df(t);
        if (lane == 0) put_sum(s_out + i, t);
    }
    __syncthreads();
}

// The same row with U blocks per trip (3x3 blocks only): all U blocks' loads (columns, values, z and p) issue
// before any of their products, so U of the row's dependent DRAM round trips overlap; the products are
// accumulated in spmv_row_z's order, so the result is identical.
template <int U, class A>
__device__ __forceinline__ void spmv_row_zu(const A &g, const float4 *z4, const float4 *p4, float beta, bool first,
                                            int a, int sub, bool valid, float &q0, float &q1, float &q2) {
    q0 = 0.f; q1 = 0.f; q2 = 0.f;
    const int tpn = g.tpn;
    if (valid) {
        const int s = a >> 5, lane = a & 31;
        const int base = __ldg(g.slice_ptr + s);
        const int len = __ldg(g.rowlen + a);
        const float *v = g.val + 9 * (size_t)base + lane;
#pragma unroll 1
        for (int k = sub; k < len; k += U * tpn) {
            int bc[U];
            float w[U][9];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int ku = k + u * tpn;
                const bool in = ku < len;
                bc[u] = in ? __ldg(g.bcol + base + 32 * ku + lane) : 0;
                const float *vk = v + (size_t)32 * 9 * ku;
#pragma unroll
                for (int i = 0; i < 9; ++i) w[u][i] = in ? __ldg(vk + 32 * i) : 0.f;
            }
            float pz[U][3];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float4 z = z4[bc[u]];
                pz[u][0] = z.x; pz[u][1] = z.y; pz[u][2] = z.z;
                if (!first) {
                    const float4 po = p4[bc[u]];
                    pz[u][0] = fmaf(beta, po.x, pz[u][0]);
                    pz[u][1] = fmaf(beta, po.y, pz[u][1]);
                    pz[u][2] = fmaf(beta, po.z, pz[u][2]);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (k + u * tpn >= len) break;
                q0 = fmaf(w[u][0], pz[u][0], q0); q0 = fmaf(w[u][1], pz[u][1], q0); q0 = fmaf(w[u][2], pz[u][2], q0);
                q1 = fmaf(w[u][3], pz[u][0], q1); q1 = fmaf(w[u][4], pz[u][1], q1); q1 = fmaf(w[u][5], pz[u][2], q1);
                q2 = fmaf(w[u][6], pz[u][0], q2); q2 = fmaf(w[u][7], pz[u][1], q2); q2 = fmaf(w[u][8], pz[u][2], q2);
            }
        }
    }
    for (int o = 1; o < tpn; o <<= 1) {
        q0 += __shfl_xor_sync(0xffffffffu, q0, o);
        q1 += __shfl_xor_sync(0xffffffffu, q1, o);
        q2 += __shfl_xor_sync(0xffffffffu, q2, o);
    }
}

// Row a of q = V p for cg_mixed_own_kernel and cg_batch_kernel: p at a neighbour b is formed from the preconditioned residual
// z_b and the previous direction, both stored as float4 per node (two 16-byte loads per neighbour).
// The same row with two blocks per trip: both blocks' loads (values, columns, z and p) issue before
// either block's products, halving the chain of dependent L2 round trips per lane. The products are
// accumulated in the same order as spmv_row_z, so the result is identical.
// a read-only load with an L2 eviction policy (createpolicy)
__device__ __forceinline__ float ldg_l2(const float *p, uint64_t policy) {
    float v;
    asm("ld.global.nc.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(policy));
    return v;
}

template <class A>
__device__ __forceinline__ void spmv_row_z2(const A &g, const float4 *z4, const float4 *p4, float beta, bool first,
                                            int a, int sub, bool valid, uint64_t policy, float &q0, float &q1, float &q2) {
    q0 = 0.f; q1 = 0.f; q2 = 0.f;
    const int tpn = g.tpn;
    if (valid) {
        const int s = a >> 5, lane = a & 31;
        const int base = __ldg(g.slice_ptr + s);
        const int len = __ldg(g.rowlen + a);
        const float *v = g.val + 9 * (size_t)base + lane;
        int k = sub;
#pragma unroll 1
        for (; k + tpn < len; k += 2 * tpn) {
            const int ba = __ldg(g.bcol + base + 32 * k + lane), bb = __ldg(g.bcol + base + 32 * (k + tpn) + lane);
            const float *va = v + (size_t)32 * 9 * k, *vb = v + (size_t)32 * 9 * (k + tpn);
            float wa[9], wb[9];
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                wa[i] = ldg_l2(va + 32 * i, policy);
                wb[i] = ldg_l2(vb + 32 * i, policy);
            }
            const float4 za = z4[ba], zb = z4[bb];
            float pa0 = za.x, pa1 = za.y, pa2 = za.z, pb0 = zb.x, pb1 = zb.y, pb2 = zb.z;
            if (!first) {
                const float4 oa = p4[ba], ob = p4[bb];
                pa0 = fmaf(beta, oa.x, pa0); pa1 = fmaf(beta, oa.y, pa1); pa2 = fmaf(beta, oa.z, pa2);
                pb0 = fmaf(beta, ob.x, pb0); pb1 = fmaf(beta, ob.y, pb1); pb2 = fmaf(beta, ob.z, pb2);
            }
            q0 = fmaf(wa[0], pa0, q0); q0 = fmaf(wa[1], pa1, q0); q0 = fmaf(wa[2], pa2, q0);
            q1 = fmaf(wa[3], pa0, q1); q1 = fmaf(wa[4], pa1, q1); q1 = fmaf(wa[5], pa2, q1);
            q2 = fmaf(wa[6], pa0, q2); q2 = fmaf(wa[7], pa1, q2); q2 = fmaf(wa[8], pa2, q2);
            q0 = fmaf(wb[0], pb0, q0); q0 = fmaf(wb[1], pb1, q0); q0 = fmaf(wb[2], pb2, q0);
            q1 = fmaf(wb[3], pb0, q1); q1 = fmaf(wb[4], pb1, q1); q1 = fmaf(wb[5], pb2, q1);
            q2 = fmaf(wb[6], pb0, q2); q2 = fmaf(wb[7], pb1, q2); q2 = fmaf(wb[8], pb2, q2);
        }
        if (k < len) {
            const int b = __ldg(g.bcol + base + 32 * k + lane);
            const float *vk = v + (size_t)32 * 9 * k;
            float w[9];
#pragma unroll
            for (int i = 0; i < 9; ++i) w[i] = ldg_l2(vk + 32 * i, policy);
            const float4 z = z4[b];
            float p0 = z.x, p1 = z.y, p2 = z.z;
            if (!first) {
                const float4 po = p4[b];
                p0 = fmaf(beta, po.x, p0); p1 = fmaf(beta, po.y, p1); p2 = fmaf(beta, po.z, p2);
            }
            q0 = fmaf(w[0], p0, q0); q0 = fmaf(w[1], p1, q0); q0 = fmaf(w[2], p2, q0);
            q1 = fmaf(w[3], p0, q1); q1 = fmaf(w[4], p1, q1); q1 = fmaf(w[5], p2, q1);
            q2 = fmaf(w[6], p0, q2); q2 = fmaf(w[7], p1, q2); q2 = fmaf(w[8], p2, q2);
        }
    }
    for (int o = 1; o < tpn; o <<= 1) {
        q0 += __shfl_xor_sync(0xffffffffu, q0, o);
        q1 += __shfl_xor_sync(0xffffffffu, q1, o);
        q2 += __shfl_xor_sync(0xffffffffu, q2, o);
    }
}

template <class A>
__device__ __forceinline__ void spmv_row_z(const A &g, const float4 *z4, const float4 *p4, float beta, bool first,
                                           int a, int sub, bool valid, float &q0, float &q1, float &q2) {
    q0 = 0.f; q1 = 0.f; q2 = 0.f;
    const int tpn = g.tpn;
    if (valid) {
        const int s = a >> 5, lane = a & 31;
        const int base = __ldg(g.slice_ptr + s);
        const int len = __ldg(g.rowlen + a);
        if (g.block3) {
            const float *v = g.val + 9 * (size_t)base + lane;
            int k = sub;
            int bn = (k < len) ? __ldg(g.bcol + base + 32 * k + lane) : 0;
#pragma unroll 1
            for (; k < len; k += tpn) {
                const int b = bn;
                if (k + tpn < len) bn = __ldg(g.bcol + base + 32 * (k + tpn) + lane);
                const float *vk = v + (size_t)32 * 9 * k;
                const float v0 = __ldg(vk), v1 = __ldg(vk + 32), v2 = __ldg(vk + 64), v3 = __ldg(vk + 96),
                            v4 = __ldg(vk + 128), v5 = __ldg(vk + 160), v6 = __ldg(vk + 192), v7 = __ldg(vk + 224),
                            v8 = __ldg(vk + 256);
                const float4 z = z4[b];
                float p0 = z.x, p1 = z.y, p2 = z.z;
                if (!first) {
                    const float4 po = p4[b];
                    p0 = fmaf(beta, po.x, p0); p1 = fmaf(beta, po.y, p1); p2 = fmaf(beta, po.z, p2);
                }
                q0 = fmaf(v0, p0, q0); q0 = fmaf(v1, p1, q0); q0 = fmaf(v2, p2, q0);
                q1 = fmaf(v3, p0, q1); q1 = fmaf(v4, p1, q1); q1 = fmaf(v5, p2, q1);
                q2 = fmaf(v6, p0, q2); q2 = fmaf(v7, p1, q2); q2 = fmaf(v8, p2, q2);
            }
        } else {
            const float *v = g.val + base + lane;
            for (int k = sub; k < len; k += tpn) {
                const int b = __ldg(g.bcol + base + 32 * k + lane);
                const float m = __ldg(v + 32 * k);
                const float4 z = z4[b];
                float p0 = z.x, p1 = z.y, p2 = z.z;
                if (!first) {
                    const float4 po = p4[b];
                    p0 = fmaf(beta, po.x, p0); p1 = fmaf(beta, po.y, p1); p2 = fmaf(beta, po.z, p2);
                }
                q0 = fmaf(m, p0, q0);
                q1 = fmaf(m, p1, q1);
                q2 = fmaf(m, p2, q2);
            }
        }
    }
    for (int o = 1; o < tpn; o <<= 1) {
        q0 += __shfl_xor_sync(0xffffffffu, q0, o);
        q1 += __shfl_xor_sync(0xffffffffu, q1, o);
        q2 += __shfl_xor_sync(0xffffffffu, q2, o);
    }
}

// The vector a staged SpMV reads, in shared memory: this block's rows at v[0, npb), then its halo. A thread's own
// published row waits in its registers until the block's reads of the previous vector have ended.
struct Staged {
    float4 *v;
    int npb;
    int row;  // the row this thread has published but not yet staged (-1: none), and its value
    float4 own;
};

// The halo of this block for publication `tag`: every thread reads its messages (two of them in flight) and puts
// them, and its own published row, into the staged vector. The first barrier ends the reads of the previous vector.
template <bool BATCH, class A>
__device__ __forceinline__ bool halo_exchange(const A &g, Staged &z, const int (&hx)[2], int h0, int nh,
                                              unsigned int tag, DevStatus *st) {
    __syncthreads();
    if (z.row >= 0) z.v[z.row] = z.own;
    z.row = -1;
    int bad = 0;
    if (nh > 0) {
        const Msg *m = g.msg + (size_t)(tag & 1u) * g.mstride;
        float4 *zh = z.v + z.npb;
        for (int h = threadIdx.x, t = 0; h < nh; h += 2 * (int)blockDim.x, ++t) {
            const int h2 = h + (int)blockDim.x;
            const bool use[2] = {true, h2 < nh};
            const Msg *const at[2] = {m + (t == 0 ? hx[0] : __ldg(g.halo_list + h0 + h)),
                                      m + (!use[1] ? 0 : t == 0 ? hx[1] : __ldg(g.halo_list + h0 + h2))};
            Msg v[2];
            if (!msg_wait_all<2>(at, use, tag, v, st, BATCH ? MSG_POLLS_BATCH : MSG_POLLS)) { bad = 1; break; }
            zh[h] = make_float4(__uint_as_float(v[0].x), __uint_as_float(v[0].y), __uint_as_float(v[0].z), 0.f);
            if (use[1])
                zh[h2] = make_float4(__uint_as_float(v[1].x), __uint_as_float(v[1].y), __uint_as_float(v[1].z), 0.f);
        }
    }
    return __syncthreads_or(bad) == 0;
}

// The warp's sums of NV values (NV <= 16) over its lanes, one value left to each pair of lanes: each round halves
// the lanes a value is spread over and the values a lane holds, so 11 values take 13 shuffles instead of 55. Returns
// the sum and its index (-1 in lanes that hold none).
template <int NV>
__device__ __forceinline__ float warp_sum_spread(const float (&v)[NV], int &index) {
    constexpr int n1 = (NV + 1) / 2, n2 = (n1 + 1) / 2, n3 = (n2 + 1) / 2, n4 = (n3 + 1) / 2;
    static_assert(n4 == 1, "up to 16 values");
    const int lane = threadIdx.x & 31;
    float a[n1];
    int at = 0, valid = NV;
    auto round = [&](auto &dst, const auto &src, int n, int h, int o) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const float lo = src[i], hi = i + h < n ? src[i + h < n ? i + h : 0] : 0.f;
            dst[i] = (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, o);
        }
        at += up ? h : 0;
        valid = up ? valid - h : min(valid, h);  // how many of this lane's values are real
    };
    round(a, v, NV, n1, 16);
    float b[n2], c[n3], d[1];
    round(b, a, n1, n2, 8);
    round(c, b, n2, n3, 4);
    round(d, c, n3, n4, 2);
    const float t = d[0] + __shfl_xor_sync(0xffffffffu, d[0], 1);
    index = (valid > 0 && (lane & 1) == 0) ? at : -1;
    return t;
}

// The sums over nb blocks (this one of rank `rank`) of NV per-thread FP32 values, as double-float pairs in s_out for the whole block: FP32 within each
// warp, double-float over the block's warps, published as one message per value, and every block adds the blocks'
// messages in the same order. `tag` counts the launch's reductions from 1. The caller must pass a __syncthreads()
// before smem (NV x 32 floats) is written again.
template <int NV, bool BATCH, class A>
__device__ __forceinline__ bool grid_reduce_msg(const A &g, int rank, int nb, const float (&v)[NV], float *smem,
                                                unsigned int tag, df32 *s_out, DevStatus *st, GridBarrier *gb) {
    const int lane = threadIdx.x & 31, wid = warp_index(), nw = blockDim.x >> 5;
    int idx;
    const float ws = warp_sum_spread<NV>(v, idx);
    if (idx >= 0) smem[idx * 32 + wid] = ws;
    __syncthreads();
    if (nb > MSG_SUM_BLOCKS) {
        float2 *const rows = reinterpret_cast<float2 *>(g.rmsg) + (size_t)(tag & 1u) * MSG_VALUES * g.stride;
        for (int i = wid; i < NV; i += nw) {
            df32 t = {lane < nw ? smem[i * 32 + lane] : 0.f, 0.f};
            t = warp_sum_df(t);
            if (lane == 0) rows[i * g.stride + rank] = make_float2(t.hi, t.lo);
        }
        unsigned int epoch = tag - 1u;
        if (!barrier_ep(gb, (unsigned)nb, st, BATCH ? WAIT_LIMIT_BATCH_NS : WAIT_LIMIT_NS, epoch)) return false;
        grid_sum_df8<NV>(rows, g.stride, nb, s_out);
        return true;
    }
    int bad = 0;
    for (int i = wid; i < NV; i += nw) {
        df32 t = {lane < nw ? smem[i * 32 + lane] : 0.f, 0.f};
        t = warp_sum_df(t);
        if (nb > 1) {
            Msg *const rows = g.rmsg + ((size_t)(tag & 1u) * MSG_VALUES + i) * MSG_COPIES * g.stride;
            const Msg *const row = rows + (size_t)(rank % MSG_COPIES) * g.stride;
            if (lane < MSG_COPIES)
                msg_put(rows + (size_t)lane * g.stride + rank, __float_as_uint(t.hi), __float_as_uint(t.lo), 0u, tag);
            t = df32{0.f, 0.f};
            if (!msg_collect(row, nb, tag, st, [&](const Msg &m) {
                    t = df_add(t, df32{__uint_as_float(m.x), __uint_as_float(m.y)});
                }, BATCH ? MSG_POLLS_BATCH : MSG_POLLS))
                bad = 1;
            __syncwarp();
            t = warp_sum_df(t);
        }
        if (lane == 0) s_out[i] = t;
    }
    return __syncthreads_or(bad) == 0;
}

// Bytes of dynamic shared memory cg_mixed_own_kernel needs for npb owned rows: x, r, q, p, D^{-1}, D, d.
constexpr int OWN_FIELDS = 21;
__host__ __device__ constexpr size_t own_smem_bytes(int npb) { return (size_t)OWN_FIELDS * npb * sizeof(float); }

// The mixed CG of cg_mixed_kernel with each block owning a fixed run of npb rows: the rows' x, r, q, p,
// D^{-1}, D and offsets stay in shared memory for the whole solve, the block computes its own rows' SpMV,
// and only what other blocks read goes to global memory: z = D^{-1} r (in the q buffer) and the search
// direction (double-buffered). The arithmetic is the same as cg_mixed_kernel's: p = z + beta p_old is
// formed identically by the owner and by every block that reads row b as a neighbour.
template <class R>
__global__ void __launch_bounds__(1024, 1) cg_mixed_own_kernel(const __grid_constant__ CgArgs<R> g) {
    static_assert(sizeof(R) == sizeof(float), "the owned-rows CG is the mixed path's");
    extern __shared__ float sn[];
    __shared__ float smemf[MIXED_A_NP * 32];
    __shared__ double s_sc[MIXED_GATHER_NP];
    __shared__ double s_A6[36];
    __shared__ df32 s_A6f[36], s_scf[MIXED_A_NP];
    __shared__ float s_alpha, s_beta, s_tau[3], s_Om[3];
    __shared__ df32 s_delta;
    __shared__ int s_conv;
    DevStatus *st = g.st;
    if (st->abort) return;
    const bool defl = g.nmodes > 0;
    FFEA_PHASES_BEGIN(g, tm);
    float2 *partials = reinterpret_cast<float2 *>(g.partials);
    const int npb = g.npb, a0 = blockIdx.x * npb;
    const int nloc = max(0, min(npb, g.N - a0));
    float *sx = sn, *sr = sn + 3 * npb, *sq = sn + 6 * npb, *sp = sn + 9 * npb, *sdi = sn + 12 * npb,
          *sdg = sn + 15 * npb, *sd = sn + 18 * npb;
    float4 *z4 = reinterpret_cast<float4 *>(g.q);
    grid_sum_df8<MIXED_GATHER_NP>(reinterpret_cast<const float2 *>(g.init_partials), g.init_stride, g.n_init, s_sc);
    const double f2 = s_sc[0];
    mixed_setup(g, s_sc, s_A6, s_tau, s_Om, &s_beta, &s_conv);
    float acc0[1] = {0.f};
    for (int l = threadIdx.x; l < nloc; l += blockDim.x) {
        const int a = a0 + l;
        float r0 = g.r[4 * a], r1 = g.r[4 * a + 1], r2 = g.r[4 * a + 2];
        const float i0 = g.dinv[4 * a], i1 = g.dinv[4 * a + 1], i2 = g.dinv[4 * a + 2];
        if (defl) {
            const float4 d = g.dpos[a];
            const float D0 = g.diag[4 * a], D1 = g.diag[4 * a + 1], D2 = g.diag[4 * a + 2];
            r0 -= D0 * (s_tau[0] + (s_Om[1] * d.z - s_Om[2] * d.y));
            r1 -= D1 * (s_tau[1] + (s_Om[2] * d.x - s_Om[0] * d.z));
            r2 -= D2 * (s_tau[2] + (s_Om[0] * d.y - s_Om[1] * d.x));
            sdg[l] = D0; sdg[npb + l] = D1; sdg[2 * npb + l] = D2;
            sd[l] = d.x; sd[npb + l] = d.y; sd[2 * npb + l] = d.z;
        }
        sr[l] = r0; sr[npb + l] = r1; sr[2 * npb + l] = r2;
        sdi[l] = i0; sdi[npb + l] = i1; sdi[2 * npb + l] = i2;
        sx[l] = 0.f; sx[npb + l] = 0.f; sx[2 * npb + l] = 0.f;
        const float z0 = i0 * r0, z1 = i1 * r1, z2 = i2 * r2;
        z4[a] = make_float4(z0, z1, z2, 0.f);
        acc0[0] += r0 * z0 + r1 * z1 + r2 * z2;
    }
    if (threadIdx.x < 36) s_A6f[threadIdx.x] = df_of(s_A6[threadIdx.x]);
    const df32 tol = df_of_up(g.eps2 * f2);
    const int row0 = MIXED_A_NP + MIXED_B_NP;
    block_reduce_store<1>(acc0, smemf, partials, g.stride, row0);
    unsigned int bar_ep = 0;  // grid barriers passed
    bool ok = grid_sync_ep(g.gb, st, g.limit_ns, bar_ep);
    if (ok) {
        grid_sum_df8<1>(partials + row0 * g.stride, 0, gridDim.x, s_scf);
        if (threadIdx.x == 0) s_delta = s_scf[0];
        __syncthreads();
    }
    const float4 *pold = reinterpret_cast<const float4 *>(g.pbuf0);
    float4 *pnew = reinterpret_cast<float4 *>(g.pbuf1);
    uint64_t keep, stream;
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(keep));
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(stream));
    const int tpn = g.tpn, gpb = blockDim.x / tpn, grp = threadIdx.x / tpn, sub = threadIdx.x % tpn;
    const int npass = (nloc + gpb - 1) / gpb;
    FFEA_MARK(g, tm, 0);
    int it = 0;
    // a zero force (a blob exactly at rest without noise) has the solution x = 0: no iteration
    if (f2 == 0.0 && threadIdx.x == 0) s_conv = 1;
    for (; ok && it < g.imax && f2 != 0.0; ++it) {
        const bool first = it == 0;
        const float beta = s_beta;
        // phase A: q = V p over the block's rows (p formed on the fly); p.q; moments of D p
        float acc[MIXED_A_NP];
#pragma unroll
        for (int i = 0; i < MIXED_A_NP; ++i) acc[i] = 0.f;
        for (int ps = 0; ps < npass; ++ps) {
            const int l = ps * gpb + grp;
            const bool valid = l < nloc;
            float q0, q1, q2;
            if (g.block3)
                spmv_row_z2(g, z4, pold, beta, first, a0 + l, sub, valid, ((a0 + l) >> 5 & 7) < g.l2_keep ? keep : stream, q0,
                            q1, q2);
            else spmv_row_z(g, z4, pold, beta, first, a0 + l, sub, valid, q0, q1, q2);
            if (!valid || sub != 0) continue;
            const float z0 = sdi[l] * sr[l], z1 = sdi[npb + l] * sr[npb + l], z2 = sdi[2 * npb + l] * sr[2 * npb + l];
            float p0 = z0, p1 = z1, p2 = z2;
            if (!first) {
                p0 = fmaf(beta, sp[l], z0); p1 = fmaf(beta, sp[npb + l], z1); p2 = fmaf(beta, sp[2 * npb + l], z2);
            }
            sp[l] = p0; sp[npb + l] = p1; sp[2 * npb + l] = p2;
            sq[l] = q0; sq[npb + l] = q1; sq[2 * npb + l] = q2;
            pnew[a0 + l] = make_float4(p0, p1, p2, 0.f);
            acc[0] += p0 * q0 + p1 * q1 + p2 * q2;
            if (defl) {
                const float dx = sd[l], dy = sd[npb + l], dz = sd[2 * npb + l];
                const float e0 = sdg[l] * p0, e1 = sdg[npb + l] * p1, e2 = sdg[2 * npb + l] * p2;
                acc[1] += e0; acc[2] += e1; acc[3] += e2;
                acc[4] += dy * e2 - dz * e1;
                acc[5] += dz * e0 - dx * e2;
                acc[6] += dx * e1 - dy * e0;
            }
        }
        FFEA_MARK(g, tm, 1);
        block_reduce_store<MIXED_A_NP>(acc, smemf, partials, g.stride, 0);
        FFEA_MARK(g, tm, 2);
        if (!(ok = grid_sync_ep(g.gb, st, g.limit_ns, bar_ep))) break;
        FFEA_MARK(g, tm, 3);
        grid_sum_df8<MIXED_A_NP>(partials, g.stride, gridDim.x, s_scf);
        if (warp_index() == 0) {
            // (tau, Omega) = A6 S; p.V~p = p.q + S . (tau, Omega); alpha = delta / p.V~p
            const int ln = threadIdx.x;
            df32 tO = {0.f, 0.f}, sv = tO;
            if (defl && ln < 6) {
                tO = df_mul(s_A6f[6 * ln], s_scf[1]);
#pragma unroll
                for (int qq = 1; qq < 6; ++qq) tO = df_add(tO, df_mul(s_A6f[6 * ln + qq], s_scf[1 + qq]));
                sv = s_scf[1 + ln];
            }
            df32 prod = df_mul(tO, sv);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) prod = df_add(prod, df_shfl_xor(prod, o));
            if (ln < 6) {
                if (ln < 3) s_tau[ln] = tO.hi; else s_Om[ln - 3] = tO.hi;
            }
            if (ln == 0) s_alpha = s_delta.hi / df_add(s_scf[0], prod).hi;
        }
        __syncthreads();
        FFEA_MARK(g, tm, 4);
        const float alpha = s_alpha;
        const float t0 = s_tau[0], t1 = s_tau[1], t2 = s_tau[2], O0 = s_Om[0], O1 = s_Om[1], O2 = s_Om[2];
        // phase B: x += alpha p ; r -= alpha (q + D (tau + Omega x d)) ; z = D^{-1} r ; r.r ; r.z
        float acc2[MIXED_B_NP] = {0.f, 0.f};
        for (int l = threadIdx.x; l < nloc; l += blockDim.x) {
            float p[3], qv[3], rv[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                p[c] = sp[c * npb + l];
                qv[c] = sq[c * npb + l];
                sx[c * npb + l] += alpha * p[c];
            }
            if (defl) {
                const float dx = sd[l], dy = sd[npb + l], dz = sd[2 * npb + l];
                qv[0] += sdg[l] * (t0 + (O1 * dz - O2 * dy));
                qv[1] += sdg[npb + l] * (t1 + (O2 * dx - O0 * dz));
                qv[2] += sdg[2 * npb + l] * (t2 + (O0 * dy - O1 * dx));
            }
            float z[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                rv[c] = sr[c * npb + l] - alpha * qv[c];
                sr[c * npb + l] = rv[c];
                z[c] = sdi[c * npb + l] * rv[c];
            }
            z4[a0 + l] = make_float4(z[0], z[1], z[2], 0.f);
            acc2[0] += rv[0] * rv[0] + rv[1] * rv[1] + rv[2] * rv[2];
            acc2[1] += rv[0] * z[0] + rv[1] * z[1] + rv[2] * z[2];
        }
        FFEA_MARK(g, tm, 5);
        block_reduce_store<MIXED_B_NP>(acc2, smemf, partials, g.stride, MIXED_A_NP);
        FFEA_MARK(g, tm, 6);
        if (!(ok = grid_sync_ep(g.gb, st, g.limit_ns, bar_ep))) break;
        FFEA_MARK(g, tm, 7);
        grid_sum_df8<MIXED_B_NP>(partials + MIXED_A_NP * g.stride, g.stride, gridDim.x, s_scf);
        if (threadIdx.x == 0) {
            s_conv = (g.check_last || it + 1 < g.imax) && (f2 == 0.0 || df_less(s_scf[0], tol));
            if (blockIdx.x == 0 && it < g.hist_cap)  // divided by |f|^2 at the end
                reinterpret_cast<float2 *>(g.history)[it] = make_float2(s_scf[0].hi, s_scf[0].lo);
            s_beta = s_scf[1].hi / s_delta.hi;
            s_delta = s_scf[1];
        }
        __syncthreads();
        FFEA_MARK(g, tm, 8);
        if (s_conv) {
            ++it;
            break;
        }
        const float4 *t = pold; pold = pnew; pnew = const_cast<float4 *>(t);
    }
    // the solution (and residual) back to global memory
    for (int l = threadIdx.x; l < nloc; l += blockDim.x) {
        const int a = a0 + l;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            g.x[4 * a + c] = sx[c * npb + l];
            g.r[4 * a + c] = sr[c * npb + l];
        }
    }
    FFEA_PHASES_END(g);
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < min(it, g.hist_cap); i += blockDim.x) {
            const float2 h = reinterpret_cast<const float2 *>(g.history)[i];
            g.history[i] = f2 == 0.0 ? 0.0 : df_double(df32{h.x, h.y}) / f2;
        }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (!ok) {
            st->abort = 1;
        } else if (!s_conv) {
            st->cg_fail = 1;
            st->abort = 1;
            st->last_iters = g.imax;
            st->total_iters += g.imax;
        } else {
            st->last_iters = it;
            st->total_iters += it;
        }
    }
}

// 3x3 blocks of each owned row of cg_mixed_sr_kernel kept in shared memory for the whole solve, kc of them after
// those in registers (RowRegs): values 0-3, 4-7 and 8 of block k of row l at a[k S + l], b[k S + l], c[k S + l], its
// local column at col[k S + l]. S is the block's row count padded to S = 8 / tpn (mod 8), so that the quarter warps'
// 16-byte reads (8 / tpn rows x the row's tpn lanes, on blocks k, k + 1, ...) fall on distinct banks.
struct SrCache {
    const float4 *a, *b;
    const float *c;
    const unsigned short *col;
    int kc, S;
};

__host__ __device__ inline int sr_cache_stride(int npb, int tpn) {
    int S = npb;
    while (tpn > 1 && (S & 7) != 8 / tpn) ++S;
    return S;
}

#define FFEA_W_FMA(WV, ZV)                                                                   \
    w0 = fmaf(WV[0], ZV.x, w0); w0 = fmaf(WV[1], ZV.y, w0); w0 = fmaf(WV[2], ZV.z, w0);        \
    w1 = fmaf(WV[3], ZV.x, w1); w1 = fmaf(WV[4], ZV.y, w1); w1 = fmaf(WV[5], ZV.z, w1);        \
    w2 = fmaf(WV[6], ZV.x, w2); w2 = fmaf(WV[7], ZV.y, w2); w2 = fmaf(WV[8], ZV.z, w2)

// The first RB 3x3 blocks of each lane of cg_mixed_sr_kernel (blocks sub, sub + tpn, ... of its row), kept in
// registers for the whole solve, with their local columns two to a word. RB = 0: none.
template <int RB>
struct RowRegs {
    float v[RB > 0 ? RB : 1][9];
    unsigned int c[RB > 0 ? (RB + 1) / 2 : 1];
};

// Row l (of its block; SELL base and length given) of w = V z for cg_mixed_sr_kernel, z staged in shared memory.
// Each lane takes blocks k = sub, sub + tpn, ... in order: first those in its
// registers, then those held in shared memory (RB tpn <= k < RB tpn + kc), then the rest from the matrix in global
// memory (two per trip where registers allow); the products are summed in block order either way, so the row does not depend on where its
// blocks are.
template <int RB, class A>
__device__ __forceinline__ void spmv_row_w(const A &g, int tpn, const SrCache &c, const RowRegs<RB> &rr, const float4 *zs,
                                           int base, int len, int lane, int l, int sub, float &w0, float &w1,
                                           float &w2) {
    w0 = 0.f; w1 = 0.f; w2 = 0.f;
    if (len > 0) {
        int k = sub;
        if constexpr (RB > 0) {
#pragma unroll
            for (int j = 0; j < RB; ++j, k += tpn) {
                if (k < len) {
                    const float4 z = zs[(j & 1) ? rr.c[j >> 1] >> 16 : rr.c[j >> 1] & 0xffffu];
                    FFEA_W_FMA(rr.v[j], z);
                }
            }
        }
        const int k0 = RB * tpn, kcl = min(k0 + c.kc, len);
#pragma unroll 1
        for (; k < kcl; k += tpn) {
            const int at = (k - k0) * c.S + l;
            const float4 va = c.a[at], vb = c.b[at];
            const float wk[9] = {va.x, va.y, va.z, va.w, vb.x, vb.y, vb.z, vb.w, c.c[at]};
            const float4 z = zs[c.col[at]];
            FFEA_W_FMA(wk, z);
        }
        const float *v = g.val + 9 * (size_t)base + lane;
#pragma unroll 1
        for (; RB == 0 && k + tpn < len; k += 2 * tpn) {
            const int ba = __ldg(g.lcol + base + 32 * k + lane), bb = __ldg(g.lcol + base + 32 * (k + tpn) + lane);
            const float *va = v + (size_t)32 * 9 * k, *vb = v + (size_t)32 * 9 * (k + tpn);
            float wa[9], wb[9];
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                wa[i] = __ldg(va + 32 * i);
                wb[i] = __ldg(vb + 32 * i);
            }
            const float4 za = zs[ba], zb = zs[bb];
            FFEA_W_FMA(wa, za);
            FFEA_W_FMA(wb, zb);
        }
#pragma unroll 1
        for (; k < len; k += tpn) {
            const int b = __ldg(g.lcol + base + 32 * k + lane);
            const float *vk = v + (size_t)32 * 9 * k;
            float wk[9];
#pragma unroll
            for (int i = 0; i < 9; ++i) wk[i] = __ldg(vk + 32 * i);
            const float4 z = zs[b];
            FFEA_W_FMA(wk, z);
        }
    }
    for (int o = 1; o < tpn; o <<= 1) {
        w0 += __shfl_xor_sync(0xffffffffu, w0, o);
        w1 += __shfl_xor_sync(0xffffffffu, w1, o);
        w2 += __shfl_xor_sync(0xffffffffu, w2, o);
    }
}
#undef FFEA_W_FMA

// cg_mixed_sr_kernel's forms: up to SR_REG_THREADS lanes a block with RB 3x3 blocks of each lane in registers (4 where a
// row has four lanes or more, so that they hold all of a usual row; else 6), or 1024 threads without (RB = 0).
constexpr int SR_REG_THREADS = 512;
template <int RB>
struct SrForm {
    static constexpr int THREADS = RB > 0 ? SR_REG_THREADS : 1024;
};
constexpr int SR_REG_ROWS = 128;  // rows a block is given while the mesh leaves SMs free

// sr_smem_bytes grows by the matrix cache of kc blocks per row at stride S: nine values and a local column each
constexpr int SR_CACHE_BYTES_PER_BLOCK = 9 * 4 + 2;
__host__ __device__ constexpr size_t sr_cache_bytes(int kc, int S) {
    return (size_t)SR_CACHE_BYTES_PER_BLOCK * kc * S;
}

// The Chebyshev preconditioner: degrees 2, 4, 6 and 8 (even degrees keep it positive definite whatever the
// estimate of lambda_max); the interval is [lambda_max / cheb_ratio(d), lambda_max]; the estimate comes from the
// Lanczos matrix of the first CHEB_REC iterations of a Jacobi-preconditioned solve. State (CHEB_STATE doubles):
// [0] the estimate (0: not yet known, -1: Jacobi kept), [1, 1 + CHEB_REC) step lengths, then as many direction
// coefficients, then [CHEB_KJ] the iterations of the Jacobi solve while the first polynomial solve (the trial)
// is pending, then (CHEB_COEF) the recurrence's coefficients for the estimate.
constexpr int CHEB_MAX = 8;
// the interval's width: degrees 4 and up gain from a wider one (40^3 Kuhn cube, degree 4, CG per step: ratio 30
// 4.24 ms, 60 4.10, 120 4.04, 250 4.06), degree 2 hardly (30 4.17, 60 4.14, 120 4.17 ms)
__host__ __device__ constexpr double cheb_ratio(int degree) { return degree > 2 ? 120.0 : 30.0; }
constexpr double CHEB_MARGIN = 1.05;
constexpr int CHEB_KJ = 1 + 2 * CHEB_REC;
constexpr int CHEB_COEF = CHEB_KJ + 1;
constexpr int CHEB_STATE = CHEB_COEF + 2 * CHEB_MAX + 2;

// Largest eigenvalue of the Lanczos matrix of n preconditioned-CG iterations (step lengths al, direction
// coefficients be, be[0] unused): T_ii = 1/al_i + be_i/al_{i-1}, T_i,i+1 = sqrt(be_{i+1})/al_i. The Sturm count of
// negative LDL^T pivots at 32 points at once, one to a lane (an FP64 instruction costs the same for one lane as for
// 32), narrows the interval between the largest diagonal entry and the Gershgorin bound 33-fold a round; by bisection
// on one thread it took 2.6 ms, three quarters of a 20^3-cell blob's first step. One whole warp, all lanes with the
// same arguments; w: scratch for 2 n doubles.
static __device__ __noinline__ double lanczos_lambda_max(const double *al, const double *be, int n, double *w) {
    const int lane = threadIdx.x & 31;
    double lo = 0.0, hi = 0.0;
    for (int i = lane; i < n; i += 32) {
        const double ia = 1.0 / al[i], ip = i > 0 ? 1.0 / al[i - 1] : 0.0, b = i > 0 ? be[i] : 0.0;
        const double d = ia + b * ip, er = i + 1 < n ? sqrt(be[i + 1]) * ia : 0.0;
        w[i] = d;
        w[n + i] = b * ip * ip;
        lo = fmax(lo, d);
        hi = fmax(hi, d + sqrt(b) * ip + er);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmax(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    __syncwarp();
    for (int it = 0; it < 8 && hi - lo > 1e-6 * hi; ++it) {
        const double h = (hi - lo) / 33.0, x = lo + (lane + 1) * h;
        int below = 0;
        double q = 1.0;
        for (int i = 0; i < n; ++i) {
            q = (w[i] - x) - (i > 0 ? w[n + i] / q : 0.0);
            if (q == 0.0) q = -1e-300;
            below += q < 0.0;
        }
        // the first point above every eigenvalue
        const unsigned int above = __ballot_sync(0xffffffffu, below == n);
        const int f = above ? __ffs(above) - 1 : 32;
        if (f < 32) hi = lo + (f + 1) * h;
        lo += f * h;
    }
    return hi;
}

// The Chebyshev recurrence's coefficients for an interval that ends at lmax, kept behind the estimate in the blob's
// state (CHEB_COEF: c1, c2, 1/theta and the rigid-mode shift's scale 1/P_d(0)). One thread.
static __device__ __noinline__ void cheb_coefficients(double *state, int degree) {
    const double b = state[0], a = b / cheb_ratio(degree), theta = 0.5 * (b + a), delta = 0.5 * (b - a);
    const double sigma = theta / delta;
    double *c = state + CHEB_COEF;
    // the same recurrence at lambda = 0, where the residual stays D^{-1} r, gives P_d(0)
    double rho = 1.0 / sigma, p0 = 1.0 / theta, d0 = p0;
    for (int j = 0; j < degree; ++j) {
        const double rn = 1.0 / (2.0 * sigma - rho);
        c[j] = rn * rho;
        c[CHEB_MAX + j] = 2.0 * rn / delta;
        d0 = rn * rho * d0 + 2.0 * rn / delta;
        p0 += d0;
        rho = rn;
    }
    c[2 * CHEB_MAX] = 1.0 / theta;
    c[2 * CHEB_MAX + 1] = 1.0 / p0;
}

// The mixed CG with one reduction per iteration (the single-synchronisation rearrangement of Chronopoulos and
// Gear, 1989): the SpMV is applied to the preconditioned residual z = M^{-1} r, w = V z, and the search
// direction's product follows from q = w~ + beta q_old, p = z + beta p_old, so beta is not needed before the
// SpMV. One sweep computes w and all the dot products the step needs (r.z, r.r, z.w, z.q_old, p_old.w and the
// rigid-mode moments of D z); p.q is then formed from them in double-float:
//     p.q = z.w~ + beta (z.q_old + p_old.w~) + beta^2 p_old.q_old,    w~ = w + D Z A6 Z^T D z.
// Rows are owned as in cg_mixed_own_kernel. With M = D (Jacobi) the iterates are, in exact arithmetic, those of the
// other mixed CG kernels; in FP32 they agree to rounding and converge in the same number of iterations.
// What bounds it is latency: a matrix pass waits for its neighbours' rows and a grid-wide sum for every block, each an
// L2 round trip or two, around little arithmetic. So the exchange and the sums travel as tagged messages (Msg: one
// round trip, no fence, no counter), the vector a pass reads is staged in shared memory (one gather of the halo
// instead of an L2 read per block), and the matrix stays on chip: RB blocks of each lane in registers, the next kc of
// each row in shared memory, what is left read from L2. 512 threads with 128 registers hold 6 blocks a lane
// (8 spilled, and the reloads missed the L1 that shared memory leaves: 3.51 against 3.09 ms per 40^3 step).
// us per step, counters and L2 reads before -> now: 6^3 cells 590 -> 306, 10^3 cells - -> 399, 20^3 1553 -> 737,
// 30^3 - -> 1221, 40^3 3805 -> 2483, 45^3 (without register blocks) 4624 -> 3756.
// Polynomial preconditioning (g.poly = d > 0, once lambda_max of D^{-1} V is known): M^{-1} = P_d(D^{-1} V) D^{-1},
// with 1 - lambda P_d(lambda) the Chebyshev polynomial of degree d + 1 on [lambda_max / cheb_ratio(d),
// lambda_max], scaled to 1 at 0. z is built by d steps of the Chebyshev iteration for V z = r from z = 0 (d SpMVs,
// each exchanging its input vector with the neighbour blocks only), which cut the number of iterations, and with
// it the number of grid-wide reductions, by 2.8x (d = 2) to 7.7x (d = 8) on the 40^3 Kuhn cube. The
// preconditioner is built from V without the rigid-mode shift: it is positive definite on the whole spectrum for
// even d, and maps a D-weighted rigid mode D Z c to P_d(0) Z c. The shift D Z A6 Z^T D is therefore scaled by
// 1 / P_d(0) while the polynomial applies, which puts the rigid modes' eigenvalue of M^{-1} V~ at 1, inside the
// cluster of the others (unscaled they sit at P_d(0), 15.7 for d = 4 on the 40^3 cube, which then needed 132
// iterations a step instead of 110). The scale changes the shifted operator only on the rigid modes, where the
// projected right-hand side has no component, so the solution is the same: the one with Z^T D x = 0.
// A batch's set-up moments of the blob's rows (sums 1 and 2 of the solve), in s_sc for the whole block; a call of its
// own, so that its 28 values share no registers with the solve.
template <class A, class B>
__device__ __noinline__ bool sr_moments(const A &g, const B &bl, int a0, int nloc, int rank, int nb, float *smemf,
                                        df32 *s_scf, double *s_sc) {
    // f.f, S1_f, S2_f and M = sum Phi^T D Phi (cf. gather_mixed_kernel), half of them per sum
    static_assert(MIXED_GATHER_NP == 28, "two sums of 14");
    float m[MIXED_GATHER_NP];
#pragma unroll
    for (int i = 0; i < MIXED_GATHER_NP; ++i) m[i] = 0.f;
    for (int l = threadIdx.x; l < nloc; l += blockDim.x) {
        const int a = a0 + l;
        const float4 d = make_float4((float)(g.px[a] - bl.xc[0]), (float)(g.py[a] - bl.xc[1]),
                                     (float)(g.pz[a] - bl.xc[2]), 0.f);
        const float F0 = g.r[4 * a], F1 = g.r[4 * a + 1], F2 = g.r[4 * a + 2];
        m[0] += F0 * F0 + F1 * F1 + F2 * F2;
        m[1] += F0; m[2] += F1; m[3] += F2;
        m[4] += d.y * F2 - d.z * F1; m[5] += d.z * F0 - d.x * F2; m[6] += d.x * F1 - d.y * F0;
        float phi[6][3];
        phi_cols(d.x, d.y, d.z, phi);
        const float D[3] = {g.diag[4 * a], g.diag[4 * a + 1], g.diag[4 * a + 2]};
        int k = 7;
#pragma unroll
        for (int i = 0; i < 6; ++i)
#pragma unroll
            for (int j = i; j < 6; ++j, ++k)
                m[k] += phi[i][0] * D[0] * phi[j][0] + phi[i][1] * D[1] * phi[j][1] + phi[i][2] * D[2] * phi[j][2];
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        float v[14];
#pragma unroll
        for (int i = 0; i < 14; ++i) v[i] = m[14 * half + i];
        if (!grid_reduce_msg<14, true>(bl, rank, nb, v, smemf, (unsigned)half + 1u, s_scf, g.st, bl.gb)) return false;
        if (threadIdx.x < 14) s_sc[14 * half + threadIdx.x] = df_double(s_scf[threadIdx.x]);
        __syncthreads();
    }
    return true;
}

// Every second iteration of a batch's solve forms q = V p from the matrix, one more pass: carried on by q = w~ + beta q
// alone, q gathers the rounding of every pass, and the batch's solutions were up to a third further from FP64 than by
// cg_batch_kernel's q = V p. rms error of the moves, streaming / q carried on / every 4th / 2nd / each direct: blobs of 4 to 8
// cells 4.9 / 6.5 / 5.9 / 5.3 / 5.2e-7, 9 to 14 8.0 / 8.5 / 8.8 / 8.1 / 8.3e-7, 20 to 30 16.7 / 19.7 / 18.2 / 17.6 / 16.7e-7;
// ms per step of 32 blobs of 8 to 32 cells 18.9 / 5.80 / 6.01 / 6.18 / 6.50. (In numpy the other vectors held in FP64 change
// nothing; a pass summed in FP64 would halve the error.)
constexpr int SR_DIRECT = 2;

// One solve by nb blocks, this one of rank `rank`, with the launch's arguments g and the blob's own bl: the whole grid for a blob (cg_mixed_sr_kernel), or one blob's
// blocks of a batch (BATCH: kernels_batch.cuh), which also forms the moments that the single blob's gather leaves in
// g.init_partials. Returns false on a timeout.
template <int RB, bool BATCH, class A, class B>
__device__ __forceinline__ bool sr_solve(const A &g, const B &bl, int rank, int nb) {
    extern __shared__ __align__(16) float4 sn_raw[];
    __shared__ float smemf[14 * 32];
    __shared__ double s_sc[MIXED_GATHER_NP];
    __shared__ double s_A6[36];
    __shared__ df32 s_scf[14];  // the iteration's sums
    __shared__ df32 s_tol;      // the stopping tolerance
    __shared__ df32 s_A6f[36];        // A6 times the shift's scale
    __shared__ df32 s_mp[6];          // moments of D p for the current direction
    __shared__ df32 s_pq;             // p.q~ of the previous iteration
    __shared__ float s_g;             // and its r.z
    __shared__ float s_alpha, s_beta, s_tau[3], s_Om[3], s_dummy;
    __shared__ float s_c1[CHEB_MAX], s_c2[CHEB_MAX], s_ith;
    __shared__ double s_shift;        // scale of the rigid-mode shift: 1 / P_d(0) with the polynomial, else 1
    __shared__ int s_conv, s_stop;
    DevStatus *st = g.st;
    const bool defl = bl.nmodes > 0;
    FFEA_PHASES_BEGIN(g, tm);
    const int npb = bl.npb, a0 = bl.row0 + rank * npb;
    const int nloc = max(0, min(npb, bl.N - rank * npb));
    // the staged vector first (16-byte aligned), then the row fields
    Staged zs;
    zs.v = reinterpret_cast<float4 *>(sn_raw);
    zs.npb = npb;
    zs.row = -1;
    zs.own = make_float4(0.f, 0.f, 0.f, 0.f);
    // then the matrix blocks in shared memory, then the row fields (see sr_smem_bytes, sr_cache_bytes)
    SrCache mc;
    mc.kc = bl.kc;
    mc.S = bl.kc > 0 ? sr_cache_stride(npb, bl.tpn) : 0;
    const int ncache = mc.kc * mc.S;
    float4 *const ca = zs.v + npb + bl.nhalo, *const cb = ca + ncache;
    float *const cc = reinterpret_cast<float *>(cb + ncache);
    float *const sn = cc + ncache;
    float *sx = sn, *sr = sn + 3 * npb, *sp = sn + 6 * npb, *sq = sn + 9 * npb, *sw = sn + 12 * npb,
          *sdi = sn + 15 * npb, *sdg = sn + 18 * npb, *sd = sn + 21 * npb;
    // polynomial preconditioner: u = M^{-1} r and the Chebyshev correction dd (the residual of the Chebyshev
    // iteration shares w's storage: w is dead between the update and the next SpMV)
    float *su = sn + 24 * npb, *sdd = sn + 27 * npb;
    {
        // the matrix blocks in shared memory, filled once for the solve; their columns after the row fields
        unsigned short *const col = reinterpret_cast<unsigned short *>(sn + (bl.poly > 0 ? SR_FIELDS_POLY : SR_FIELDS) * npb);
        const int k0 = RB * bl.tpn;
        for (int t = threadIdx.x; t < mc.kc * nloc; t += blockDim.x) {
            const int kl = t / nloc, l = t - kl * nloc, a = a0 + l, k = k0 + kl;
            if (k >= __ldg(g.rowlen + a)) continue;
            const int base = __ldg(g.slice_ptr + (a >> 5)), lane = a & 31, at = kl * mc.S + l;
            const float *vk = g.val + 9 * (size_t)base + lane + (size_t)32 * 9 * k;
            ca[at] = make_float4(__ldg(vk), __ldg(vk + 32), __ldg(vk + 64), __ldg(vk + 96));
            cb[at] = make_float4(__ldg(vk + 128), __ldg(vk + 160), __ldg(vk + 192), __ldg(vk + 224));
            cc[at] = __ldg(vk + 256);
            col[at] = __ldg(g.lcol + base + 32 * k + lane);
        }
        mc.a = ca; mc.b = cb; mc.c = cc; mc.col = col;
    }
    // this block's halo; a thread's first two entries in registers
    const int h0 = __ldg(bl.halo_ptr + rank), nh = __ldg(bl.halo_ptr + rank + 1) - h0;
    int hx[2];
    hx[0] = (int)threadIdx.x < nh ? __ldg(g.halo_list + h0 + threadIdx.x) : 0;
    hx[1] = (int)(threadIdx.x + blockDim.x) < nh ? __ldg(g.halo_list + h0 + threadIdx.x + blockDim.x) : 0;
    const int poly = bl.poly;
    const double lmax = poly > 0 ? bl.cheb[0] : 0.0;
    const bool cheb = lmax > 0.0;              // Chebyshev this solve
    const bool rec = poly > 0 && lmax == 0.0;  // Jacobi this solve, recording the Lanczos coefficients
    if (cheb) {
        const double *c = bl.cheb + CHEB_COEF;
        if ((int)threadIdx.x < poly) {
            s_c1[threadIdx.x] = (float)c[threadIdx.x];
            s_c2[threadIdx.x] = (float)c[CHEB_MAX + threadIdx.x];
        }
        if (threadIdx.x == 0) {
            s_ith = (float)c[2 * CHEB_MAX];
            s_shift = c[2 * CHEB_MAX + 1];
        }
    }
    if (!cheb && threadIdx.x == 0) s_shift = 1.0;
    unsigned int red_ep = 0;  // epochs of the sums over the blocks
    auto offset = [&](int a) {
        if constexpr (BATCH)
            return make_float4((float)(g.px[a] - bl.xc[0]), (float)(g.py[a] - bl.xc[1]), (float)(g.pz[a] - bl.xc[2]), 0.f);
        else
            return g.dpos[a];
    };
    if constexpr (BATCH) {
        if (!sr_moments(g, bl, a0, nloc, rank, nb, smemf, s_scf, s_sc)) return false;
        red_ep = 2;
    } else {
        grid_sum_df8<MIXED_GATHER_NP>(reinterpret_cast<const float2 *>(g.init_partials), g.init_stride, g.n_init, s_sc);
    }
    const double f2 = s_sc[0];
    mixed_setup(bl, s_sc, s_A6, s_tau, s_Om, &s_dummy, &s_conv);
    __syncthreads();
    const float ith = cheb ? s_ith : 0.f;
    // tpn lanes to a row, every row of the block at once (npb tpn <= blockDim)
    const int tpn = bl.tpn, l = threadIdx.x / tpn, sub = threadIdx.x % tpn;
    const bool valid = l < nloc;
    RowRegs<RB> rr;
    int rbase = 0, rlen = 0;
    if constexpr (RB > 0) {
        if (valid) {
            const int a = a0 + l, lane = a & 31;
            rbase = __ldg(g.slice_ptr + (a >> 5));
            rlen = __ldg(g.rowlen + a);
#pragma unroll
            for (int j = 0; j < RB; ++j) {
                const int k = sub + j * tpn;
                const bool in = k < rlen;
#pragma unroll
                for (int i = 0; i < 9; ++i)
                    rr.v[j][i] = in ? __ldg(g.val + 9 * (size_t)rbase + lane + (size_t)32 * (9 * k + i)) : 0.f;
                const unsigned int lc = in ? __ldg(g.lcol + rbase + 32 * k + lane) : 0u;
                rr.c[j >> 1] = (j & 1) ? rr.c[j >> 1] | lc << 16 : lc;
            }
        }
    }
    // row l of w = V z over the staged vector
    auto spmv = [&](float &w0, float &w1, float &w2) {
        int base = rbase, len = rlen;
        if constexpr (RB == 0) {
            base = valid ? __ldg(g.slice_ptr + ((a0 + l) >> 5)) : 0;
            len = valid ? __ldg(g.rowlen + a0 + l) : 0;
        }
        spmv_row_w<RB>(g, tpn, mc, rr, zs.v, base, len, (a0 + l) & 31, l, sub, w0, w1, w2);
    };
    unsigned int ep = 0;      // epochs of the published vectors
    // row l of the vector published as epoch `tag`: to the block's staged vector and to the other blocks
    auto publish = [&](unsigned int tag, int row, float v0, float v1, float v2) {
        zs.row = row;
        zs.own = make_float4(v0, v1, v2, 0.f);
        msg_put(g.msg + (size_t)(tag & 1u) * g.mstride + a0 + row, __float_as_uint(v0), __float_as_uint(v1), __float_as_uint(v2),
                tag);
    };
    // Chebyshev steps 1..d after step 0 published y0 = D^{-1} r / theta and left D^{-1} r in sw:
    // res -= D^{-1} V y, dd = c1 dd + c2 res, u += dd; each step publishes dd for the next one's SpMV, the last one
    // publishes u as z
    auto cheb_steps = [&]() -> bool {
        for (int j = 1; j <= poly; ++j) {
            const float c1 = s_c1[j - 1], c2 = s_c2[j - 1];
            float t[3];
            spmv(t[0], t[1], t[2]);
            if (valid && sub == 0) {
                float o[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const float res = sw[c * npb + l] - sdi[c * npb + l] * t[c];
                    sw[c * npb + l] = res;
                    const float dd = fmaf(c1, sdd[c * npb + l], c2 * res);
                    sdd[c * npb + l] = dd;
                    const float u = su[c * npb + l] + dd;
                    su[c * npb + l] = u;
                    o[c] = j < poly ? dd : u;
                }
                publish(ep + 1, l, o[0], o[1], o[2]);
            }
            ++ep;
            FFEA_MARK(g, tm, 6);
            if (!halo_exchange<BATCH>(g, zs, hx, h0, nh, ep, st)) return false;
            FFEA_MARK(g, tm, 7);
        }
        return true;
    };
    // r = f^ (projected), x = 0, p = q = 0, z = M^{-1} r published
    for (int l = threadIdx.x; l < nloc; l += blockDim.x) {
        const int a = a0 + l;
        float r0 = g.r[4 * a], r1 = g.r[4 * a + 1], r2 = g.r[4 * a + 2];
        const float i0 = g.dinv[4 * a], i1 = g.dinv[4 * a + 1], i2 = g.dinv[4 * a + 2];
        if (defl) {
            const float4 d = offset(a);
            const float D0 = g.diag[4 * a], D1 = g.diag[4 * a + 1], D2 = g.diag[4 * a + 2];
            r0 -= D0 * (s_tau[0] + (s_Om[1] * d.z - s_Om[2] * d.y));
            r1 -= D1 * (s_tau[1] + (s_Om[2] * d.x - s_Om[0] * d.z));
            r2 -= D2 * (s_tau[2] + (s_Om[0] * d.y - s_Om[1] * d.x));
            sdg[l] = D0; sdg[npb + l] = D1; sdg[2 * npb + l] = D2;
            sd[l] = d.x; sd[npb + l] = d.y; sd[2 * npb + l] = d.z;
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            sx[c * npb + l] = 0.f;
            sp[c * npb + l] = 0.f;
            sq[c * npb + l] = 0.f;
        }
        sr[l] = r0; sr[npb + l] = r1; sr[2 * npb + l] = r2;
        sdi[l] = i0; sdi[npb + l] = i1; sdi[2 * npb + l] = i2;
        const float z0 = i0 * r0, z1 = i1 * r1, z2 = i2 * r2;
        if (cheb) {
            const float y[3] = {z0 * ith, z1 * ith, z2 * ith}, zz[3] = {z0, z1, z2};
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                sw[c * npb + l] = zz[c];
                su[c * npb + l] = y[c];
                sdd[c * npb + l] = y[c];
            }
            publish(1u, l, y[0], y[1], y[2]);
        } else {
            publish(1u, l, z0, z1, z2);
        }
    }
    if (threadIdx.x < 6) s_mp[threadIdx.x] = df32{0.f, 0.f};
    if (threadIdx.x < 36) s_A6f[threadIdx.x] = df_of(s_A6[threadIdx.x] * s_shift);
    if (threadIdx.x == 0) { s_g = 0.f; s_pq = df32{0.f, 0.f}; s_stop = 0; }
    if (threadIdx.x == 0) s_tol = df_of_up(g.eps2 * f2);
    bool ok = halo_exchange<BATCH>(g, zs, hx, h0, nh, ++ep, st);
    if (ok && cheb) ok = cheb_steps();
    FFEA_MARK(g, tm, 0);
    int k = 0;  // updates applied so far
    s_conv = 0;
    for (; ok; ++k) {
        // w = V z over the block's rows, and the iteration's dot products
        float acc[MIXED_SR_NP];
#pragma unroll
        for (int i = 0; i < MIXED_SR_NP; ++i) acc[i] = 0.f;
        float w0, w1, w2;
        spmv(w0, w1, w2);
        if (valid && sub == 0) {
            sw[l] = w0; sw[npb + l] = w1; sw[2 * npb + l] = w2;
            const float r0 = sr[l], r1 = sr[npb + l], r2 = sr[2 * npb + l];
            float z0, z1, z2;
            if (cheb) {
                z0 = su[l]; z1 = su[npb + l]; z2 = su[2 * npb + l];
            } else {
                z0 = sdi[l] * r0; z1 = sdi[npb + l] * r1; z2 = sdi[2 * npb + l] * r2;
            }
            acc[0] += r0 * z0 + r1 * z1 + r2 * z2;
            acc[1] += r0 * r0 + r1 * r1 + r2 * r2;
            acc[2] += z0 * w0 + z1 * w1 + z2 * w2;
            acc[3] += z0 * sq[l] + z1 * sq[npb + l] + z2 * sq[2 * npb + l];
            acc[4] += sp[l] * w0 + sp[npb + l] * w1 + sp[2 * npb + l] * w2;
            if (defl) {
                const float dx = sd[l], dy = sd[npb + l], dz = sd[2 * npb + l];
                const float e0 = sdg[l] * z0, e1 = sdg[npb + l] * z1, e2 = sdg[2 * npb + l] * z2;
                acc[5] += e0; acc[6] += e1; acc[7] += e2;
                acc[8] += dy * e2 - dz * e1;
                acc[9] += dz * e0 - dx * e2;
                acc[10] += dx * e1 - dy * e0;
            }
        }
        FFEA_MARK(g, tm, 1);
        if (!(ok = grid_reduce_msg<MIXED_SR_NP, BATCH>(bl, rank, nb, acc, smemf, ++red_ep, s_scf, st, bl.gb))) break;
        FFEA_MARK(g, tm, 3);
        if (warp_index() == 0) {
            // The iteration's scalars, in double-float as the sums arrive: this chain is on every block's critical path
            // and FP64 runs at 1/64 of the FP32 rate (4.0 us per iteration; see below for the pairs').
            const int ln = threadIdx.x;
            // c = s A6 m(z): the rigid-mode coefficients of s D Z A6 Z^T D z, over six lanes
            df32 c = {0.f, 0.f}, mz = c, mp = c;
            if (defl && ln < 6) {
                c = df_mul(s_A6f[6 * ln], s_scf[5]);
#pragma unroll
                for (int qq = 1; qq < 6; ++qq) c = df_add(c, df_mul(s_A6f[6 * ln + qq], s_scf[5 + qq]));
                mz = s_scf[5 + ln];
                mp = s_mp[ln];
            }
            df32 mzc = df_mul(mz, c), mpc = df_mul(mp, c);  // m(z).c, m(p_old).c
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) {
                mzc = df_add(mzc, df_shfl_xor(mzc, o));
                mpc = df_add(mpc, df_shfl_xor(mpc, o));
            }
            const df32 gam = s_scf[0], rr2 = s_scf[1];
            // |r|^2/|f|^2 < epsilon2 after an update, as NoMassCGSolver::solve tests it (a zero force: x = 0 at once)
            const bool conv = f2 == 0.0 || (k > 0 && (g.check_last || k < g.imax) && df_less(rr2, s_tol));
            if (ln == 0 && rank == 0 && k > 0 && k - 1 < g.hist_cap)
                reinterpret_cast<float2 *>(g.history)[k - 1] = make_float2(rr2.hi, rr2.lo);
            const bool stop = conv || k >= g.imax;
            const float beta = (k == 0) ? 0.f : gam.hi / s_g;
            const df32 zw = df_add(s_scf[2], mzc), pw = df_add(s_scf[4], mpc), b1 = {beta, 0.f};
            const df32 pq = df_add(df_add(zw, df_mul(b1, df_add(s_scf[3], pw))), df_mul(df_mul(b1, b1), s_pq));
            const float alpha = gam.hi / pq.hi;
            if (rec && ln == 0 && rank == 0 && !stop && k < CHEB_REC) {
                bl.cheb[1 + k] = df_double(gam) / df_double(pq);
                bl.cheb[1 + CHEB_REC + k] = beta;
            }
            __syncwarp();
            if (ln < 6) s_mp[ln] = df_add(mz, df_mul(b1, mp));
            if constexpr (BATCH) {
                if (k % SR_DIRECT == SR_DIRECT - 1) {  // the coefficients for p in place of z
                    __syncwarp();
                    if (defl && ln < 6) {
                        c = df_mul(s_A6f[6 * ln], s_mp[0]);
#pragma unroll
                        for (int qq = 1; qq < 6; ++qq) c = df_add(c, df_mul(s_A6f[6 * ln + qq], s_mp[qq]));
                    }
                }
            }
            if (ln < 3) s_tau[ln] = c.hi; else if (ln < 6) s_Om[ln - 3] = c.hi;
            if (ln == 0) {
                s_conv = conv;
                s_stop = stop;
                s_beta = beta;
                s_alpha = alpha;
                s_g = gam.hi;
                s_pq = pq;
            }
        }
        __syncthreads();
        FFEA_MARK(g, tm, 4);
        if (s_stop) break;
        const float alpha = s_alpha, beta = s_beta;
        const float t0 = s_tau[0], t1 = s_tau[1], t2 = s_tau[2], O0 = s_Om[0], O1 = s_Om[1], O2 = s_Om[2];
        bool direct = false;  // q = V p of this iteration from the matrix
        if constexpr (BATCH) {
            direct = k % SR_DIRECT == SR_DIRECT - 1;
            if (direct) {
                if ((int)threadIdx.x < nloc) {
                    const int l = threadIdx.x;
                    float pv[3];
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float zc = cheb ? su[c * npb + l] : sdi[c * npb + l] * sr[c * npb + l];
                        sp[c * npb + l] = pv[c] = fmaf(beta, sp[c * npb + l], zc);
                    }
                    publish(ep + 1, l, pv[0], pv[1], pv[2]);
                }
                ++ep;
                if (!(ok = halo_exchange<BATCH>(g, zs, hx, h0, nh, ep, st))) break;
                float w0, w1, w2;
                spmv(w0, w1, w2);
                if (valid && sub == 0) { sw[l] = w0; sw[npb + l] = w1; sw[2 * npb + l] = w2; }
                __syncthreads();
            }
        }
        // p = z + beta p ; q = w~ + beta q ; x += alpha p ; r -= alpha q ; z = M^{-1} r published (Jacobi), or
        // the Chebyshev iteration's first step (polynomial)
        for (int l = threadIdx.x; l < nloc; l += blockDim.x) {
            float wv[3] = {sw[l], sw[npb + l], sw[2 * npb + l]};
            if (defl) {
                const float dx = sd[l], dy = sd[npb + l], dz = sd[2 * npb + l];
                wv[0] += sdg[l] * (t0 + (O1 * dz - O2 * dy));
                wv[1] += sdg[npb + l] * (t1 + (O2 * dx - O0 * dz));
                wv[2] += sdg[2 * npb + l] * (t2 + (O0 * dy - O1 * dx));
            }
            float zn[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float r = sr[c * npb + l], di = sdi[c * npb + l];
                const float zc = cheb ? su[c * npb + l] : di * r;
                const float pv = direct ? sp[c * npb + l] : fmaf(beta, sp[c * npb + l], zc);
                const float qv = direct ? wv[c] : fmaf(beta, sq[c * npb + l], wv[c]);
                sp[c * npb + l] = pv;
                sq[c * npb + l] = qv;
                sx[c * npb + l] += alpha * pv;
                const float rn = r - alpha * qv;
                sr[c * npb + l] = rn;
                zn[c] = di * rn;
                if (cheb) {
                    const float y = zn[c] * ith;
                    sw[c * npb + l] = zn[c];
                    su[c * npb + l] = y;
                    sdd[c * npb + l] = y;
                    zn[c] = y;
                }
            }
            publish(ep + 1, l, zn[0], zn[1], zn[2]);
        }
        FFEA_MARK(g, tm, 5);
        ++ep;
        if (!(ok = halo_exchange<BATCH>(g, zs, hx, h0, nh, ep, st))) break;
        FFEA_MARK(g, tm, 7);
        if (cheb && !(ok = cheb_steps())) break;
    }
    for (int l = threadIdx.x; l < nloc; l += blockDim.x) {
        const int a = a0 + l;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            g.x[4 * a + c] = sx[c * npb + l];
            g.r[4 * a + c] = sr[c * npb + l];
        }
    }
    FFEA_PHASES_END(g);
    if (rank == 0)  // the history's |r|^2, kept as pairs, become |r|^2 / |f|^2
        for (int i = threadIdx.x; i < min(k, g.hist_cap); i += blockDim.x) {
            const float2 h = reinterpret_cast<const float2 *>(g.history)[i];
            g.history[i] = f2 == 0.0 ? 0.0 : df_double(df32{h.x, h.y}) / f2;
        }
    double lm = 0.0;
    if (rank == 0 && rec && ok) {
        __syncthreads();  // the staged vector is done with
        if (warp_index() == 0 && s_conv && k >= 2)
            lm = lanczos_lambda_max(bl.cheb + 1, bl.cheb + 1 + CHEB_REC, min(k, CHEB_REC),
                                    reinterpret_cast<double *>(sn_raw));
    }
    if (rank == 0 && threadIdx.x == 0) {
        if (!ok) {
            atomicExch(&st->abort, 1);
        } else if (!s_conv) {
            atomicExch(&st->cg_fail, 1);
            if constexpr (BATCH) {
                // cg_fail alone: `abort` raised now could stop a block that another blob's blocks wait for;
                // batch_finish_kernel raises it
                *bl.blob_iters = g.imax;
            } else {
                st->abort = 1;
                st->last_iters = g.imax;
                st->total_iters += g.imax;
            }
        } else {
            if constexpr (BATCH) {
                *bl.blob_iters = k;
                atomicMax(&st->last_iters, k);
                atomicAdd(reinterpret_cast<unsigned long long *>(&st->total_iters), (unsigned long long)k);
            } else {
                st->last_iters = k;
                st->total_iters += k;
            }
            if (rec && k >= 2) {
                // the estimate of lambda_max(D^-1 V) for the next solves, from this Jacobi solve's Lanczos matrix
                if (isfinite(lm) && lm > 0.0) {
                    bl.cheb[0] = CHEB_MARGIN * lm;
                    bl.cheb[CHEB_KJ] = (double)k;
                    cheb_coefficients(bl.cheb, poly);
                }
            } else if (cheb && bl.cheb[CHEB_KJ] > 0.0) {
                // the trial: the polynomial is kept when its iterations, each costing 1 + poly * cheb_cost Jacobi
                // iterations, took less than the Jacobi solve (a well-conditioned matrix, e.g. with a large
                // Stokes drag on its diagonal, converges in a few Jacobi iterations and keeps Jacobi)
                if ((double)k * (1.0 + poly * (double)g.cheb_cost) >= bl.cheb[CHEB_KJ]) bl.cheb[0] = -1.0;
                bl.cheb[CHEB_KJ] = 0.0;
            }
        }
    }
    return ok;
}

template <class R, int RB>
__global__ void __launch_bounds__(SrForm<RB>::THREADS, 1) cg_mixed_sr_kernel(const __grid_constant__ CgArgs<R> g) {
    static_assert(sizeof(R) == sizeof(float), "the single-reduction CG is the mixed path's");
    if (g.st->abort) return;
    sr_solve<RB, false>(g, g, (int)blockIdx.x, (int)gridDim.x);
}

}  // namespace ffea
