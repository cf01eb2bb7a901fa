// Element kernels of P2 elements around the return mapping.
//
//   p2tet_factor           nine doubles per point in place of 30 (p2tet.cuh), checked against
//                          the gradients the mesh was given
//   k_response3d           strain, Davis reduction, return mapping (with or without the
//                          tangent) and internal force of P2 tetrahedra in one pass over the
//                          points (CONSTITUTIVE.m:178-285)
//   k_response2d           the same for P2 triangles
//   k_element_blocks_fact  element stiffness blocks from the tangent through the moments of
//                          the rule (assemble_K_tangent_vals.c:77-171)
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <utility>
#include <vector>

#include "instr.cuh"
#include "mc_point.cuh"
#include "mesh.h"
#include "p2tet.cuh"
#include "sg_common.cuh"

namespace sg {

// ------------------------------------------------------------------ factored gradients

// the two vertices of local edge 4 + m
__host__ __device__ constexpr int p2_edge_a(int m) { return m == 1 ? 1 : m == 3 ? 1 : m == 4 ? 2 : 0; }
__host__ __device__ constexpr int p2_edge_b(int m) { return m == 0 ? 1 : (m == 1 || m == 2) ? 2 : 3; }

struct P2TetFit {
    double fit[P2T_MAXQ][3][10];   // G_k = sum_i fit[q][k - 1][i] grad(phi_i), least squares
};

// One thread per point: G_1..3 by the least-squares fit of the point's ten gradients, and
// the largest deviation of the gradients rebuilt from them against the given ones.
__global__ void __launch_bounds__(128) k_p2tet_factor(int64_t n_int, int nq, const double *__restrict__ dphi,
                                                      const __grid_constant__ P2TetRule rule,
                                                      const P2TetFit *__restrict__ fit, double *__restrict__ gxi,
                                                      int32_t *__restrict__ bad) {
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < n_int; g += (int64_t)gridDim.x * blockDim.x) {
        const int q = (int)(g % nq);
        const double l[4] = {rule.lam[q][0], rule.lam[q][1], rule.lam[q][2], rule.lam[q][3]};
        const double *d = dphi + g * 30;
        double big = 0.0, off = 0.0;
        for (int c = 0; c < 3; ++c) {
            double G[4];
            for (int k = 0; k < 3; ++k) {
                double s = 0.0;
                for (int i = 0; i < 10; ++i) s += fit->fit[q][k][i] * d[c * 10 + i];
                G[k + 1] = s;
                gxi[(g / nq * 9 + k * 3 + c) * nq + q] = s;
            }
            G[0] = -(G[1] + G[2] + G[3]);
            for (int i = 0; i < 10; ++i) {
                double r;
                if (i < 4) r = (4.0 * l[i] - 1.0) * G[i];
                else {
                    const int a = p2_edge_a(i - 4), b = p2_edge_b(i - 4);
                    r = 4.0 * (l[b] * G[a] + l[a] * G[b]);
                }
                big = fmax(big, fabs(d[c * 10 + i]));
                off = fmax(off, fabs(r - d[c * 10 + i]));
            }
        }
        // a few roundings of the point's largest gradient; NaN fails the test too
        if (!(off <= 64.0 * 2.220446049250313e-16 * big)) atomicOr(bad, 1);
    }
}

int p2tet_factor(sg_mesh *m, const double *D1, const double *D2, const double *D3) {
    if (m->dim != 3 || m->np != 10 || m->nq > P2T_MAXQ || m->n_e == 0) return SG_OK;
    const int nq = m->nq;
    // Barycentric coordinates of the rule from the first element: with the basis numbered as in
    // p2tet.cuh, G_a = grad(phi_a) + 1/2 sum of the gradients of a's three edges at any point, and
    // grad(phi_a) = (4 lambda_a - 1) G_a.
    P2TetRule rule = {};
    const double *D[3] = {D1, D2, D3};
    for (int q = 0; q < nq; ++q) {
        long double G[4][3], sum = 0.0L;
        for (int c = 0; c < 3; ++c) {
            const double *d = D[c] + (int64_t)q * 10;
            for (int a = 0; a < 4; ++a) G[a][c] = d[a];
            for (int e = 0; e < 6; ++e) {
                G[p2_edge_a(e)][c] += 0.5L * d[4 + e];
                G[p2_edge_b(e)][c] += 0.5L * d[4 + e];
            }
        }
        for (int a = 1; a < 4; ++a) {
            long double dot = 0.0L, sq = 0.0L;
            for (int c = 0; c < 3; ++c) {
                dot += (long double)D[c][(int64_t)q * 10 + a] * G[a][c];
                sq += G[a][c] * G[a][c];
            }
            if (!(sq > 0.0L)) return SG_OK;
            rule.lam[q][a] = (double)((dot / sq + 1.0L) / 4.0L);
            sum += rule.lam[q][a];
        }
        rule.lam[q][0] = (double)(1.0L - sum);
    }
    // grad(phi_i) = sum_k c_ik G_k over k = 1..3: the 10 x 3 coefficients of each point and
    // their pseudo-inverse
    std::vector<P2TetFit> fit(1);
    for (int q = 0; q < nq; ++q) {
        const double *l = rule.lam[q];
        long double c[10][4] = {}, N[3][3] = {};
        for (int i = 0; i < 4; ++i) c[i][i] = 4.0L * l[i] - 1.0L;
        for (int e = 0; e < 6; ++e) {
            c[4 + e][p2_edge_a(e)] = 4.0L * l[p2_edge_b(e)];
            c[4 + e][p2_edge_b(e)] = 4.0L * l[p2_edge_a(e)];
        }
        for (int i = 0; i < 10; ++i)
            for (int k = 1; k < 4; ++k) c[i][k] -= c[i][0];
        for (int r = 0; r < 3; ++r)
            for (int s = 0; s < 3; ++s)
                for (int i = 0; i < 10; ++i) N[r][s] += c[i][r + 1] * c[i][s + 1];
        const long double det = N[0][0] * (N[1][1] * N[2][2] - N[1][2] * N[2][1]) -
                                N[0][1] * (N[1][0] * N[2][2] - N[1][2] * N[2][0]) +
                                N[0][2] * (N[1][0] * N[2][1] - N[1][1] * N[2][0]);
        if (!(std::fabs(det) > 1e-12L)) return SG_OK;
        long double inv[3][3];
        for (int r = 0; r < 3; ++r)
            for (int s = 0; s < 3; ++s) {
                const int r1 = (s + 1) % 3, r2 = (s + 2) % 3, s1 = (r + 1) % 3, s2 = (r + 2) % 3;
                inv[r][s] = (N[r1][s1] * N[r2][s2] - N[r1][s2] * N[r2][s1]) / det;
            }
        for (int k = 0; k < 3; ++k)
            for (int i = 0; i < 10; ++i) {
                long double v = 0.0L;
                for (int s = 0; s < 3; ++s) v += inv[k][s] * c[i][s + 1];
                fit[0].fit[q][k][i] = (double)v;
            }
    }
    struct Temp {
        void *p = nullptr;
        ~Temp() { cudaFree(p); }
    } tfit, tbad;
    double *gxi = nullptr;
    SG_CUDA(device_alloc(reinterpret_cast<char **>(&tfit.p), sizeof(P2TetFit)));
    SG_CUDA(device_alloc(reinterpret_cast<char **>(&tbad.p), sizeof(int32_t)));
    SG_CUDA(device_alloc(&gxi, sizeof(double) * 9 * (size_t)m->n_int));
    m->d_gxi = gxi;   // freed with the mesh whatever happens below
    SG_CUDA(cudaMemcpy(tfit.p, fit.data(), sizeof(P2TetFit), cudaMemcpyHostToDevice));
    SG_CUDA(cudaMemset(tbad.p, 0, sizeof(int32_t)));
    k_p2tet_factor<<<grid_for(m->n_int, 128, 16), 128>>>(m->n_int, nq, m->d_dphi, rule,
                                                         static_cast<const P2TetFit *>(tfit.p), gxi,
                                                         static_cast<int32_t *>(tbad.p));
    SG_CUDA(cudaGetLastError());
    int32_t bad = 0;
    SG_CUDA(cudaMemcpy(&bad, tbad.p, sizeof(int32_t), cudaMemcpyDeviceToHost));
    if (bad) {
        cudaFree(m->d_gxi);
        m->d_gxi = nullptr;
        return SG_OK;
    }
    for (int q = 0; q < nq; ++q)
        for (int k = 0; k < 4; ++k) m->rule[q][k] = rule.lam[q][k];
    return SG_OK;
}

static P2TetRule rule_of(const sg_mesh *m) {
    P2TetRule r;
    for (int q = 0; q < P2T_MAXQ; ++q)
        for (int k = 0; k < 4; ++k) r.lam[q][k] = m->rule[q][k];
    return r;
}

// ------------------------------------------------------------------ strain -> stress -> force

struct ResponseArgs {
    const int32_t *elem;
    const double *dphi, *gxi, *w;
    int nq, el;                       // points per element, elements per CTA pass
    int64_t n_e, n_int;
    const double *U;
    const double *c0, *phi, *psi;     // reduced in the kernel when davis != 0
    double lambda;
    char davis;
    double *c_bar, *sin_phi;          // read when davis == 0, written otherwise
    const double *shear, *lame;
    double *E, *S, *DS;               // E, S may be null
    uint8_t *branch;                  // may be null
    double *F;                        // zeroed by the caller
};

__device__ __forceinline__ void response_strength(const ResponseArgs &A, int64_t g, double &cb, double &sp) {
    if (A.davis) {
        davis_reduce(A.c0[g], A.phi[g], A.psi[g], A.lambda, A.davis, cb, sp);
        A.c_bar[g] = cb;
        A.sin_phi[g] = sp;
    } else {
        cb = A.c_bar[g];
        sp = A.sin_phi[g];
    }
}

// A CTA takes el elements at a time (8 at the 11-point rule: 88 of 96 threads own a point).
// Every load of a pass is issued at its top, the strength reduction runs while the nodal
// displacements arrive and are staged in shared memory; phase 1, a thread per point: the
// displacement gradient in barycentric directions from the rule's table and the staged nodes,
// nine G values for the physical gradient, and the return mapping in registers; phase 2: the
// moments of the tractions w S G_k over the element's points, then a thread per (element,
// node) adds the node's force with atomics.  With FACT = false (a mesh whose gradients do not
// factor) the gradients are read from d_dphi in both phases.
// TANGENT stores E, S and DS: a warp stages its 32 points in shared memory (odd pitch) and writes
// contiguous runs, as k_mc3d does.
//
// What bounds it: latency, with the L1 data pipe 68 % busy behind it (FP64 pipe 38 %, DRAM 24 %; with
// the tangent 62, 23 and 45 %).  The three phases of a pass depend on one another and the return
// mapping is a long FP64 chain, so the time goes with the passes in flight: 96-thread CTAs, eight
// per SM (24 warps) at 80 registers without the tangent (a few spills cost less than the resident
// CTAs they buy: 141 us against 163 with six CTAs on the 40 m slope), four at 168 registers with
// it (five with spills: 1.43 against 1.25 ms on the layered slope).  Measured on B200, against
// the reduction, strain, return-mapping and force kernels in turn (stress only: the reduction and
// the former fused residual with 240 gradient bytes per point): 40 m slope, 1.72M points, stress
// only 285 -> 130 us; layered slope, 8.0M points, with the tangent 2.25 -> 1.09 ms (3.3 TB/s of
// the 449 bytes a point cannot do without); 36,400 points in 2D 46 -> 16 us a call.
constexpr int RSP_THREADS = 96, RSP_EL = 8, RSP_WARPS = RSP_THREADS / 32;
constexpr int RSP_TP = 13;                       // doubles per point of the traction stage
constexpr int RSP_DSP = 37, RSP_SP = 7;          // staging pitches of DS and of E, S
constexpr size_t RSP_SMEM = sizeof(double) * (RSP_EL * 30 + RSP_THREADS * RSP_TP + RSP_EL * 48);
constexpr size_t RSP_SMEM_DS = RSP_SMEM + sizeof(double) * RSP_WARPS * 32 * (RSP_DSP + RSP_SP);
static_assert(RSP_SMEM_DS <= 48 * 1024, "within the default limit of dynamic shared memory");

// NQ > 0: the rule's size at compile time (its table then sits in the instructions' constant operands).
template <bool TANGENT, bool FACT, int NQ>
__global__ void __launch_bounds__(RSP_THREADS, TANGENT ? 4 : 8)
    k_response3d(const __grid_constant__ ResponseArgs A, const __grid_constant__ P2TetRule rule) {
    extern __shared__ double rsp_sm[];
    double *su = rsp_sm, *sT = su + RSP_EL * 30, *sm = sT + RSP_THREADS * RSP_TP;
    double *sds = sm + RSP_EL * 48 + (threadIdx.x >> 5) * 32 * (RSP_DSP + RSP_SP), *ss = sds + 32 * RSP_DSP;
    const int t = threadIdx.x, lane = t & 31, nq = NQ > 0 ? NQ : A.nq;
    const int le = t / nq, q = t - le * nq;
    double l4[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) l4[k] = FACT && q < P2T_MAXQ ? 4.0 * rule.lam[q][k] : 0.0;
    int32_t v_next = 0;   // this thread's node of the coming pass, and its element's first
    {
        const int64_t e0 = (int64_t)blockIdx.x * A.el;
        if (e0 < A.n_e && t < (A.n_e - e0 < A.el ? (int)(A.n_e - e0) : A.el) * 10) {
            v_next = A.elem[e0 * 10 + t];
        }
    }
    for (int64_t e0 = (int64_t)blockIdx.x * A.el; e0 < A.n_e; e0 += (int64_t)gridDim.x * A.el) {
        const int ne = (int)(A.n_e - e0 < A.el ? A.n_e - e0 : A.el);
        const int np = ne * nq;                 // points of this pass: g = e0 * nq + t
        const int64_t g = e0 * nq + t;
        const bool live = t < np, stages = t < ne * 10;
        // every load of the pass is issued before the first is needed, and the strength reduction
        // runs while the displacements arrive
        double un[3] = {0.0, 0.0, 0.0}, G[9], wq = 0.0, cb = 0.0, sp = 0.0, shear = 0.0, lame = 0.0;
        if (stages) {
            const int64_t v = v_next;
#pragma unroll
            for (int c = 0; c < 3; ++c) un[c] = A.U[3 * v + c];
        }
        if (live) {
            wq = A.w[g];
            shear = A.shear[g];
            lame = A.lame[g];
            if constexpr (FACT)
#pragma unroll
                for (int k = 0; k < 9; ++k) G[k] = A.gxi[(e0 + le) * 9 * nq + k * nq + q];
            response_strength(A, g, cb, sp);
        }
        if (stages)
#pragma unroll
            for (int c = 0; c < 3; ++c) su[t / 10 * 30 + c * 10 + t % 10] = un[c];
        const int32_t v_node = v_next;
        {   // the next pass's nodes
            const int64_t en = e0 + (int64_t)gridDim.x * A.el;
            if (en < A.n_e && t < (A.n_e - en < A.el ? (int)(A.n_e - en) : A.el) * 10) {
                v_next = A.elem[en * 10 + t];
            }
        }
        __syncthreads();
        double E[6], st[6];
        if (live) {
            const double *u = su + le * 30;
            if constexpr (FACT) {
                // gradient in barycentric directions, direction 0 eliminated
                double h[3][3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    double x[10];
#pragma unroll
                    for (int i = 0; i < 5; ++i) {
                        const double2 w2 = *reinterpret_cast<const double2 *>(u + c * 10 + 2 * i);
                        x[2 * i] = w2.x;
                        x[2 * i + 1] = w2.y;
                    }
#pragma unroll
                    for (int i = 1; i < 10; ++i) x[i] -= x[0];   // the element's translation carries no strain
                    const double h0 = l4[1] * x[4] + l4[2] * x[6] + l4[3] * x[9];
                    h[0][c] = (l4[1] - 1.0) * x[1] + l4[0] * x[4] + l4[2] * x[5] + l4[3] * x[7] - h0;
                    h[1][c] = (l4[2] - 1.0) * x[2] + l4[1] * x[5] + l4[0] * x[6] + l4[3] * x[8] - h0;
                    h[2][c] = (l4[3] - 1.0) * x[3] + l4[1] * x[7] + l4[2] * x[8] + l4[0] * x[9] - h0;
                }
#pragma unroll
                for (int a = 0; a < 6; ++a) E[a] = 0.0;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const double gx = G[k * 3], gy = G[k * 3 + 1], gz = G[k * 3 + 2];
                    E[0] += gx * h[k][0];
                    E[1] += gy * h[k][1];
                    E[2] += gz * h[k][2];
                    E[3] += gy * h[k][0] + gx * h[k][1];
                    E[4] += gz * h[k][1] + gy * h[k][2];
                    E[5] += gz * h[k][0] + gx * h[k][2];
                }
            } else {
                const double *d = A.dphi + g * 30;
#pragma unroll
                for (int a = 0; a < 6; ++a) E[a] = 0.0;
                for (int i = 0; i < 10; ++i) {
                    const double d1 = d[i], d2 = d[10 + i], d3 = d[20 + i];
                    const double ux = u[i], uy = u[10 + i], uz = u[20 + i];
                    E[0] += d1 * ux;
                    E[1] += d2 * uy;
                    E[2] += d3 * uz;
                    E[3] += d2 * ux + d1 * uy;
                    E[4] += d3 * uy + d2 * uz;
                    E[5] += d3 * ux + d1 * uz;
                }
            }
            const int b = mc3d_point<TANGENT>(E, cb, sp, shear, lame, st, sds + lane * RSP_DSP);
            if (A.branch) A.branch[g] = (uint8_t)b;
            double *T = sT + t * RSP_TP;
            if constexpr (FACT) {
                double t0[3] = {0.0, 0.0, 0.0};
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const double gx = wq * G[k * 3], gy = wq * G[k * 3 + 1], gz = wq * G[k * 3 + 2];
                    const double tx = gx * st[0] + gy * st[3] + gz * st[5];
                    const double ty = gy * st[1] + gx * st[3] + gz * st[4];
                    const double tz = gz * st[2] + gy * st[4] + gx * st[5];
                    T[(k + 1) * 3] = tx;
                    T[(k + 1) * 3 + 1] = ty;
                    T[(k + 1) * 3 + 2] = tz;
                    t0[0] -= tx;
                    t0[1] -= ty;
                    t0[2] -= tz;
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) T[c] = t0[c];
            } else {
#pragma unroll
                for (int c = 0; c < 6; ++c) T[c] = wq * st[c];
            }
        }
        if constexpr (TANGENT) {
            // the warp's points are contiguous in global memory
            const int w0 = t - lane;
            const int cnt = np - w0 < 32 ? np - w0 : 32;
            const int64_t base = e0 * nq + w0;
            __syncwarp();
            for (int k = lane; k < cnt * 36; k += 32) {
                const int p = k / 36;
                A.DS[36 * base + k] = sds[p * RSP_DSP + k - p * 36];
            }
#pragma unroll
            for (int what = 0; what < 2; ++what) {
                double *out = what ? A.S : A.E;
                if (!out) continue;
                if (live)
#pragma unroll
                    for (int c = 0; c < 6; ++c) ss[lane * RSP_SP + c] = what ? st[c] : E[c];
                __syncwarp();
                for (int k = lane; k < cnt * 6; k += 32) {
                    const int p = k / 6;
                    out[6 * base + k] = ss[p * RSP_SP + k - p * 6];
                }
                __syncwarp();
            }
        }
        __syncthreads();
        if constexpr (FACT) {
            // a thread per (element, direction a, component): M_b = sum_q 4 lambda_b t_a
            for (int k = t; k < ne * 12; k += RSP_THREADS) {
                const int fe = k / 12, ac = k - fe * 12;
                const double *T = sT + fe * nq * RSP_TP + ac;
                double m0 = 0.0, m1 = 0.0, m2 = 0.0, m3 = 0.0;
#pragma unroll
                for (int p = 0; p < (NQ > 0 ? NQ : nq); ++p) {
                    const double v = 4.0 * T[p * RSP_TP];
                    m0 += rule.lam[p][0] * v;
                    m1 += rule.lam[p][1] * v;
                    m2 += rule.lam[p][2] * v;
                    m3 += rule.lam[p][3] * v;
                }
                double *o = sm + fe * 48 + ac;
                o[0] = m0;
                o[12] = m1;
                o[24] = m2;
                o[36] = m3;
            }
            __syncthreads();
            // vertex a: M_a - sum_b M_b / 4 (the lambdas add to one), edge (a, b): M_b(t_a) + M_a(t_b)
            if (stages) {
                const int fe = t / 10, fi = t - fe * 10;
                const int a = fi < 4 ? fi : p2_edge_a(fi - 4), b = fi < 4 ? fi : p2_edge_b(fi - 4);
                const double *o = sm + fe * 48;
#pragma unroll
                for (int c = 0; c < 3; ++c, ++o) {
                    const double *oa = o + a * 3;
                    const double f = fi < 4 ? oa[a * 12] - 0.25 * (oa[0] + oa[12] + oa[24] + oa[36])
                                            : o[b * 12 + a * 3] + o[a * 12 + b * 3];
                    atomicAdd(&A.F[3 * (int64_t)v_node + c], f);
                }
            }
        } else {
            if (stages) {
                const int fe = t / 10, fi = t - fe * 10;
                double f0 = 0.0, f1 = 0.0, f2 = 0.0;
                for (int p = 0; p < nq; ++p) {
                    const double *T = sT + (fe * nq + p) * RSP_TP;
                    const double *d = A.dphi + ((e0 + fe) * nq + p) * 30;
                    const double d1 = d[fi], d2 = d[10 + fi], d3 = d[20 + fi];
                    f0 += d1 * T[0] + d2 * T[3] + d3 * T[5];
                    f1 += d2 * T[1] + d1 * T[3] + d3 * T[4];
                    f2 += d3 * T[2] + d2 * T[4] + d1 * T[5];
                }
                atomicAdd(&A.F[3 * (int64_t)v_node], f0);
                atomicAdd(&A.F[3 * (int64_t)v_node + 1], f1);
                atomicAdd(&A.F[3 * (int64_t)v_node + 2], f2);
            }
        }
    }
}
static_assert(RSP_EL * 10 <= RSP_THREADS, "a thread per node of a pass");

// P2 triangles: a CTA takes el elements at a time (18 at the 7-point rule: 126 of 128
// threads own a point), the same two phases with the gradients read from d_dphi.  The 2D
// meshes are small (36,400 points at h = 0.5): what counts is that one launch replaces
// reduction, strain, return mapping and force.
constexpr int RSP2_THREADS = 128;
template <bool TANGENT>
__global__ void __launch_bounds__(RSP2_THREADS) k_response2d(const __grid_constant__ ResponseArgs A) {
    __shared__ double sT[RSP2_THREADS * 3];
    __shared__ double sds[TANGENT ? RSP2_THREADS * 9 : 1];
    const int t = threadIdx.x, nq = A.nq;
    const int le = t / nq;
    for (int64_t e0 = (int64_t)blockIdx.x * A.el; e0 < A.n_e; e0 += (int64_t)gridDim.x * A.el) {
        const int ne = (int)(A.n_e - e0 < A.el ? A.n_e - e0 : A.el);
        const int np = ne * nq;
        const int64_t g = e0 * nq + t;
        if (t < np) {
            const double *d = A.dphi + g * 12;
            const int32_t *el = A.elem + (e0 + le) * 6;
            double E[3] = {0.0, 0.0, 0.0}, st[4];
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                const int64_t v = el[i];
                const double ux = A.U[2 * v], uy = A.U[2 * v + 1], d1 = d[i], d2 = d[6 + i];
                E[0] += d1 * ux;
                E[1] += d2 * uy;
                E[2] += d2 * ux + d1 * uy;
            }
            double cb, sp;
            response_strength(A, g, cb, sp);
            const int b = mc2d_point<TANGENT>(E, cb, sp, A.shear[g], A.lame[g], st, sds + (TANGENT ? t * 9 : 0));
            if (A.branch) A.branch[g] = (uint8_t)b;
            const double wq = A.w[g];
#pragma unroll
            for (int c = 0; c < 3; ++c) sT[t * 3 + c] = wq * st[c];
            if (A.E)
#pragma unroll
                for (int c = 0; c < 3; ++c) A.E[3 * g + c] = E[c];
            if (A.S)
#pragma unroll
                for (int c = 0; c < 4; ++c) A.S[4 * g + c] = st[c];
        }
        __syncthreads();
        if (TANGENT)
            for (int k = t; k < np * 9; k += RSP2_THREADS) A.DS[9 * e0 * nq + k] = sds[k];
        for (int k = t; k < ne * 6; k += RSP2_THREADS) {
            const int fe = k / 6, fi = k - fe * 6;
            double f0 = 0.0, f1 = 0.0;
            for (int p = 0; p < nq; ++p) {
                const double *d = A.dphi + ((e0 + fe) * nq + p) * 12, *T = sT + (fe * nq + p) * 3;
                const double d1 = d[fi], d2 = d[6 + fi];
                f0 += d1 * T[0] + d2 * T[2];
                f1 += d2 * T[1] + d1 * T[2];
            }
            const int64_t v = A.elem[e0 * 6 + k];
            atomicAdd(&A.F[2 * v], f0);
            atomicAdd(&A.F[2 * v + 1], f1);
        }
        __syncthreads();
    }
}

static int launch_response(const sg_mesh *m, ResponseArgs A, int kind, cudaStream_t st) {
    A.elem = m->d_elem;
    A.dphi = m->d_dphi;
    A.gxi = m->d_gxi;
    A.w = m->d_w;
    A.nq = m->nq;
    A.n_e = m->n_e;
    A.n_int = m->n_int;
    SG_CUDA(cudaMemsetAsync(A.F, 0, sizeof(double) * m->n_n * m->dim, st));
    if (m->n_e == 0) return SG_OK;
    const bool tangent = A.DS != nullptr;
    const InstrToken tk = instr_begin(kind, st);
    count_launch();
    if (m->dim == 3) {
        A.el = std::min(RSP_EL, RSP_THREADS / m->nq);
        const int64_t ctas = (m->n_e + A.el - 1) / A.el;
        const unsigned grid = (unsigned)std::min<int64_t>(ctas, (int64_t)sm_count() * 24);
        const P2TetRule rule = rule_of(m);
        // the factored kernel at the 11-point rule is compiled for it; other rules and meshes
        // whose gradients do not factor share the general ones
        const bool fact = m->d_gxi != nullptr, r11 = fact && m->nq == P2T_REF_RULE;
        const size_t smem = tangent ? RSP_SMEM_DS : RSP_SMEM;
        if (tangent) {
            if (r11) k_response3d<true, true, P2T_REF_RULE><<<grid, RSP_THREADS, smem, st>>>(A, rule);
            else if (fact) k_response3d<true, true, 0><<<grid, RSP_THREADS, smem, st>>>(A, rule);
            else k_response3d<true, false, 0><<<grid, RSP_THREADS, smem, st>>>(A, rule);
        } else {
            if (r11) k_response3d<false, true, P2T_REF_RULE><<<grid, RSP_THREADS, smem, st>>>(A, rule);
            else if (fact) k_response3d<false, true, 0><<<grid, RSP_THREADS, smem, st>>>(A, rule);
            else k_response3d<false, false, 0><<<grid, RSP_THREADS, smem, st>>>(A, rule);
        }
    } else {
        A.el = RSP2_THREADS / m->nq;
        const int64_t ctas = (m->n_e + A.el - 1) / A.el;
        const unsigned grid = (unsigned)std::min<int64_t>(ctas, (int64_t)sm_count() * 16);
        if (tangent) k_response2d<true><<<grid, RSP2_THREADS, 0, st>>>(A);
        else k_response2d<false><<<grid, RSP2_THREADS, 0, st>>>(A);
    }
    instr_end(tk, st);
    SG_CUDA(cudaGetLastError());
    return SG_OK;
}

static bool response_covers(const sg_mesh *m) {
    return ((m->dim == 3 && m->np == 10) || (m->dim == 2 && m->np == 6)) && m->nq >= 1 && m->nq <= P2T_MAXQ;
}

// ------------------------------------------------------------------ element stiffness blocks

// The element's node blocks K_ij = sum_q w_q B_i' sym(D_q) B_j through the moments of the rule.
// With grad(phi_i) = sum_k c_ik(lambda) G_k and c_ik linear in the barycentric coordinates,
//     K_ij[a][b] = sum_{k,l} sum_q c_ik c_jl Y_q[k a][l b],   Y_q = w_q Z_q' sym(D_q) Z_q,
// Z_q the strain of G_1, G_2, G_3 in the three components (6 x 9): 45 values per point instead
// of the products with 30 columns.  As c_ik c_jl is quadratic, the ten moments
// sum_q lambda_s lambda_t Y_q carry everything, and each block is a short combination of them with
// integer coefficients.  14k FP64 operations per element against 36k of the direct sum.
//
//   A  a thread per point: D from shared memory, Y_q (486 operations), 45 values to shared memory
//   B  a thread per (element, value): the value at the 11 points -> its ten moments, in place
//   C  a thread per (element, component pair a b): 10 x 9 moments (the directions 0 follow from
//      G_0 = -(G_1 + G_2 + G_3)) -> the 55 entries [a][b] of the element's upper blocks
// Eight elements per pass of a 96-thread CTA (88 points); D, G and w come by cp.async, the next
// pass's while B and C run; three CTAs per SM (65 KB each, registers to spare for C's 55 sums).
//
// What bounds it: the latency of the FP64 chains with nine warps on an SM (0.38 instructions a cycle and
// scheduler, FP64 pipe 37 % busy, L1 data pipe 53 %); DRAM carries DS, G and w in and 3,960 bytes an
// element out.  Measured on
// B200 against the direct sum (k_element_blocks_p2tet_bulk): 446k points 243 -> 99 us, layered
// slope (8.0M points) 4.06 -> 1.62 ms (3.6 TB/s).
constexpr int EB_EL = 8, EB_THREADS = 96, EB_NQ = P2T_REF_RULE, EB_DP = 38, EB_Y = 45;
constexpr size_t EB_SMEM = sizeof(double) * EB_EL * EB_NQ * (EB_DP + EB_Y + 10);

struct P2TetMoments {
    double c[EB_NQ][10];   // lambda_s lambda_t, s <= t, of every point
};

constexpr int eb_s(int m) { return m < 4 ? 0 : m < 7 ? 1 : m < 9 ? 2 : 3; }
constexpr int eb_t(int m) { return m < 4 ? m : m < 7 ? m - 3 : m < 9 ? m - 5 : 3; }
// upper pair index -> (i, j), i <= j, ten nodes
constexpr int eb_i(int p) {
    int i = 0;
    while (p >= 10 - i) p -= 10 - i++;
    return i;
}
constexpr int eb_j(int p) {
    int i = 0;
    while (p >= 10 - i) p -= 10 - i++;
    return i + p;
}
// coefficient of lambda_s in c_ik
constexpr int eb_coef(int i, int k, int s) {
    if (i < 4) return k == i ? (s == i ? 3 : -1) : 0;
    const int a = p2_edge_a(i - 4), b = p2_edge_b(i - 4);
    return k == a ? (s == b ? 4 : 0) : k == b ? (s == a ? 4 : 0) : 0;
}
constexpr int eb_weight(int m, int i, int j, int k, int l) {
    const int s = eb_s(m), t = eb_t(m);
    return eb_coef(i, k, s) * eb_coef(j, l, t) + (s != t ? eb_coef(i, k, t) * eb_coef(j, l, s) : 0);
}
template <int M, int P, int KL>
__device__ __forceinline__ void eb_term(double &acc, const double (&X)[4][4]) {
    constexpr int w = eb_weight(M, eb_i(P), eb_j(P), KL / 4, KL % 4);
    if constexpr (w != 0) acc += (double)w * X[KL / 4][KL % 4];
}
template <int M, int P, int... KL>
__device__ __forceinline__ void eb_entry(double &acc, const double (&X)[4][4], std::integer_sequence<int, KL...>) {
    (eb_term<M, P, KL>(acc, X), ...);
}
template <int M, int... P>
__device__ __forceinline__ void eb_moment(double (&acc)[55], const double (&X)[4][4], std::integer_sequence<int, P...>) {
    (eb_entry<M, P>(acc[P], X, std::make_integer_sequence<int, 16>()), ...);
}
template <int M>
__device__ __forceinline__ void eb_moments(double (&acc)[55], const double *Y, const int (&off)[3][3]) {
    if constexpr (M < 10) {
        double X[4][4];
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int l = 0; l < 3; ++l) X[k + 1][l + 1] = Y[M * EB_Y + off[k][l]];
#pragma unroll
        for (int l = 1; l < 4; ++l) {
            X[0][l] = -(X[1][l] + X[2][l] + X[3][l]);
            X[l][0] = -(X[l][1] + X[l][2] + X[l][3]);
        }
        X[0][0] = -(X[0][1] + X[0][2] + X[0][3]);
        eb_moment<M>(acc, X, std::make_integer_sequence<int, 55>());
        eb_moments<M + 1>(acc, Y, off);
    }
}

// entry [a][b] of every block; diagonal blocks are made exactly symmetric
template <int P>
__device__ __forceinline__ void eb_store_one(double v, double *out, int a, int b) {
    if constexpr (eb_i(P) != eb_j(P)) out[P * 9] = v;
    else if (a <= b) {
        out[P * 9] = v;
        if (a < b) out[P * 9 + 2 * (b - a)] = v;    // entry [b][a] lies 2 (b - a) behind [a][b]
    }
}
template <int... P>
__device__ __forceinline__ void eb_store(const double (&acc)[55], double *out, int a, int b,
                                         std::integer_sequence<int, P...>) {
    (eb_store_one<P>(acc[P], out, a, b), ...);
}

// position of Y[(k, a)][(l, b)], k, l = 0..2 for G_1..G_3, (k, a) <= (l, b): blocks (0,0) (0,1)
// (1,1) (0,2) (1,2) (2,2), the diagonal ones as their upper triangles
__device__ __forceinline__ int eb_pos(int k, int a, int l, int b) {
    if (k > l || (k == l && a > b)) {
        int s = k;
        k = l;
        l = s;
        s = a;
        a = b;
        b = s;
    }
    const int base = l == 0 ? 0 : l == 1 ? (k == 0 ? 6 : 15) : (k == 0 ? 21 : k == 1 ? 30 : 39);
    return base + (k == l ? a * 3 - a * (a - 1) / 2 + (b - a) : a * 3 + b);
}

__device__ __forceinline__ void eb_copy16(double *dst, const double *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void eb_copy8(double *dst, const double *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

template <bool ALIGNED>
__global__ void __launch_bounds__(EB_THREADS, 3)
    k_element_blocks_fact(int64_t n_e, const double *__restrict__ gxi, const double *__restrict__ w,
                          const double *__restrict__ DS, const __grid_constant__ P2TetMoments mom,
                          double *__restrict__ Ke) {
    extern __shared__ __align__(16) double eb_sm[];
    double *sD = eb_sm, *sY = sD + EB_EL * EB_NQ * EB_DP, *sG = sY + EB_EL * EB_NQ * EB_Y, *sW = sG + EB_EL * EB_NQ * 9;
    const int t = threadIdx.x;
    auto stage = [&](int64_t e0) {
        const int ne = (int)(n_e - e0 < EB_EL ? n_e - e0 : EB_EL);
        const double *D = DS + e0 * EB_NQ * 36;
        if (ALIGNED) {
            for (int k = t; k < ne * EB_NQ * 18; k += EB_THREADS) {
                const int p = k / 18, c = k - p * 18;
                eb_copy16(sD + p * EB_DP + 2 * c, D + 2 * k);
            }
        } else {
            for (int k = t; k < ne * EB_NQ * 36; k += EB_THREADS) {
                const int p = k / 36, c = k - p * 36;
                eb_copy8(sD + p * EB_DP + c, D + k);
            }
        }
        for (int k = t; k < ne * EB_NQ * 9; k += EB_THREADS) eb_copy8(sG + k, gxi + e0 * EB_NQ * 9 + k);
        for (int k = t; k < ne * EB_NQ; k += EB_THREADS) eb_copy8(sW + k, w + e0 * EB_NQ + k);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // phase C: this thread's component pair and where its moments lie
    const int ce = t / 9, ab = t - ce * 9, ca = ab / 3, cb = ab - ca * 3;
    int off[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = 0; l < 3; ++l) off[k][l] = eb_pos(k, ca, l, cb);
    int64_t e0 = (int64_t)blockIdx.x * EB_EL;
    if (e0 < n_e) stage(e0);
    for (; e0 < n_e; e0 += (int64_t)gridDim.x * EB_EL) {
        const int ne = (int)(n_e - e0 < EB_EL ? n_e - e0 : EB_EL);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (t < ne * EB_NQ) {
            const double *D = sD + t * EB_DP;
            double d[6][6];
            {
                double raw[36];
#pragma unroll
                for (int k = 0; k < 18; ++k) {
                    const double2 v = *reinterpret_cast<const double2 *>(D + 2 * k);
                    raw[2 * k] = v.x;
                    raw[2 * k + 1] = v.y;
                }
                const double wq = sW[t], hw = 0.5 * wq;
#pragma unroll
                for (int a = 0; a < 6; ++a) {
                    d[a][a] = wq * raw[7 * a];
#pragma unroll
                    for (int b = a + 1; b < 6; ++b) d[a][b] = d[b][a] = hw * (raw[a + 6 * b] + raw[b + 6 * a]);
                }
            }
            const int le = t / EB_NQ, q = t - le * EB_NQ;
            double G[3][3];
#pragma unroll
            for (int k = 0; k < 9; ++k) G[k / 3][k % 3] = sG[(le * 9 + k) * EB_NQ + q];
            double *Y = sY + t * EB_Y;
            // rows of the strain of (direction, component c): v[m] at row rw[c][m]
            constexpr int rw[3][3] = {{0, 3, 5}, {1, 3, 4}, {2, 4, 5}};
            constexpr int dir[3][3] = {{0, 1, 2}, {1, 0, 2}, {2, 1, 0}};
            constexpr int base[3][3] = {{0, 6, 21}, {0, 15, 30}, {0, 0, 39}};
#pragma unroll
            for (int l = 0; l < 3; ++l) {
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    double db[6];
#pragma unroll
                    for (int a = 0; a < 6; ++a)
                        db[a] = d[a][rw[b][0]] * G[l][dir[b][0]] + d[a][rw[b][1]] * G[l][dir[b][1]] +
                                d[a][rw[b][2]] * G[l][dir[b][2]];
#pragma unroll
                    for (int k = 0; k <= l; ++k)
#pragma unroll
                        for (int a = 0; a < 3; ++a) {
                            if (k == l && a > b) continue;
                            const int pos = base[k][l] + (k == l ? a * 3 - a * (a - 1) / 2 + (b - a) : a * 3 + b);
                            Y[pos] = db[rw[a][0]] * G[k][dir[a][0]] + db[rw[a][1]] * G[k][dir[a][1]] +
                                     db[rw[a][2]] * G[k][dir[a][2]];
                        }
                }
            }
        }
        __syncthreads();
        if (e0 + (int64_t)gridDim.x * EB_EL < n_e) stage(e0 + (int64_t)gridDim.x * EB_EL);
        for (int k = t; k < ne * EB_Y; k += EB_THREADS) {
            const int e = k / EB_Y, y = k - e * EB_Y;
            double *Y = sY + e * EB_NQ * EB_Y + y;
            double m[10];
#pragma unroll
            for (int i = 0; i < 10; ++i) m[i] = 0.0;
#pragma unroll
            for (int q = 0; q < EB_NQ; ++q) {
                const double v = Y[q * EB_Y];
#pragma unroll
                for (int i = 0; i < 10; ++i) m[i] += mom.c[q][i] * v;
            }
#pragma unroll
            for (int i = 0; i < 10; ++i) Y[i * EB_Y] = m[i];
        }
        __syncthreads();
        if (ce < ne) {
            double acc[55];
#pragma unroll
            for (int p = 0; p < 55; ++p) acc[p] = 0.0;
            eb_moments<0>(acc, sY + ce * EB_NQ * EB_Y, off);
            eb_store(acc, Ke + (e0 + ce) * 495 + ab, ca, cb, std::make_integer_sequence<int, 55>());
        }
    }
}

int p2tet_element_blocks(const sg_mesh *m, const double *DS, double *Ke, cudaStream_t st) {
    P2TetMoments mom;
    for (int q = 0; q < EB_NQ; ++q)
        for (int i = 0; i < 10; ++i) mom.c[q][i] = m->rule[q][eb_s(i)] * m->rule[q][eb_t(i)];
    const int64_t passes = (m->n_e + EB_EL - 1) / EB_EL;
    const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(passes, (int64_t)sm_count() * 3));
    count_launch();
    const auto kernel = (reinterpret_cast<uintptr_t>(DS) & 15) == 0 ? k_element_blocks_fact<true>
                                                                     : k_element_blocks_fact<false>;
    SG_CUDA(allow_dynamic_smem(kernel, EB_SMEM));
    kernel<<<grid, EB_THREADS, EB_SMEM, st>>>(m->n_e, m->d_gxi, m->d_w, DS, mom, Ke);
    SG_CUDA(cudaGetLastError());
    return SG_OK;
}

}  // namespace sg

using namespace sg;

extern "C" int sg_residual_dev(const sg_mesh *m, const double *U, const double *c_bar, const double *sin_phi,
                               const double *shear, const double *lame, uint8_t *branch, double *F, void *stream) {
    SG_CHECK_ARG(m && U && c_bar && sin_phi && shear && lame && F, "null argument");
    SG_CHECK_ARG(m->dim == 3 && m->np == 10, "the fused residual is for P2 tetrahedra");
    SG_CHECK_ARG(response_covers(m), "too many integration points per element");
    ResponseArgs A = {};
    A.U = U;
    A.c_bar = const_cast<double *>(c_bar);      // read only: no reduction asked for
    A.sin_phi = const_cast<double *>(sin_phi);
    A.shear = shear;
    A.lame = lame;
    A.branch = branch;
    A.F = F;
    return launch_response(m, A, IK_RESIDUAL, as_stream(stream));
}

extern "C" int sg_element_response_dev(const sg_mesh *m, const double *U, const double *c0, const double *phi,
                                       const double *psi, double lambda, char davis_type, double *c_bar,
                                       double *sin_phi, const double *shear, const double *lame, double *E, double *S,
                                       double *DS, uint8_t *branch, double *F, void *stream) {
    SG_CHECK_ARG(m && U && c_bar && sin_phi && shear && lame && F, "null argument");
    SG_CHECK_ARG(response_covers(m), "the fused element response is for P2 triangles and tetrahedra");
    if (c0) {
        SG_CHECK_ARG(phi && psi, "null argument");
        SG_CHECK_ARG(davis_type == 'A' || davis_type == 'B' || davis_type == 'C',
                     "Davis type must be 'A', 'B' or 'C'");
        SG_CHECK_ARG(lambda > 0.0, "lambda must be positive");
    }
    SG_CHECK_ARG(m->dim == 2 || DS || (!E && !S), "on tetrahedra E and S are stored with the tangent only");
    ResponseArgs A = {};
    A.U = U;
    A.c0 = c0;
    A.phi = phi;
    A.psi = psi;
    A.lambda = lambda;
    A.davis = c0 ? davis_type : (char)0;
    A.c_bar = c_bar;
    A.sin_phi = sin_phi;
    A.shear = shear;
    A.lame = lame;
    A.E = E;
    A.S = S;
    A.DS = DS;
    A.branch = branch;
    A.F = F;
    return launch_response(m, A, DS ? IK_CONST_SDS : IK_RESIDUAL, as_stream(stream));
}
