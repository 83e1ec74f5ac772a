// Direct (displacement / traction) formulation on the device: the
// double-layer operator K_l with its P1 basis, its same-triangle parts and the
// diagonal blocks of V_l on the Duffy-type DIAG rule, the direct
// post-processing operators, and the direct time marching.
//
// Reference (paths relative to the reference project root; "DIR/" =
// functions/BEMenerg_dir/, "PP/" = functions/BEMenerg_dirPP/):
//   P1 basis         DIR/BEMenerg_dir_calcCostantData.m:17-21
//   K_l              DIR/CUDAkernels/kernelK.cu:14-460, launched by
//                    DIR/BEMenerg_dir_timeMarchingN.m:172-266
//   singular K_l     DIR/BEMenerg_dir_calcSubBlockSingK.m:1-41, DIR/BEMenerg_dir_calcKIntgSing.m
//   diagonal V_l     DIR/BEMenerg_dir_calcSubBlockDiagV.m:1-118
//   DIAG rule        functions/utility/quadRules/doppioGauss1D.m:1-43
//   post-processing  PP/CUDAkernels/kernelG.cu, PP/CUDAkernels/kernelP.cu,
//                    PP/BEMenerg_ppN_calc.m:115-124, PP/BEMenerg_ppD_calc.m:91-99
//   time marching    DIR/BEMenerg_dir_timeMarchingN.m:268-299 (least squares),
//                    DIR/BEMenerg_dir_timeMarchingD.m:272-296, DIR/BEMenerg_dir_calcBetaVgpu.m,
//                    DIR/BEMenerg_dir_calcBetaKgpu.m
//
// B200 design (not the reference's): a warp per (row triangle, vertex) pair of K
// and per (evaluation, vertex) of the traction part sorts its node pairs by
// the level of a front's arrival and evaluates each once per front; it visits only
// the triangles that contain the vertex (an adjacency list; the reference scans
// all N triangles per block).  Post-processing is contracted with the data
// in the kernel (no nHat x N matrices), with the reference's matrices available
// for verification.  The DN system is factorised once (QR), the reference
// re-solves densely every step.
#include "ebem_internal.h"

#include <cublas_v2.h>
#include <cusolverDn.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "front_bins.cuh"
#include "sa_math.cuh"

namespace ebem {

// ---------------------------------------------------------------------------
// DIAG rule (doppioGauss1D): n = n1^2 nodes on the triangle (A, B, C) with the
// singular vertex C: node (i, j) = ((1-x_j)(1-x_i), x_j (1-x_i), x_i) with
// weight 2 w_i w_j (1 - x_i), x, w the n1-point Gauss-Legendre rule on (0,1)
// (Newton's iteration on the Legendre polynomial).
int diag_rule(int n, std::vector<double>& nodes, std::vector<double>& w) {
    int n1 = (int)std::lround(std::sqrt((double)n));
    if (n1 < 1 || n1 * n1 != n) return EBEM_ERR_INVALID;
    std::vector<double> x(n1), wt(n1);
    for (int i = 0; i < n1; i++) {
        double z = std::cos(kPi * (i + 0.75) / (n1 + 0.5));
        double dp = 1.0;
        for (int it = 0; it < 100; it++) {
            double p0 = 1.0, p1 = z;
            for (int k = 2; k <= n1; k++) {
                double p2 = ((2 * k - 1) * z * p1 - (k - 1) * p0) / k;
                p0 = p1;
                p1 = p2;
            }
            dp = n1 * (z * p1 - p0) / (z * z - 1);
            double dz = p1 / dp;
            z -= dz;
            if (std::fabs(dz) < 1e-16) break;
        }
        double p0 = 1.0, p1 = z;
        for (int k = 2; k <= n1; k++) {
            double p2 = ((2 * k - 1) * z * p1 - (k - 1) * p0) / k;
            p0 = p1;
            p1 = p2;
        }
        dp = n1 * (z * p1 - p0) / (z * z - 1);
        x[n1 - 1 - i] = z;
        wt[n1 - 1 - i] = 2 / ((1 - z * z) * dp * dp);
    }
    if (n1 == 1) { x[0] = 0.0; wt[0] = 2.0; }
    nodes.resize(3 * (size_t)n);
    w.resize(n);
    for (int j = 0; j < n1; j++)
        for (int i = 0; i < n1; i++) {
            const double xi = 0.5 + x[i] / 2, xj = 0.5 + x[j] / 2, wi = wt[i] / 2, wj = wt[j] / 2;
            const int k = i + n1 * j;
            nodes[3 * k] = (1 - xj) * (1 - xi);
            nodes[3 * k + 1] = xj * (1 - xi);
            nodes[3 * k + 2] = xi;
            w[k] = 2 * wj * (wi * (1 - xi));
        }
    return EBEM_OK;
}

// ---------------------------------------------------------------------------
// mesh data

__global__ void dir_prep_kernel(const double* __restrict__ coords, const int32_t* __restrict__ tris, int nt,
                                DirTri* __restrict__ out) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nt) return;
    DirTri d;
    for (int a = 0; a < 3; a++)
        for (int c = 0; c < 3; c++) d.V[a][c] = coords[3 * tris[3 * t + a] + c];
    double g1[3], g2[3], g3[3];
    for (int c = 0; c < 3; c++) {
        g1[c] = d.V[0][c] - d.V[2][c];
        g2[c] = d.V[1][c] - d.V[2][c];
        g3[c] = d.V[0][c] - d.V[1][c];
    }
    double nn[3] = {g1[1] * g2[2] - g2[1] * g1[2], -g1[0] * g2[2] + g2[0] * g1[2], g1[0] * g2[1] - g2[0] * g1[1]};
    d.area = sqrt(nn[0] * nn[0] + nn[1] * nn[1] + nn[2] * nn[2]) / 2;
    for (int c = 0; c < 3; c++) d.n[c] = nn[c] / (2 * d.area);
    d.maxL = fmax(fmax(sqrt(g3[0] * g3[0] + g3[1] * g3[1] + g3[2] * g3[2]), sqrt(g2[0] * g2[0] + g2[1] * g2[1] + g2[2] * g2[2])),
                  sqrt(g1[0] * g1[0] + g1[1] * g1[1] + g1[2] * g1[2]));
    // P1 basis: M = A B^-1, B = [l21, l31, l21 x l31]; rows of B^-1 are
    // (l31 x n, n x l21, l21 x l31) / det
    double l21[3], l31[3];
    for (int c = 0; c < 3; c++) { l21[c] = d.V[1][c] - d.V[0][c]; l31[c] = d.V[2][c] - d.V[0][c]; }
    double cn[3] = {l21[1] * l31[2] - l21[2] * l31[1], l21[2] * l31[0] - l21[0] * l31[2], l21[0] * l31[1] - l21[1] * l31[0]};
    double r0[3] = {l31[1] * cn[2] - l31[2] * cn[1], l31[2] * cn[0] - l31[0] * cn[2], l31[0] * cn[1] - l31[1] * cn[0]};
    double r1[3] = {cn[1] * l21[2] - cn[2] * l21[1], cn[2] * l21[0] - cn[0] * l21[2], cn[0] * l21[1] - cn[1] * l21[0]};
    double det = l21[0] * r0[0] + l21[1] * r0[1] + l21[2] * r0[2];
    for (int c = 0; c < 3; c++) {
        r0[c] /= det;
        r1[c] /= det;
        d.M[c] = -r0[c] - r1[c];
        d.M[3 + c] = r0[c];
        d.M[6 + c] = r1[c];
    }
    for (int k = 0; k < 3; k++)
        d.v[k] = (k == 0 ? 1.0 : 0.0) - (d.M[3 * k] * d.V[0][0] + d.M[3 * k + 1] * d.V[0][1] + d.M[3 * k + 2] * d.V[0][2]);
    out[t] = d;
}

int prep_direct(MeshData& m, cudaStream_t s) {
    if (m.d_dir) return EBEM_OK;
    std::vector<int32_t> tris(3 * (size_t)m.nt);
    EBEM_CUDA_TRY(cudaMemcpy(tris.data(), m.d_tris, sizeof(int32_t) * tris.size(), cudaMemcpyDeviceToHost));
    std::vector<int32_t> off(m.nv + 1, 0), lst(3 * (size_t)m.nt);
    for (int32_t v : tris) off[v + 1]++;
    for (int v = 0; v < m.nv; v++) off[v + 1] += off[v];
    std::vector<int32_t> pos(off.begin(), off.end() - 1);
    for (int t = 0; t < m.nt; t++)
        for (int k = 0; k < 3; k++) lst[pos[tris[3 * t + k]]++] = t;      // ascending triangle order per vertex
    if (cudaMalloc(&m.d_dir, sizeof(DirTri) * (size_t)m.nt) != cudaSuccess ||
        cudaMalloc(&m.d_vt_off, sizeof(int32_t) * off.size()) != cudaSuccess ||
        cudaMalloc(&m.d_vt_tri, sizeof(int32_t) * lst.size()) != cudaSuccess) {
        cudaGetLastError();
        free_direct(m);
        return fail(EBEM_ERR_NOMEM, "direct-formulation mesh data allocation failed");
    }
    // d_dir marks the data as built: on a failure below it is released, so
    // the next call starts over instead of using a half-built table
    std::vector<DirTri> h(m.nt);
    cudaError_t e = cudaMemcpyAsync(m.d_vt_off, off.data(), sizeof(int32_t) * off.size(), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(m.d_vt_tri, lst.data(), sizeof(int32_t) * lst.size(), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        dir_prep_kernel<<<(m.nt + 127) / 128, 128, 0, s>>>(m.d_coords, m.d_tris, m.nt, m.d_dir);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h.data(), m.d_dir, sizeof(DirTri) * h.size(), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        free_direct(m);
        return fail(EBEM_ERR_CUDA, std::string("direct-formulation mesh data: ") + cudaGetErrorString(e));
    }
    m.max_len = 0.0;
    for (const DirTri& d : h) m.max_len = std::max(m.max_len, d.maxL);
    return EBEM_OK;
}

void free_direct(MeshData& m) {
    if (m.d_dir) cudaFree(m.d_dir);
    if (m.d_vt_off) cudaFree(m.d_vt_off);
    if (m.d_vt_tri) cudaFree(m.d_vt_tri);
    m.d_dir = nullptr;
    m.d_vt_off = m.d_vt_tri = nullptr;
}

// ---------------------------------------------------------------------------
// kernels of the direct formulation

struct Mat {
    double lam, mu, rho, cP, cS;
};

struct TimeF {
    double HP, HS, RP, RS, SP, SS;   // fronts, (t - r/c) H, (t - r/c)^2 (t + 2r/c) / 6 H
};

__device__ __forceinline__ TimeF time_f(double r, double t, const Mat& p) {
    TimeF f;
    const double tP = r / p.cP, tS = r / p.cS, aP = t - tP, aS = t - tS;
    f.HP = aP > 0 ? 1.0 : 0.0;
    f.HS = aS > 0 ? 1.0 : 0.0;
    f.RP = aP * f.HP;
    f.RS = aS * f.HS;
    f.SP = aP * aP * (t + 2 * tP) * (1.0 / 6) * f.HP;
    f.SS = aS * aS * (t + 2 * tS) * (1.0 / 6) * f.HS;
    return f;
}

__device__ __forceinline__ int levi(int a, int b, int c) {
    return (a == b || b == c || a == c) ? 0 : (((a + 1) % 3 == b) ? 1 : -1);
}

// Double-layer kernel (kernelK.cu: nucleoKL + nucleoKT - sum_j vms_j nucleoKRj)
// for basis value phik and vms = n x grad phi, x = outer - inner node.
// with_xn: the (x . n) terms (dropped on the same triangle); bad_front: the
// H(r - r/c_P) of kernelK.cu:414-449.
__device__ void kern_k(double out[9], const double x[3], double r, const double n[3], double t, const double vms[3],
                       double phik, const Mat& p, bool with_xn, bool bad_front) {
    const TimeF f = time_f(r, t, p);
    const double a1 = p.lam / (p.lam + p.mu), a2 = p.mu / (p.lam + p.mu);
    const double c1 = p.lam * p.mu / (p.rho * (p.lam + p.mu)), c2 = 2 * p.mu / p.rho;
    const double ir = q_rcp(r), ir2 = ir * ir, ir3 = ir2 * ir, ir5 = ir3 * ir2;
    const double icP = 1 / p.cP, icS = 1 / p.cS, icP2 = 1 / (p.cP * p.cP), icS2 = 1 / (p.cS * p.cS);
    const double xn = x[0] * n[0] + x[1] * n[1] + x[2] * n[2];
    const double D = f.RP - f.RS, DT = f.HP * icP - f.HS * icS;
    const double RPl = bad_front ? (t - r / p.cP) * ((r - r / p.cP) > 0 ? 1.0 : 0.0) : f.RP;
    const double Dl = f.RS * icS2 - RPl * icP2;
    const double Dd = f.RS * icS2 - f.RP * icP2;
    const double Hh = f.SS - f.SP;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const double mix = a1 * x[i] * n[k] + a2 * x[k] * n[i];
            double kl = mix * ir3 * D, kt = mix * ir2 * DT;
            if (with_xn && i == k) {
                kl += xn * ir3 * f.RS;
                kt += xn * ir2 * f.HS * icS;
            }
            double kr = 0.0;
#pragma unroll
            for (int j = 0; j < 3; j++) {
                double h = 0.0, d = 0.0;
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    const int e = levi(j, i, q);
                    if (e == 0) continue;
                    h += e * (3 * x[q] * x[k] * ir5 - ((q == k) ? ir3 : 0.0));
                    d += e * (x[q] * x[k] * ir3);
                }
                kr += vms[j] * (c1 * levi(j, k, i) * ir * Dl + c2 * h * Hh + c2 * d * Dd);
            }
            out[3 * i + k] = -kr + phik * (kl + kt);
        }
}

// Lame kernel twice integrated in time (kernelGHC.cu nucleo).  One reciprocal of r:
// with a quotient per entry and power the V diagonal took 324 us on 448 triangles, now
// 84, and the G part of 64 evaluations 310, now below 150.
__device__ __forceinline__ void kern_v(double nu[9], const double x[3], double r, double t, double cP, double cS) {
    const double HP = (t - r / cP) > 0 ? 1.0 : 0.0, HS = (t - r / cS) > 0 ? 1.0 : 0.0;
    const double ir = q_rcp(r), ir3 = ir * ir * ir, icP2 = 1 / (cP * cP), icS2 = 1 / (cS * cS);
    const double tail = t * t * (HP - HS) - r * r * (icP2 * HP - icS2 * HS);      // t^2 drops out past both fronts
    const double f = ir3 * (icP2 * HP - icS2 * HS) + 1.5 * (ir3 * ir * ir) * tail, d = ir * icS2 * HS - 0.5 * ir3 * tail;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) nu[3 * i + j] = f * (x[i] * x[j]) + (i == j ? d : 0.0);
}

__device__ __forceinline__ void bary_point(double y[3], const double* b, const double V[3][3]) {
#pragma unroll
    for (int c = 0; c < 3; c++) y[c] = b[0] * V[0][c] + b[1] * V[1][c] + b[2] * V[2][c];
}

__device__ __forceinline__ int local_index(const int32_t* tris, int t, int s) {
    return (tris[3 * t] == s) ? 1 : (tris[3 * t + 1] == s) ? 2 : (tris[3 * t + 2] == s) ? 3 : 0;
}

// ---------------------------------------------------------------------------
// K_l, off-singular part: one thread per (row triangle x, vertex s)

struct KArgs {
    const DirTri* tri;
    const double* coords;
    const int32_t* tris;
    const int32_t* vt_off;
    const int32_t* vt_tri;
    const double* outer;     // n_gh x 3
    const double* wout;      // n_gh
    const double* inner;     // n_in x 3 (n_sub x n_sing)
    const double* win;       // n_sing
    int n_gh, n_in, n_sing;
    int N, Nv;
    Mat p;
    double dt, max_len;
    int lag0, nlag, nblocks, fix;
    double* K;
    size_t ld, ld_lag;
};

__device__ __forceinline__ void k_emit(const KArgs& A, int l, int x, int s, const double Tm3[9], const double Tm2[9],
                                       const double Tm1[9], const double T[9], bool clamp) {
    double* base = A.K + (size_t)(l - A.lag0) * A.ld_lag + (3 * (size_t)s) * A.ld + 3 * (size_t)x;
    const double c = 4 * kPi * A.dt;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const int e = 3 * i + j;
            const double v = ((-Tm3[e] + 3 * Tm2[e]) + (-3 * Tm1[e])) + T[e];
            if (!clamp || fabs(v) > 1.0e-14) base[(size_t)j * A.ld + i] += v / c;
        }
}

// Third difference over the window of lag l, E_l = T_{l+1} - 3 T_l + 3 T_{l-1}
// - T_{l-2} on the levels t_k = k dt with levels k < 1 read as 0 (the lag
// combination of kernelK.cu), taken per node pair on the scalar time
// functions of one front X (arrival tX = r / c_X):
//   R = (t - tX) H,  H = [t - tX > 0],  S = (t - tX)^2 (t + 2 tX) / 6 H.
// Before the front all three vanish; with the whole window after it R is
// linear, H constant and S a cubic of leading coefficient 1/6, so the
// differences are exactly (0, 0, dt^3).  Only windows that a front crosses,
// or that reach below level 1, are summed level by level.
struct Win3 {
    double R, H, S;
};

// tl: the four levels, rounded products.
__device__ __forceinline__ Win3 front_window3(double tX, int l, const double tl[4], double dt) {
    Win3 d = {0.0, 0.0, 0.0};
    if (tl[3] - tX <= 0) return d;
    if (l >= 3 && tl[0] - tX > 0) {
        d.S = dt * dt * dt;
        return d;
    }
    const double c[4] = {-1.0, 3.0, -3.0, 1.0};
#pragma unroll
    for (int w = 0; w < 4; w++) {
        if (l - 2 + w < 1) continue;
        const double a = tl[w] - tX;
        if (a > 0) {
            d.R += c[w] * a;
            d.H += c[w];
            d.S += c[w] * (a * a * (tl[w] + 2 * tX) / 6);
        }
    }
    return d;
}

// Third difference of the linear (t - tP) of the reference's H(r - r/c_P)
// term (kernelK.cu:414-449): zero unless the window reaches below level 1.
__host__ __device__ __forceinline__ double lin_window3(double tP, int l, double dt) {
    if (l >= 3) return 0.0;
    const double c[4] = {-1.0, 3.0, -3.0, 1.0};
    double d = 0.0;
    for (int w = 0; w < 4; w++) {
        const int k = l - 2 + w;
        if (k >= 1) d += c[w] * (k * dt - tP);
    }
    return d;
}

struct KCoef {
    double a1, a2, c1, c2, icP, icS, icP2, icS2;
};

__host__ __device__ inline KCoef k_coef(const Mat& p) {
    KCoef c;
    c.a1 = p.lam / (p.lam + p.mu);
    c.a2 = p.mu / (p.lam + p.mu);
    c.c1 = p.lam * p.mu / (p.rho * (p.lam + p.mu));
    c.c2 = 2 * p.mu / p.rho;
    c.icP = 1 / p.cP;
    c.icS = 1 / p.cS;
    c.icP2 = 1 / (p.cP * p.cP);
    c.icS2 = 1 / (p.cS * p.cS);
    return c;
}

// One node pair's share of the lag-l third difference of the double-layer
// kernel (nucleoKL + nucleoKT - sum_j vms_j nucleoKRj of kernelK.cu), x =
// outer - inner node, n the field triangle's normal, v = vms.  With the
// window differences dRP, dRS, dHP, dHS, dRPl (the lambda-mu term's R_P) and
// dHh = dS_S - dS_P the kernel collapses to
//   out_ik = b1 (a1 x_i n_k + a2 x_k n_i) + b2 delta_ik - b3 w_i x_k - b4 u_ik,
//   w = v x x,  u_ik = sum_j eps_jik v_j,
//   b1 = phik (ir^3 (dRP - dRS) + ir^2 (dHP/c_P - dHS/c_S)),
//   b2 = phik (x.n) (ir^3 dRS + ir^2 dHS/c_S),
//   b3 = c2 ir^3 (dRP/c_P^2 - dRS/c_S^2) - 3 c2 ir^5 dHh,
//   b4 = c1 ir (dRPl/c_P^2 - dRS/c_S^2) - c2 ir^3 dHh,
// a1 = lambda/(lambda+mu), a2 = mu/(lambda+mu), c1 = lambda mu/(rho(lambda+mu)),
// c2 = 2 mu/rho.
__host__ __device__ __forceinline__ void k_pair(double out[9], const double x[3], double ir, const double n[3],
                                                const double v[3], double phik, double dRP, double dRS, double dHP,
                                                double dHS, double dRPl, double dHh, const KCoef& c) {
    const double ir2 = ir * ir, ir3 = ir2 * ir, ir5 = ir3 * ir2;
    const double xn = x[0] * n[0] + x[1] * n[1] + x[2] * n[2];
    const double b1 = phik * (ir3 * (dRP - dRS) + ir2 * (dHP * c.icP - dHS * c.icS));
    const double b2 = phik * xn * (ir3 * dRS + ir2 * dHS * c.icS);
    const double b3 = c.c2 * ir3 * (dRP * c.icP2 - dRS * c.icS2) - 3 * c.c2 * ir5 * dHh;
    const double b4 = c.c1 * ir * (dRPl * c.icP2 - dRS * c.icS2) - c.c2 * ir3 * dHh;
    const double w[3] = {v[1] * x[2] - v[2] * x[1], v[2] * x[0] - v[0] * x[2], v[0] * x[1] - v[1] * x[0]};
    const double u[9] = {0, v[2], -v[1], -v[2], 0, v[0], v[1], -v[0], 0};
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int k = 0; k < 3; k++)
            out[3 * i + k] = b1 * (c.a1 * x[i] * n[k] + c.a2 * x[k] * n[i]) + ((i == k) ? b2 : 0.0) -
                             b3 * w[i] * x[k] - b4 * u[3 * i + k];
}

// Thread per pair, for the rules of fewer than 6 node pairs a triangle on many
// pairs (see the launch): 128 registers (4 blocks an SM; 2800-triangle bar, rule
// 7/4/3: 633 ms, uncapped 725, 80 registers 721).
__global__ void __launch_bounds__(128, 4) k_assemble_thread_kernel(KArgs A) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (long long)A.N * A.Nv) return;
    const int x = (int)(p % A.N), s = (int)(p / A.N);
    const DirTri& X = A.tri[x];
    // isBlockNull (kernelK.cu:234-262), distMin starting at 100 unless fixed
    double distMax = 0.0, distMin = A.fix ? 1e300 : 100.0;
    for (int a = 0; a < 3; a++) {
        const double d0 = X.V[a][0] - A.coords[3 * s], d1 = X.V[a][1] - A.coords[3 * s + 1],
                     d2 = X.V[a][2] - A.coords[3 * s + 2];
        const double d = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
        distMax = fmax(distMax, d);
        distMin = fmin(distMin, d);
    }
    int llo = -1, lhi = -2;
    for (int q = 0; q < A.nlag; q++) {
        const int l = A.lag0 + q;
        if (l >= A.nblocks) break;
        const bool null = ((l - 2) * A.p.cS * A.dt > distMax + A.max_len) || ((l + 1) * A.p.cP * A.dt < distMin - 2 * A.max_len);
        if (!null) {
            if (llo < 0) llo = l;
            lhi = l;
        }
    }
    if (llo < 0) return;
    const int e0 = A.vt_off[s], e1 = A.vt_off[s + 1];
    const double cP = A.p.cP, cS = A.p.cS, dt = A.dt;
    const KCoef cd = k_coef(A.p);
    for (int l = llo; l <= lhi; l++) {
        // node pairs provably outside the window's fronts are skipped on r^2:
        // all four levels before the P front, or all after the S front
        const bool lin = !A.fix && l < 3;
        const double tl[4] = {level_time(l - 2, dt), level_time(l - 1, dt), level_time(l, dt), level_time(l + 1, dt)};
        const double skipP2 = lin ? 1e300 : (cP * tl[3]) * (cP * tl[3]) * (1 + 1e-12);
        const double skipS2 = (l >= 3) ? (cS * tl[0]) * (cS * tl[0]) * (1 - 1e-12) : -1.0;
        double T[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        for (int ee = e0; ee < e1; ee++) {
            const int m = A.vt_tri[ee];
            if (m == x) continue;
            const int kv = local_index(A.tris, m, s);
            const DirTri& F = A.tri[m];
            const double g[3] = {F.M[3 * (kv - 1)], F.M[3 * (kv - 1) + 1], F.M[3 * (kv - 1) + 2]};
            const double vms[3] = {F.n[1] * g[2] - F.n[2] * g[1], F.n[2] * g[0] - F.n[0] * g[2], F.n[0] * g[1] - F.n[1] * g[0]};
            for (int q = 0; q < A.n_in; q++) {
                double y[3];
                bary_point(y, A.inner + 3 * q, F.V);
                const double phik = F.v[kv - 1] + g[0] * y[0] + g[1] * y[1] + g[2] * y[2];
                const double wi = A.win[q % A.n_sing] * F.area;
                for (int o = 0; o < A.n_gh; o++) {
                    double xo[3];
                    bary_point(xo, A.outer + 3 * o, X.V);
                    const double pt[3] = {xo[0] - y[0], xo[1] - y[1], xo[2] - y[2]};
                    const double r2 = pt[0] * pt[0] + pt[1] * pt[1] + pt[2] * pt[2];
                    if (r2 > skipP2 || r2 < skipS2) continue;
                    const double r = sqrt(r2);
                    const double tP = r / cP, tS = r / cS;
                    const Win3 P = front_window3(tP, l, tl, dt), S = front_window3(tS, l, tl, dt);
                    const double dRPl = A.fix ? P.R : ((r - tP > 0) ? lin_window3(tP, l, dt) : 0.0);
                    const double dHh = S.S - P.S;
                    const double w = (A.wout[o] * X.area) * wi;
                    double v[9];
                    k_pair(v, pt, 1.0 / r, F.n, vms, phik, P.R, S.R, P.H, S.H, dRPl, dHh, cd);
#pragma unroll
                    for (int e = 0; e < 9; e++) T[e] += w * v[e];
                }
            }
        }
        double* base = A.K + (size_t)(l - A.lag0) * A.ld_lag + (3 * (size_t)s) * A.ld + 3 * (size_t)x;
        const double c = 4 * kPi * dt;
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++)
                if (fabs(T[3 * i + j]) > 1.0e-14) base[(size_t)j * A.ld + i] += T[3 * i + j] / c;
    }
}

// Warp per (row triangle x, vertex s), by front arrivals (front_bins.cuh).
// Bound by FP64 issue of the items, about 160 operations each, a quarter of them
// lanes without an item: rule 7/4/3 on 448 triangles 1000 items a pair.  The
// form before evaluated every node pair in every lag between its P and S
// arrival.  Rule 7/4/3: 448 triangles, 40 lags 16.1 -> 2.9 ms, 700 triangles
// 43 -> 7.5 ms, 2800 triangles, lags 40..49 283 -> 62 ms.  168 registers, 3
// blocks an SM; 2 blocks without the 100 bytes of spills 3.4 ms, 4 blocks 3.7.
//
// Over the levels k, k + 1, k + 2 from a front's arrival on, with a = t_k - tX
// and S_j = (a + j dt)^2 (a + j dt + 3 tX) / 6, the third difference is
//   lag k - 1:  a A + B + S_0 C,
//   lag k:      (dt - 2 a) A - 2 B + (S_1 - 3 S_0) C,
//   lag k + 1:  (a - dt) A + B + (S_2 - 3 S_1 + 3 S_0) C,
//   later:      dt^3 C,
// with the coefficients of R, H and S of the kernel as k_pair collects them,
// per front (sigma = 1 for P, -1 for S; M_ik = a1 x_i n_k + a2 x_k n_i):
//   A = sigma phik ir^3 M - sigma c2 ir^3/c^2 (w x) - sigma c1 ir/c^2 u
//       + [S] phik (x.n) ir^3 I   (the u term of P only with `fix`),
//   B = sigma phik ir^2/c M + [S] phik (x.n) ir^2/c I,
//   C = -sigma (3 c2 ir^5 (w x) + c2 ir^3 u).
// Without `fix` the reference's linear u term (lin_window3) is added over all
// node pairs in the lags below 3.
constexpr int kKWarps = 4;
constexpr size_t kKSmem = 200 * 1024;      // as kGHCSmem in ghc.cu
constexpr int kKNode = 12;               // x, y, z, weight, phik, -, normal, vms

// inner nodes of one chunk; 73 fill kBinChunk at 7 outer nodes, and the 170 of 3
// outer nodes would take the shared memory of a third block
inline __host__ __device__ int k_chunk(int n_gh) { return kBinChunk / n_gh < 73 ? kBinChunk / n_gh : 73; }
inline __host__ __device__ size_t k_warp_bytes(int n_gh, int lag0, int nlag) {
    const size_t b = (size_t)(kKNode * k_chunk(n_gh) + 4 * n_gh + 9 * nlag + 1) / 2 * 16 +
                     front_bins_bytes(bin_window(lag0, nlag).bins);
    return (b + 15) / 16 * 16;
}

__global__ void __launch_bounds__(32 * kKWarps, 3) k_assemble_kernel(KArgs A) {
    extern __shared__ __align__(16) unsigned char k_smem[];
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    const int chunk = k_chunk(A.n_gh);
    const BinWindow win = bin_window(A.lag0, A.nlag);
    double* nodes = reinterpret_cast<double*>(k_smem + (threadIdx.x >> 5) * k_warp_bytes(A.n_gh, A.lag0, A.nlag));
    double* xs = nodes + kKNode * chunk;
    double* acc = xs + 4 * A.n_gh;                     // 9 per lag
    FrontBins B = front_bins_at(reinterpret_cast<unsigned char*>(nodes + (kKNode * chunk + 4 * A.n_gh + 9 * A.nlag + 1) / 2 * 2),
                                win.bins);
    const float iout = 1.0f / (float)A.n_gh;           // (t + 1/2) iout: exact quotient for t < kBinChunk
    const double cP = A.p.cP, cS = A.p.cS, dt = A.dt, icdtP = 1 / (cP * dt), icdtS = 1 / (cS * dt);
    const double tail = dt * dt * dt, isc = 1 / (4 * kPi * dt);
    const KCoef cd = k_coef(A.p);
    for (long long p = warp; p < (long long)A.N * A.Nv; p += nwarps) {
        const int s = (int)((p <= 0xffffffffLL) ? (long long)((unsigned)p / (unsigned)A.N) : p / A.N);
        const int x = (int)(p - (long long)s * A.N);
        const DirTri& X = A.tri[x];
        // isBlockNull (kernelK.cu:234-262), distMin starting at 100 unless fixed
        double distMax = 0.0, distMin = A.fix ? 1e300 : 100.0;
        for (int a = 0; a < 3; a++) {
            const double d0 = X.V[a][0] - A.coords[3 * s], d1 = X.V[a][1] - A.coords[3 * s + 1],
                         d2 = X.V[a][2] - A.coords[3 * s + 2];
            const double d = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
            distMax = fmax(distMax, d);
            distMin = fmin(distMin, d);
        }
        int llo = 0x7fffffff, lhi = -1;
        for (int q = lane; q < A.nlag; q += 32) {
            const int l = A.lag0 + q;
            if (l >= A.nblocks) break;
            const bool null = ((l - 2) * A.p.cS * A.dt > distMax + A.max_len) ||
                              ((l + 1) * A.p.cP * A.dt < distMin - 2 * A.max_len);
            if (!null) {
                llo = min(llo, l);
                lhi = l;
            }
        }
        llo = __reduce_min_sync(0xffffffffu, llo);
        lhi = __reduce_max_sync(0xffffffffu, lhi);
        if (lhi < llo) continue;
        // star triangles but x itself
        const int e0 = A.vt_off[s], deg = A.vt_off[s + 1] - e0;
        int own = deg;
        for (int e = 0; e < deg; e++)
            if (A.vt_tri[e0 + e] == x) own = e;
        const int n_all = (deg - (own < deg)) * A.n_in;
        __syncwarp();
        for (int o = lane; o < A.n_gh; o += 32) {
            bary_point(xs + 4 * o, A.outer + 3 * o, X.V);
            xs[4 * o + 3] = A.wout[o] * X.area;
        }
        for (int t = lane; t < 9 * A.nlag; t += 32) acc[t] = 0.0;
        __syncwarp();
        bool any = false;
        for (int q0 = 0; q0 < n_all; q0 += chunk) {
            const int nq = min(chunk, n_all - q0), n = nq * A.n_gh;
            for (int q = lane; q < nq; q += 32) {
                int e = (q0 + q) / A.n_in;
                const int qi = (q0 + q) - e * A.n_in;
                e += e >= own;
                const int m = A.vt_tri[e0 + e], kv = local_index(A.tris, m, s) - 1;
                const DirTri& F = A.tri[m];
                const double g[3] = {F.M[3 * kv], F.M[3 * kv + 1], F.M[3 * kv + 2]};
                double* d = nodes + kKNode * q;
                bary_point(d, A.inner + 3 * qi, F.V);
                d[3] = A.win[qi % A.n_sing] * F.area;
                d[4] = F.v[kv] + g[0] * d[0] + g[1] * d[1] + g[2] * d[2];
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    d[6 + c] = F.n[c];
                    d[9 + c] = F.n[(c + 1) % 3] * g[(c + 2) % 3] - F.n[(c + 2) % 3] * g[(c + 1) % 3];
                }
            }
            __syncwarp();
            bool late = false, met = false;
            for (int t = lane; t < n; t += 32) {
                const int q = (int)(((float)t + 0.5f) * iout), o = t - q * A.n_gh;
                const double* d = nodes + kKNode * q;
                const double x0 = xs[4 * o] - d[0], x1 = xs[4 * o + 1] - d[1], x2 = xs[4 * o + 2] - d[2];
                const double r2 = x0 * x0 + x1 * x1 + x2 * x2, r = q_sqrt(r2);
                unsigned bP = front_bin(r2, r, cP, icdtP, dt, win);
                unsigned bS = front_bin(r2, r, cS, icdtS, dt, win);
                if (bS == 0) bP = bS = kNoBin;                    // past both fronts before the window: the constants cancel
                else late = late || bS == kNoBin;
                met = met || bP != kNoBin;
                B.bin[t] = make_ushort2((unsigned short)bP, (unsigned short)bS);
            }
            if (!A.fix && A.lag0 < 3) {
                for (int l = llo; l <= min(lhi, 2); l++) {
                    double u0 = 0.0, u1 = 0.0, u2 = 0.0;
                    for (int t = lane; t < n; t += 32) {
                        const int q = (int)(((float)t + 0.5f) * iout), o = t - q * A.n_gh;
                        const double* d = nodes + kKNode * q;
                        const double x0 = xs[4 * o] - d[0], x1 = xs[4 * o + 1] - d[1], x2 = xs[4 * o + 2] - d[2];
                        const double r = q_sqrt(x0 * x0 + x1 * x1 + x2 * x2), tP = r / cP;
                        if (r - tP > 0) {
                            const double f = lin_window3(tP, l, dt) * (xs[4 * o + 3] * d[3]) / r;
                            u0 += f * d[9];
                            u1 += f * d[10];
                            u2 += f * d[11];
                        }
                    }
                    for (int off = 16; off > 0; off >>= 1) {
                        u0 += __shfl_xor_sync(0xffffffffu, u0, off);
                        u1 += __shfl_xor_sync(0xffffffffu, u1, off);
                        u2 += __shfl_xor_sync(0xffffffffu, u2, off);
                    }
                    if (lane == 0) {
                        const double f = -cd.c1 * cd.icP2;
                        double* a = acc + 9 * (l - A.lag0);
                        a[1] += f * u2;
                        a[2] -= f * u1;
                        a[3] -= f * u2;
                        a[5] += f * u0;
                        a[6] += f * u1;
                        a[7] -= f * u0;
                    }
                    any = true;
                }
                __syncwarp();
            }
            if (!__any_sync(0xffffffffu, met)) continue;            // both fronts miss the window
            late = __any_sync(0xffffffffu, late);
            any = true;
            const int total = bins_sort(B, n, win.bins, lane);
            double cur[9] = {0}, n1[9] = {0}, n2[9] = {0}, run[9] = {0};
            double last = 0.0, last9 = 0.0;           // this lane's reduced entry and entry 33 of the lag before
            int first = B.off[0], idle = 0;           // idle: bins without items up to this one
            for (int i = lane; i < first; i += 32) {  // bin 0: the constant only
                const unsigned it = B.list[i];
                const int t = (int)(it & 0x7fffffffu), q = (int)(((float)t + 0.5f) * iout), o = t - q * A.n_gh;
                const double* d = nodes + kKNode * q;
                const double y[3] = {xs[4 * o] - d[0], xs[4 * o + 1] - d[1], xs[4 * o + 2] - d[2]}, v[3] = {d[9], d[10], d[11]};
                const double r2 = y[0] * y[0] + y[1] * y[1] + y[2] * y[2], ir = q_rcp(q_sqrt(r2)), ir2 = ir * ir;
                const double w = xs[4 * o + 3] * d[3], uC = -cd.c2 * (it >> 31 ? -w : w) * (ir2 * ir), wC = 3 * uC * ir2;
                const double wx[3] = {v[1] * y[2] - v[2] * y[1], v[2] * y[0] - v[0] * y[2], v[0] * y[1] - v[1] * y[0]};
                if (r2 > 0)
#pragma unroll
                    for (int e = 0; e < 9; e++) {
                        const int r = e / 3, c = e - 3 * r;
                        double g = tail * (wC * (wx[r] * y[c]));
                        if (r != c) g += tail * (uC * ((c - r + 3) % 3 == 1 ? v[(c + 1) % 3] : -v[(r + 1) % 3]));
                        run[e] += g;
                    }
            }
            for (int b = 1; b < win.bins; b++) {
                const int k = win.kbase + b - 1, l = k - 1, lastitem = B.off[b], items = lastitem - first;
                if (items == 0 && first == 0) continue;                 // before the first arrival
                if (l > lhi) break;
                idle = items ? 0 : idle + 1;
                const double tk = k * dt;
                for (int i = first + lane; i < lastitem; i += 32) {
                    const unsigned it = B.list[i];
                    const bool isS = it >> 31;
                    const int t = (int)(it & 0x7fffffffu), q = (int)(((float)t + 0.5f) * iout), o = t - q * A.n_gh;
                    const double* d = nodes + kKNode * q;
                    const double y[3] = {xs[4 * o] - d[0], xs[4 * o + 1] - d[1], xs[4 * o + 2] - d[2]};
                    const double nn[3] = {d[6], d[7], d[8]}, v[3] = {d[9], d[10], d[11]};
                    const double r2 = y[0] * y[0] + y[1] * y[1] + y[2] * y[2], r = q_sqrt(r2), ir = q_rcp(r);
                    const double w = xs[4 * o + 3] * d[3], sw = isS ? -w : w, wp = w * d[4];
                    const double ic = isS ? cd.icS : cd.icP, ic2 = isS ? cd.icS2 : cd.icP2;
                    const double ir2 = ir * ir, ir3 = ir2 * ir, tX = r * ic;
                    const double mB = (isS ? -wp : wp) * ir2 * ic, mA = (isS ? -wp : wp) * ir3;
                    const double xn = isS ? y[0] * nn[0] + y[1] * nn[1] + y[2] * nn[2] : 0.0;
                    const double uC = -cd.c2 * sw * ir3, wA = uC * ic2, wC = 3 * uC * ir2;
                    const double uA = isS || A.fix ? -cd.c1 * sw * ir * ic2 : 0.0;
                    const double a0 = tk - tX, a1 = a0 + dt, a2 = a1 + dt;
                    const double S0 = a0 * a0 * (a0 + 3 * tX) * (1.0 / 6), S1 = a1 * a1 * (a1 + 3 * tX) * (1.0 / 6),
                                 S2 = a2 * a2 * (a2 + 3 * tX) * (1.0 / 6);
                    const double al[3] = {a0, dt - 2 * a0, a0 - dt}, be[3] = {1.0, -2.0, 1.0};
                    const double ga[3] = {S0 - tail, S1 - 3 * S0 - tail, S2 - 3 * S1 + 3 * S0 - tail};
                    const double wx[3] = {v[1] * y[2] - v[2] * y[1], v[2] * y[0] - v[0] * y[2], v[0] * y[1] - v[1] * y[0]};
                    double pM[3], pI[3], pW[3], pU[3];
#pragma unroll
                    for (int j = 0; j < 3; j++) {
                        pM[j] = al[j] * mA + be[j] * mB;
                        pI[j] = -xn * pM[j];
                        pW[j] = al[j] * wA + ga[j] * wC;
                        pU[j] = al[j] * uA + ga[j] * uC;
                    }
#pragma unroll
                    for (int i = 0; i < 3; i++)
#pragma unroll
                        for (int c = 0; c < 3; c++) {
                            const int e = 3 * i + c;
                            const double M = cd.a1 * y[i] * nn[c] + cd.a2 * y[c] * nn[i], W = wx[i] * y[c];
                            double f[3], g = tail * (wC * W);
#pragma unroll
                            for (int j = 0; j < 3; j++) f[j] = pM[j] * M + pW[j] * W;
                            if (i == c) {
#pragma unroll
                                for (int j = 0; j < 3; j++) f[j] += pI[j];
                            } else {
                                const double u = (c - i + 3) % 3 == 1 ? v[(c + 1) % 3] : -v[(i + 1) % 3];
#pragma unroll
                                for (int j = 0; j < 3; j++) f[j] += pU[j] * u;
                                g += tail * (uC * u);
                            }
                            cur[e] += f[0];
                            n1[e] += f[1];
                            n2[e] += f[2];
                            if (r2 > 0) run[e] += g;                    // r = 0: both fronts here at once, no constant remains
                        }
                }
                if (l >= A.lag0) {
                    if (idle < 4 || l == A.lag0) {
                        double v[8];
#pragma unroll
                        for (int e = 0; e < 8; e++) v[e] = cur[e] + run[e];
                        last = warp_reduce_scatter8(v, lane);
                        last9 = cur[8] + run[8];
                        for (int off = 16; off > 0; off >>= 1) last9 += __shfl_xor_sync(0xffffffffu, last9, off);
                    }
                    double* a = acc + 9 * (l - A.lag0);
                    if ((lane & 3) == 0) a[scatter8_entry(lane)] += last;
                    if (lane == 1) a[8] += last9;
                }
                first = lastitem;
#pragma unroll
                for (int e = 0; e < 9; e++) {
                    cur[e] = n1[e];
                    n1[e] = n2[e];
                    n2[e] = 0.0;
                }
                if (!late && first == total && idle > 1) break;         // every node pair is past both fronts
            }
            __syncwarp();
        }
        if (!any) continue;
        double* base = A.K + (3 * (size_t)s) * A.ld + 3 * (size_t)x;
        for (int t = lane; t < 9 * (lhi - llo + 1); t += 32) {
            const int l = t / 9, e = t - 9 * l, j = e / 3, i = e - 3 * j;
            const double v = acc[9 * (llo + l - A.lag0) + 3 * i + j];
            if (fabs(v) > 1.0e-14) base[(size_t)(llo + l - A.lag0) * A.ld_lag + (size_t)j * A.ld + i] += v * isc;
        }
    }
}

// Same-triangle parts of K_l, in two passes.  Levels: one warp per (triangle
// x, local vertex kv, level k) over the call's levels kmin..kmin+nk-1, the
// lanes over the (outer node, child, DIAG node) evaluations, reduced over the
// warp into Tb[3x + kv - 1][k - kmin]; a level outside the triangle's own
// range klo..khi (its parts vanish from lag lmax on) is left unwritten and
// never read.  Emission: one thread per (x, kv, lag) adds the third
// difference (k_emit), levels below klo read as zero.  (One thread per
// (x, kv) walking all levels left most SMs idle on small meshes.)
struct KSingRange {
    int llo, lhi, klo, khi;
};
__device__ __forceinline__ KSingRange k_sing_range(const KArgs& A, const DirTri& X) {
    KSingRange r;
    const int lmax = (int)ceil(X.maxL / (A.p.cS * A.dt)) + 2;      // lags >= lmax are zero
    r.llo = A.lag0;
    r.lhi = min(A.lag0 + A.nlag - 1, lmax - 1);
    r.klo = max(1, r.llo - 2);
    r.khi = r.lhi + 1;
    return r;
}

__global__ void __launch_bounds__(128) k_sing_level_kernel(KArgs A, const double* __restrict__ dn,
                                                           const double* __restrict__ dw, int n_diag, int kmin, int nk,
                                                           double* __restrict__ Tb) {
    const int lane = threadIdx.x & 31;
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= 3LL * A.N * nk) return;                    // uniform across the warp
    const int p = (int)(w / nk), kk = (int)(w - (long long)p * nk);
    const int x = p / 3, kv = p % 3 + 1;
    const DirTri& X = A.tri[x];
    const KSingRange rg = k_sing_range(A, X);
    const int k = kmin + kk;
    if (rg.lhi < rg.llo || k < rg.klo || k > rg.khi) return;
    const double t = k * A.dt;
    const double g[3] = {X.M[3 * (kv - 1)], X.M[3 * (kv - 1) + 1], X.M[3 * (kv - 1) + 2]};
    const double vms[3] = {X.n[1] * g[2] - X.n[2] * g[1], X.n[2] * g[0] - X.n[0] * g[2], X.n[0] * g[1] - X.n[1] * g[0]};
    const int per_o = 3 * n_diag, total = A.n_gh * per_o;
    double T[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int c = lane; c < total; c += 32) {
        const int o = c / per_o, rem = c - o * per_o, ch = rem / n_diag, d = rem - ch * n_diag;
        double xo[3];
        bary_point(xo, A.outer + 3 * o, X.V);
        const int a = ch, b = (ch + 2) % 3;               // children (V1,V3,x), (V2,V1,x), (V3,V2,x)
        const double ea[3] = {X.V[a][0] - xo[0], X.V[a][1] - xo[1], X.V[a][2] - xo[2]};
        const double eb[3] = {X.V[b][0] - xo[0], X.V[b][1] - xo[1], X.V[b][2] - xo[2]};
        const double cr[3] = {ea[1] * eb[2] - ea[2] * eb[1], ea[2] * eb[0] - ea[0] * eb[2], ea[0] * eb[1] - ea[1] * eb[0]};
        const double ac = sqrt(cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2]) / 2;
        const double* bd = dn + 3 * d;
        double y[3];
#pragma unroll
        for (int q = 0; q < 3; q++) y[q] = bd[0] * X.V[a][q] + bd[1] * X.V[b][q] + bd[2] * xo[q];
        const double R[3] = {xo[0] - y[0], xo[1] - y[1], xo[2] - y[2]};
        const double r = sqrt(R[0] * R[0] + R[1] * R[1] + R[2] * R[2]);
        const double phik = X.v[kv - 1] + g[0] * y[0] + g[1] * y[1] + g[2] * y[2];
        double v[9];
        kern_k(v, R, r, X.n, t, vms, phik, A.p, false, false);
        const double wgt = (X.area * A.wout[o]) * (dw[d] * ac);
#pragma unroll
        for (int e = 0; e < 9; e++) T[e] += wgt * v[e];
    }
#pragma unroll
    for (int e = 0; e < 9; e++)
        for (int off = 16; off > 0; off >>= 1) T[e] += __shfl_xor_sync(0xffffffffu, T[e], off);
    if (lane < 9) {
        double v = 0.0;
#pragma unroll
        for (int e = 0; e < 9; e++)
            if (e == lane) v = T[e];
        Tb[((size_t)p * nk + kk) * 9 + lane] = v;
    }
}

__global__ void __launch_bounds__(128) k_sing_emit_kernel(KArgs A, int kmin, int nk, const double* __restrict__ Tb) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= 3LL * A.N * A.nlag) return;
    const int p = (int)(idx / A.nlag), q = (int)(idx - (long long)p * A.nlag);
    const int x = p / 3, kv = p % 3 + 1;
    const KSingRange rg = k_sing_range(A, A.tri[x]);
    const int l = A.lag0 + q;
    if (l > rg.lhi) return;
    double Tl[4][9];                                    // levels l-2, l-1, l, l+1
#pragma unroll
    for (int h = 0; h < 4; h++) {
        const int k = l - 2 + h;
#pragma unroll
        for (int e = 0; e < 9; e++) Tl[h][e] = (k >= rg.klo) ? Tb[((size_t)p * nk + (k - kmin)) * 9 + e] : 0.0;
    }
    k_emit(A, l, x, A.tris[3 * x + kv - 1], Tl[0], Tl[1], Tl[2], Tl[3], false);
}

// Diagonal blocks of V_l on the DIAG rule, in two passes.  Levels: one warp
// per (triangle x, time level k), the lanes over the (outer node, child, DIAG
// node) evaluations of the level integral T_k (9 entries), reduced over the
// warp into Tb[x][k - kmin].  Combine: one thread per (triangle, lag, entry),
// V_l = (T_{l+1} - 2 T_l + T_{l-1}) / (4 pi rho) with T_0 taken as zero.
// (One thread per triangle walking every level left all but a few SMs idle
// on meshes of a few hundred triangles.)
__global__ void __launch_bounds__(128) v_diag_level_kernel(const DirTri* __restrict__ tri, int N,
                                                           const double* __restrict__ outer,
                                                           const double* __restrict__ wout, int n_gh,
                                                           const double* __restrict__ dn, const double* __restrict__ dw,
                                                           int n_diag, double cP, double cS, double dt, int kmin, int nk,
                                                           double* __restrict__ Tb) {
    const int lane = threadIdx.x & 31;
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= (long long)N * nk) return;                 // uniform across the warp
    const int x = (int)(w / nk), kk = (int)(w - (long long)x * nk);
    const double t = (kmin + kk) * dt;
    const DirTri& X = tri[x];
    const int per_o = 3 * n_diag, total = n_gh * per_o;
    double T[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int c = lane; c < total; c += 32) {
        const int o = c / per_o, rem = c - o * per_o, ch = rem / n_diag, d = rem - ch * n_diag;
        double xo[3];
        bary_point(xo, outer + 3 * o, X.V);
        const int a = ch, b = (ch + 2) % 3;
        const double ea[3] = {X.V[a][0] - xo[0], X.V[a][1] - xo[1], X.V[a][2] - xo[2]};
        const double eb[3] = {X.V[b][0] - xo[0], X.V[b][1] - xo[1], X.V[b][2] - xo[2]};
        const double cr[3] = {ea[1] * eb[2] - ea[2] * eb[1], ea[2] * eb[0] - ea[0] * eb[2], ea[0] * eb[1] - ea[1] * eb[0]};
        const double ac = sqrt(cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2]) / 2;
        const double* bd = dn + 3 * d;
        double X3[3];
#pragma unroll
        for (int q = 0; q < 3; q++) X3[q] = (bd[0] * X.V[a][q] + bd[1] * X.V[b][q] + bd[2] * xo[q]) - xo[q];
        double nu[9];
        kern_v(nu, X3, sqrt(X3[0] * X3[0] + X3[1] * X3[1] + X3[2] * X3[2]), t, cP, cS);
        const double wgt = (X.area * wout[o]) * (dw[d] * ac);
#pragma unroll
        for (int e = 0; e < 9; e++) T[e] += wgt * nu[e];
    }
#pragma unroll
    for (int e = 0; e < 9; e++)
        for (int off = 16; off > 0; off >>= 1) T[e] += __shfl_xor_sync(0xffffffffu, T[e], off);
    if (lane < 9) {
        double v = 0.0;
#pragma unroll
        for (int e = 0; e < 9; e++)
            if (e == lane) v = T[e];
        Tb[((size_t)x * nk + kk) * 9 + lane] = v;
    }
}

__global__ void __launch_bounds__(128) v_diag_combine_kernel(const double* __restrict__ Tb, int N, int kmin, int nk,
                                                             int lag0, int nlag, double c4pirho, double* __restrict__ V,
                                                             size_t ld, size_t ld_lag) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)N * nlag * 9) return;
    const int e = (int)(idx % 9);
    const long long r = idx / 9;
    const int q = (int)(r % nlag), x = (int)(r / nlag);
    const int l = lag0 + q, k = l + 1;
    auto level = [&](int kk) {
        return (kk >= kmin && kk < kmin + nk) ? Tb[((size_t)x * nk + (kk - kmin)) * 9 + e] : 0.0;
    };
    const double prev = (l - 1 >= 1) ? level(k - 2) : 0.0;
    const int i = e / 3, j = e - 3 * i;
    V[(size_t)q * ld_lag + (3 * (size_t)x + j) * ld + 3 * (size_t)x + i] = ((level(k) - 2 * level(k - 1)) + prev) / c4pirho;
}

// Rule tables in one device buffer.
struct Tables {
    double* d = nullptr;
    size_t outer = 0, wout = 0, inner = 0, win = 0, dn = 0, dw = 0;
    cudaStream_t st = nullptr;
    ~Tables() { ws_free(d, st); }
};

static int upload_tables(Tables& T, int n_gh, int n_sub, int n_sing, int n_diag, cudaStream_t s) {
    std::vector<double> buf;
    double ob[28 * 3], ow[28];
    if (n_gh > 0) {
        if (gh_composite(n_gh, 1, ob, ow)) return fail(EBEM_ERR_INVALID, "unsupported outer rule");
        T.outer = buf.size(); buf.insert(buf.end(), ob, ob + 3 * n_gh);
        T.wout = buf.size(); buf.insert(buf.end(), ow, ow + n_gh);
    }
    if (n_sing > 0) {
        std::vector<double> ib((size_t)3 * n_sub * n_sing), iw(n_sing);
        if (gh_composite(n_sing, n_sub, ib.data(), iw.data())) return fail(EBEM_ERR_INVALID, "unsupported inner rule");
        T.inner = buf.size(); buf.insert(buf.end(), ib.begin(), ib.end());
        T.win = buf.size(); buf.insert(buf.end(), iw.begin(), iw.end());
    }
    if (n_diag > 0) {
        std::vector<double> dn, dw;
        if (diag_rule(n_diag, dn, dw)) return fail(EBEM_ERR_INVALID, "DIAG rule size must be a square");
        T.dn = buf.size(); buf.insert(buf.end(), dn.begin(), dn.end());
        T.dw = buf.size(); buf.insert(buf.end(), dw.begin(), dw.end());
    }
    if (buf.empty()) buf.push_back(0.0);
    T.st = s;
    EBEM_CUDA_TRY(ws_malloc(&T.d, buf.size() * sizeof(double), s));
    EBEM_CUDA_TRY(cudaMemcpyAsync(T.d, buf.data(), buf.size() * sizeof(double), cudaMemcpyHostToDevice, s));
    return EBEM_OK;
}

static Mat mat_of(const PhysParams& P) {
    Mat p;
    p.lam = P.lam;
    p.mu = P.mu;
    p.rho = P.rho;
    p.cP = P.velP;
    p.cS = P.velS;
    return p;
}

int launch_k_assemble(const MeshData& m, const PhysParams& P, int n_gh, int n_sub, int n_sing, int n_diag, int lag0,
                      int nlag, int nblocks, int fix, double* d_K, cudaStream_t s) {
    Tables T;
    if (int rc = upload_tables(T, n_gh, n_sub, n_sing, n_diag, s)) return rc;
    KArgs A;
    A.tri = m.d_dir;
    A.coords = m.d_coords;
    A.tris = m.d_tris;
    A.vt_off = m.d_vt_off;
    A.vt_tri = m.d_vt_tri;
    A.outer = T.d + T.outer;
    A.wout = T.d + T.wout;
    A.inner = T.d + T.inner;
    A.win = T.d + T.win;
    A.n_gh = n_gh;
    A.n_in = n_sub * n_sing;
    A.n_sing = n_sing;
    A.N = m.nt;
    A.Nv = m.nv;
    A.p = mat_of(P);
    A.dt = P.dt;
    A.max_len = m.max_len;
    A.lag0 = lag0;
    A.nlag = nlag;
    A.nblocks = nblocks;
    A.fix = fix;
    A.K = d_K;
    A.ld = 3 * (size_t)m.nt;
    A.ld_lag = A.ld * 3 * (size_t)m.nv;
    const long long pairs = (long long)m.nt * m.nv;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m.device);
    // The pair's sums per lag cost the warp kernel a fixed share: rule 3/1/1 takes
    // it 29 ms on the 2800-triangle bar (lags 40..49) against 14 by threads, rule
    // 3/1/3 25 against 34, 7/1/3 30 against 72.  On few pairs the threads do not
    // fill the chip (3/1/1: 448 triangles 1.4 against 2.0 ms, 80: 0.13 against 0.60).
    // On windows of few lags, as in ghc.cu: rule 3/1/3, lags from the middle of the
    // run, 1 and 4 of them 3.8 and 14.5 ms by threads against 12.4 and 16.8 on the
    // bar (12 lags 41.4 against 26.9), 0.20 and 0.64 against 0.33 and 0.46 on 448
    // triangles; 7/4/3, 1 lag 29.8 against 33.0 and 1.26 against 0.68.
    const int np = n_gh * n_sub * n_sing;
    const bool byThread = (np < 6 && pairs >= 1024LL * sms) ||
                          (pairs >= 128LL * sms && nlag * (np * (1 + 5.2 * sms / m.nt)) < 47 + 0.73 * np);
    if (byThread) {
        k_assemble_thread_kernel<<<(unsigned)((pairs + 127) / 128), 128, 0, s>>>(A);
        EBEM_CUDA_TRY(cudaGetLastError());
    }
    KArgs W = A;
    for (int l0 = 0; !byThread && l0 < nlag; l0 += kBinLags) {
        W.lag0 = lag0 + l0;
        W.nlag = std::min(nlag - l0, kBinLags);
        W.K = d_K + (size_t)l0 * A.ld_lag;
        const size_t each = k_warp_bytes(n_gh, W.lag0, W.nlag);
        const int warps = (int)std::max<size_t>(1, std::min<size_t>(kKWarps, kKSmem / each));
        EBEM_CUDA_TRY(cudaFuncSetAttribute(k_assemble_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kKSmem));
        const long long want = (pairs + warps - 1) / warps, cap = (long long)sms * 64;
        k_assemble_kernel<<<(unsigned)(want < cap ? want : cap), 32 * warps, warps * each, s>>>(W);
        EBEM_CUDA_TRY(cudaGetLastError());
    }
    if (n_diag > 0) {
        const int kmin = std::max(1, lag0 - 2), nk = lag0 + nlag - kmin + 1;
        double* Tb = nullptr;
        EBEM_CUDA_TRY(ws_malloc(&Tb, sizeof(double) * 27 * (size_t)m.nt * nk, s));
        const long long lv_threads = 32LL * 3 * m.nt * nk, em_threads = 3LL * m.nt * nlag;
        k_sing_level_kernel<<<(unsigned)((lv_threads + 127) / 128), 128, 0, s>>>(A, T.d + T.dn, T.d + T.dw, n_diag, kmin,
                                                                                  nk, Tb);
        k_sing_emit_kernel<<<(unsigned)((em_threads + 127) / 128), 128, 0, s>>>(A, kmin, nk, Tb);
        cudaError_t e = cudaGetLastError();
        ws_free(Tb, s);
        if (e != cudaSuccess) return fail(EBEM_ERR_CUDA, std::string("K same-triangle parts: ") + cudaGetErrorString(e));
    }
    EBEM_CUDA_TRY(cudaStreamSynchronize(s));
    return EBEM_OK;
}

int launch_v_diag(const MeshData& m, const PhysParams& P, int n_gh, int n_diag, int lag0, int nlag, double* d_V,
                  cudaStream_t s) {
    Tables T;
    if (int rc = upload_tables(T, n_gh, 0, 0, n_diag, s)) return rc;
    const size_t ld = 3 * (size_t)m.nt;
    // levels k = kmin .. lag0 + nlag (t = k dt; t = 0 contributes nothing)
    const int kmin = std::max(1, lag0 - 1), nk = lag0 + nlag - kmin + 1;
    double* Tb = nullptr;
    EBEM_CUDA_TRY(ws_malloc(&Tb, sizeof(double) * 9 * (size_t)m.nt * nk, s));
    const long long lv_threads = 32LL * m.nt * nk, cb_threads = 9LL * m.nt * nlag;
    v_diag_level_kernel<<<(unsigned)((lv_threads + 127) / 128), 128, 0, s>>>(
        m.d_dir, m.nt, T.d + T.outer, T.d + T.wout, n_gh, T.d + T.dn, T.d + T.dw, n_diag, P.velP, P.velS, P.dt, kmin,
        nk, Tb);
    v_diag_combine_kernel<<<(unsigned)((cb_threads + 127) / 128), 128, 0, s>>>(Tb, m.nt, kmin, nk, lag0, nlag,
                                                                               4 * kPi * P.rho, d_V, ld, ld * ld);
    cudaError_t e = cudaGetLastError();
    ws_free(Tb, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail(EBEM_ERR_CUDA, std::string("V diagonal blocks: ") + cudaGetErrorString(e));
    return EBEM_OK;
}

// ---------------------------------------------------------------------------
// post-processing: the G part a thread per (triangle, evaluation (t, x), chunk of
// slices), the P part a warp per (vertex, evaluation, chunk of slices)

struct PPArgs {
    const DirTri* tri;
    const int32_t* tris;
    const int32_t* vt_off;
    const int32_t* vt_tri;
    const double* pn;        // n_sub * n_sing x 3
    const double* pw;        // n_sing
    int n_sub, n_sing, gstride;
    int N, Nv;
    Mat p;
    double dt;
    const double* pts;       // npts x 3
    const double* times;     // ntimes (device copy)
    int npts, ntimes, nT;
    const double* a;         // 3N x nT  (multiplies G)
    const double* b;         // 3Nv x nT (multiplies P)
    double* u;               // ntimes x npts x 3
    double* G;               // matrix mode
    double* Pm;
    int mode;
};

__device__ __forceinline__ void warp_add3(double* dst, double v0, double v1, double v2) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v0 += __shfl_xor_sync(0xffffffffu, v0, o);
        v1 += __shfl_xor_sync(0xffffffffu, v1, o);
        v2 += __shfl_xor_sync(0xffffffffu, v2, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (v0 != 0.0) atomicAdd(dst, v0);
        if (v1 != 0.0) atomicAdd(dst + 1, v1);
        if (v2 != 0.0) atomicAdd(dst + 2, v2);
    }
}

// G part: sum over slices n of clamp(G(t - (n-1) dt) - G(t - n dt)) / (4 pi rho) a_n.
// Block (x-tile, evaluation, chunk c) takes the slices n in
// [c kchunk + 1, (c + 1) kchunk] and evaluates G at the levels n_lo - 1 .. n_hi
// (one level more than its slices), so that short meshes still fill the GPU.
// 128 registers (4 blocks per SM); 16 points x 4 times on the 448-triangle bar,
// G and P together, 0.46 ms, and 0.44 with 2 or 6 blocks.
__global__ void __launch_bounds__(128, 4) pp_g_kernel(PPArgs A, int kchunk) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int ev = blockIdx.y;                          // evaluation index q * npts + ip
    const int q = ev / A.npts, ip = ev % A.npts;
    const double t = A.times[q];
    const double* src = A.pts + 3 * ip;
    const int nhat = (t > 0) ? (int)ceil(t / A.dt) : 0;
    const int n_lo = blockIdx.z * kchunk + 1, n_hi = min((int)(blockIdx.z + 1) * kchunk, nhat);
    double u0 = 0.0, u1 = 0.0, u2 = 0.0;
    if (x < A.N && n_lo <= n_hi) {
        const DirTri& X = A.tri[x];
        double Gp[9] = {0}, Gk[9];
        const double c4 = 4 * kPi * A.p.rho;
        for (int k = n_lo - 1; k <= n_hi; k++) {
            const double tk = t - level_time(k, A.dt);
#pragma unroll
            for (int e = 0; e < 9; e++) Gk[e] = 0.0;
            if (tk > 0) {
                for (int tx = 0; tx < A.n_sub; tx++)
                    for (int l = 0; l < A.n_sing; l++) {
                        double y[3];
                        bary_point(y, A.pn + 3 * (A.gstride * tx + l), X.V);
                        const double pt[3] = {y[0] - src[0], y[1] - src[1], y[2] - src[2]};
                        double nu[9];
                        kern_v(nu, pt, sqrt(pt[0] * pt[0] + pt[1] * pt[1] + pt[2] * pt[2]), tk, A.p.cP, A.p.cS);
                        const double w = A.pw[l] * X.area;
#pragma unroll
                        for (int e = 0; e < 9; e++) Gk[e] += w * nu[e];
                    }
            }
            if (k >= n_lo) {
                const int n = k;                        // slice n uses instants t - (n-1) dt and t - n dt
                double S[9];
#pragma unroll
                for (int e = 0; e < 9; e++) {
                    const double v = Gp[e] - Gk[e];
                    S[e] = (fabs(v) > 1.0e-14) ? v / c4 : 0.0;
                }
                if (A.mode == 1) {
                    const size_t R = 3 * (size_t)nhat;
#pragma unroll
                    for (int i = 0; i < 3; i++)
#pragma unroll
                        for (int j = 0; j < 3; j++) A.G[(3 * (size_t)x + j) * R + 3 * (size_t)(n - 1) + i] = S[3 * i + j];
                } else if (n <= A.nT) {
                    const double* an = A.a + (size_t)(n - 1) * 3 * A.N + 3 * (size_t)x;
                    u0 += S[0] * an[0] + S[1] * an[1] + S[2] * an[2];
                    u1 += S[3] * an[0] + S[4] * an[1] + S[5] * an[2];
                    u2 += S[6] * an[0] + S[7] * an[1] + S[8] * an[2];
                }
            }
#pragma unroll
            for (int e = 0; e < 9; e++) Gp[e] = Gk[e];
        }
    }
    if (A.mode == 0) warp_add3(A.u + 3 * (size_t)ev, u0, u1, u2);
}

// P part: minus the sum over slices n of clamp(P_{n-1} - 2 P_n + P_{n+1}) / (4 pi rho dt) b_n.
//
// Warp per (evaluation, vertex, chunk of slices), by front arrivals
// (front_bins.cuh) in the levels j = nhat + 1 - k, ascending in time: slice n has
// the centre c = nhat + 1 - n and takes the levels c - 1, c, c + 1.  With a the
// time since the arrival at the first level k of a front and S_j = (a + j dt)^2
// (a + j dt + 3 tX) / 6, its second difference is
//   centre k - 1:  H + a R + S_0 S,   centre k:  -H + (dt - a) R + (S_1 - 2 S_0) S,
//   later:         dt^2 t_c S,
// H, R, S the coefficients of the front's time functions in the traction kernel
// of kernelP.cu times phik, x = source - node, xn = x . n, in x_i n_j, x_j n_i,
// xn delta_ij, xn x_i x_j:
//   P:  H  (lam, 0, 0, 2 mu ir^2) ir^2 / c_P^3,  S: H  mu (0, 1, 1, -2 ir^2) ir^2 / c_S^3,
//       R  (lam - 2 mu, -2 mu, -2 mu, 12 mu ir^2) ir^3 / c_P^2,
//                                                  R  mu (2, 3, 3, -12 ir^2) ir^3 / c_S^2,
//       S  mu (-6, -6, -6, 30 ir^2) ir^5,          S  minus P's.
// Evaluating the kernel at every level (thread per vertex) was bound by FP64 latency, most of
// it at levels past both fronts, where the second difference vanishes: 16 points
// x 4 times on the 448-triangle bar 2.62 -> 0.17 ms.  Of the 3 blocks an SM that
// the registers allow, shared memory (76 864 bytes a block, the bins sized for
// kBinChunk node pairs) admits 2.
constexpr int kPPWarps = 4, kPPSlices = 64, kPPNodes = 128, kPPNode = 8;

inline __host__ __device__ size_t pp_warp_bytes() {
    return (size_t)(kPPNode * kPPNodes + 9 * kPPSlices) * sizeof(double) + (front_bins_bytes(kPPSlices + 3) + 15) / 16 * 16;
}

// Bin (bin_window(c0, .) of the centres from c0 on) of the first level j with
// t_k - r / c > 0, t_k = t - k dt, k = nhat + 1 - j, as the reference tests it.
__device__ __forceinline__ unsigned pp_front_bin(double r2, double r, double c, double ic, double t, double dt, double idt,
                                                 int nhat, const BinWindow& w) {
    const double g = (t - r * ic) * idt;               // levels k < g are past the arrival
    if (!(g > -1.0)) return kNoBin;
    int k = (int)ceil(g) - 1;
    if (fabs(g - rint(g)) <= 1e-9 * (t * idt) + 1e-12) {
        const double tX = sqrt(r2) / c;
        for (k += 3; k >= 0; k--) {
            if (t - level_time(k, dt) - tX > 0) break;
        }
    }
    if (k < 0) return kNoBin;
    const int j = nhat + 1 - k;
    return j > w.kbase + w.bins - 2 ? kNoBin : j < w.kbase ? 0u : (unsigned)(j - w.kbase + 1);
}

__global__ void __launch_bounds__(32 * kPPWarps, 3) pp_p_kernel(PPArgs A, int nz) {
    extern __shared__ __align__(16) unsigned char pp_smem[];
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    double* nodes = reinterpret_cast<double*>(pp_smem + (threadIdx.x >> 5) * pp_warp_bytes());
    double* acc = nodes + kPPNode * kPPNodes;          // 9 per centre
    FrontBins B = front_bins_at(reinterpret_cast<unsigned char*>(acc + 9 * kPPSlices), kPPSlices + 3);
    const double cP = A.p.cP, cS = A.p.cS, icP = 1 / cP, icS = 1 / cS, dt = A.dt, idt = 1 / dt, dt2 = dt * dt;
    const double lam = A.p.lam, mu = A.p.mu, ic4 = 1 / (4 * kPi * A.p.rho * A.dt);
    const int n_in = A.n_sub * A.n_sing;
    for (long long w0 = warp; w0 < (long long)A.npts * A.ntimes * A.Nv * nz; w0 += nwarps) {
        const int z = (int)(w0 % nz), s = (int)(w0 / nz % A.Nv), ev = (int)(w0 / nz / A.Nv);
        const int q = ev / A.npts, ip = ev % A.npts;
        const double t = A.times[q];
        const double src[3] = {A.pts[3 * ip], A.pts[3 * ip + 1], A.pts[3 * ip + 2]};
        const int nhat = (t > 0) ? (int)ceil(t / A.dt) : 0;
        const int c0 = z * kPPSlices + 1, nc = min(kPPSlices, nhat + 1 - c0);      // centres c0 .. c0 + nc - 1
        if (nc <= 0) continue;
        const BinWindow win = bin_window(c0, nc);
        const int e0 = A.vt_off[s], n_all = (A.vt_off[s + 1] - e0) * n_in;
        __syncwarp();
        for (int i = lane; i < 9 * nc; i += 32) acc[i] = 0.0;
        for (int q0 = 0; q0 < n_all; q0 += kPPNodes) {
            const int n = min(kPPNodes, n_all - q0);
            bool met = false, late = false;
            __syncwarp();
            for (int i = lane; i < n; i += 32) {
                const int e = (q0 + i) / n_in, qi = (q0 + i) - e * n_in;
                const int m = A.vt_tri[e0 + e], kv = local_index(A.tris, m, s) - 1;
                const DirTri& F = A.tri[m];
                double y[3], *d = nodes + kPPNode * i;
                bary_point(y, A.pn + 3 * qi, F.V);
                const double phik = F.v[kv] + F.M[3 * kv] * y[0] + F.M[3 * kv + 1] * y[1] + F.M[3 * kv + 2] * y[2];
                double r2 = 0.0;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    d[c] = src[c] - y[c];
                    d[3 + c] = F.n[c];
                }
                d[6] = A.pw[qi % A.n_sing] * F.area * phik;
                r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
                const double r = q_sqrt(r2);
                unsigned bP = pp_front_bin(r2, r, cP, icP, t, dt, idt, nhat, win);
                unsigned bS = pp_front_bin(r2, r, cS, icS, t, dt, idt, nhat, win);
                if (bS == 0 && r2 > 0) bP = bS = kNoBin;          // past both fronts before the window: nothing left
                else late = late || bS == kNoBin;
                met = met || bP != kNoBin;
                B.bin[i] = make_ushort2((unsigned short)bP, (unsigned short)bS);
            }
            if (!__any_sync(0xffffffffu, met)) continue;
            late = __any_sync(0xffffffffu, late);
            const int total = bins_sort(B, n, win.bins, lane);
            double cur[9] = {0}, nxt[9] = {0}, run[9] = {0};
            double last = 0.0, last9 = 0.0;           // this lane's reduced entry and entry 33 of run
            int first = 0, idle = 0;                  // idle: bins without items up to this one
            for (int b = 0; b < win.bins; b++) {
                const int k = win.kbase + b - 1, c = k - 1, lastitem = B.off[b], items = lastitem - first;
                if (items == 0 && first == 0) continue;                 // before the first arrival
                if (c >= c0 + nc) break;
                idle = items ? 0 : idle + 1;
                const double early = b == 0 ? 0.0 : 1.0;                // bin 0: the linear part only
                const double tk = t - (nhat + 1 - k) * dt, tc = t - (nhat + 1 - c) * dt;
                const double f1 = dt2 * tc, f2 = dt2 * tk;
                for (int i = first + lane; i < lastitem; i += 32) {
                    const unsigned it = B.list[i];
                    const bool isS = it >> 31;
                    const double* d = nodes + kPPNode * (int)(it & 0x7fffffffu);
                    const double x[3] = {d[0], d[1], d[2]}, nn[3] = {d[3], d[4], d[5]}, w = d[6];
                    const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2], r = q_sqrt(r2), ir = q_rcp(r);
                    const double xn = x[0] * nn[0] + x[1] * nn[1] + x[2] * nn[2];
                    const double ic = isS ? icS : icP, tX = r * ic, ir2 = ir * ir;
                    const double h = early * (w * ic * ic * ic * ir2), g = early * (w * ic * ic * ir2 * ir);
                    // coefficients of x_i n_j, x_j n_i, xn delta_ij, xn x_i x_j
                    const double H[4] = {isS ? 0.0 : lam * h, isS ? mu * h : 0.0, isS ? mu * h : 0.0,
                                         (isS ? -2 * mu : 2 * mu) * h * ir2};
                    const double R[4] = {(isS ? 2 * mu : lam - 2 * mu) * g, (isS ? 3 * mu : -2 * mu) * g,
                                         (isS ? 3 * mu : -2 * mu) * g, (isS ? -12 * mu : 12 * mu) * g * ir2};
                    const double sc = (isS ? 6 * mu : -6 * mu) * w * ir2 * ir2 * ir, sx = -5 * sc * ir2;
                    const double a0 = tk - tX, a1 = a0 + dt;
                    const double S0 = a0 * a0 * (a0 + 3 * tX) * (1.0 / 6), S1 = a1 * a1 * (a1 + 3 * tX) * (1.0 / 6);
                    const double g1 = early * (S0 - f1), g2 = early * (S1 - 2 * S0 - f2);
                    double p1[4], p2[4];
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        const double sm = m == 3 ? sx : sc;
                        p1[m] = H[m] + a0 * R[m] + g1 * sm;
                        p2[m] = (dt - a0) * R[m] - H[m] + g2 * sm;
                    }
#pragma unroll
                    for (int i = 0; i < 3; i++)
#pragma unroll
                        for (int j = 0; j < 3; j++) {
                            const double a = x[i] * nn[j], bb = x[j] * nn[i], xx = xn * x[i] * x[j], dd = i == j ? xn : 0.0;
                            cur[3 * i + j] += p1[0] * a + p1[1] * bb + p1[2] * dd + p1[3] * xx;
                            nxt[3 * i + j] += p2[0] * a + p2[1] * bb + p2[2] * dd + p2[3] * xx;
                            run[3 * i + j] += sc * (a + bb + dd) + sx * xx;
                        }
                }
                if (b > 0 && c >= c0) {
                    // idle: run is the sum of the slice before, and all there is from the third slice on
                    const bool all = idle < 2;
                    if (all || idle == 2 || c == c0) {
                        double v[8];
#pragma unroll
                        for (int e = 0; e < 8; e++) v[e] = all ? cur[e] + f1 * run[e] : run[e];
                        last = warp_reduce_scatter8(v, lane);
                        last9 = all ? cur[8] + f1 * run[8] : run[8];
                        for (int off = 16; off > 0; off >>= 1) last9 += __shfl_xor_sync(0xffffffffu, last9, off);
                    }
                    double* a = acc + 9 * (c - c0);
                    if ((lane & 3) == 0) a[scatter8_entry(lane)] += all ? last : f1 * last;
                    if (lane == 1) a[8] += all ? last9 : f1 * last9;
                }
                first = lastitem;
#pragma unroll
                for (int e = 0; e < 9; e++) {
                    cur[e] = nxt[e];
                    nxt[e] = 0.0;
                }
                if (!late && first == total && items == 0) break;       // every node is past both fronts
            }
        }
        __syncwarp();
        double u[3] = {0.0, 0.0, 0.0};
        for (int i = lane; i < 3 * nc; i += 32) {      // column j of slice n
            const int c = i / 3, j = i - 3 * c, n = nhat + 1 - (c0 + c);
            double S[3];
#pragma unroll
            for (int r = 0; r < 3; r++) {
                const double v = acc[9 * c + 3 * r + j];
                S[r] = (fabs(v) > 1.0e-14) ? v * ic4 : 0.0;
            }
            if (A.mode == 1) {
                const size_t R = 3 * (size_t)nhat;
#pragma unroll
                for (int r = 0; r < 3; r++) A.Pm[(3 * (size_t)s + j) * R + 3 * (size_t)(n - 1) + r] = S[r];
            } else if (n <= A.nT) {
                const double bn = A.b[(size_t)(n - 1) * 3 * A.Nv + 3 * (size_t)s + j];
#pragma unroll
                for (int r = 0; r < 3; r++) u[r] -= S[r] * bn;
            }
        }
        if (A.mode == 0) warp_add3(A.u + 3 * (size_t)ev, u[0], u[1], u[2]);
    }
}

int launch_pp_dir(const MeshData& m, const PhysParams& P, int n_sub, int n_sing, int fix, const double* d_pts, int npts,
                  const double* h_times, int ntimes, const double* d_a, const double* d_b, double* d_u, double* d_G,
                  double* d_P, int mode, cudaStream_t s) {
    const int gstride = fix ? n_sing : 3;
    if (3 * (n_sub - 1) + n_sing > n_sub * n_sing && !fix)
        return fail(EBEM_ERR_INVALID, "the reference's node stride 3 needs n_sing >= 3 (or the fixed stride)");
    if ((long long)npts * ntimes > 65535)
        return fail(EBEM_ERR_INVALID, "at most 65535 (point, time) evaluations per call");
    Tables T;
    if (int rc = upload_tables(T, 0, n_sub, n_sing, 0, s)) return rc;
    double* d_times = nullptr;
    EBEM_CUDA_TRY(ws_malloc(&d_times, sizeof(double) * ntimes, s));
    cudaError_t e = cudaMemcpyAsync(d_times, h_times, sizeof(double) * ntimes, cudaMemcpyHostToDevice, s);
    PPArgs A;
    A.tri = m.d_dir;
    A.tris = m.d_tris;
    A.vt_off = m.d_vt_off;
    A.vt_tri = m.d_vt_tri;
    A.pn = T.d + T.inner;
    A.pw = T.d + T.win;
    A.n_sub = n_sub;
    A.n_sing = n_sing;
    A.gstride = gstride;
    A.N = m.nt;
    A.Nv = m.nv;
    A.p = mat_of(P);
    A.dt = P.dt;
    A.pts = d_pts;
    A.times = d_times;
    A.npts = npts;
    A.ntimes = ntimes;
    A.nT = P.nT;
    A.a = d_a;
    A.b = d_b;
    A.u = d_u;
    A.G = d_G;
    A.Pm = d_P;
    A.mode = mode;
    if (e == cudaSuccess) {
        // slices split into chunks over grid z so that about 8 blocks per SM
        // run (G; a chunk re-evaluates 1 boundary level: at least 4 slices
        // per chunk keep that under a quarter)
        int nhat_max = 0;
        for (int q = 0; q < ntimes; q++)
            if (h_times[q] > 0) nhat_max = std::max(nhat_max, (int)std::ceil(h_times[q] / P.dt));
        nhat_max = std::max(nhat_max, 1);
        int sms = 148;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m.device);
        const long long evs = (long long)npts * ntimes, target = 8LL * sms;
        auto chunk_of = [&](long long bxy, int kmin) {
            const long long want = (nhat_max * bxy + target - 1) / target;
            return (int)std::min<long long>(nhat_max, std::max<long long>(kmin, want));
        };
        const long long bg = (m.nt + 127) / 128;
        const int kg = chunk_of(bg * evs, 4), nz = (nhat_max + kPPSlices - 1) / kPPSlices;
        dim3 gg((unsigned)bg, (unsigned)evs, (unsigned)((nhat_max + kg - 1) / kg));
        const long long gp = std::min<long long>((evs * m.nv * nz + kPPWarps - 1) / kPPWarps, 64LL * sms);
        if (mode == 0) e = cudaMemsetAsync(d_u, 0, sizeof(double) * 3 * (size_t)npts * ntimes, s);
        if (e == cudaSuccess) {
            pp_g_kernel<<<gg, 128, 0, s>>>(A, kg);
            const size_t smem = kPPWarps * pp_warp_bytes();
            e = cudaFuncSetAttribute(pp_p_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e == cudaSuccess) {
                pp_p_kernel<<<(unsigned)gp, 32 * kPPWarps, smem, s>>>(A, nz);
                e = cudaGetLastError();
            }
        }
    }
    ws_free(d_times, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail(EBEM_ERR_CUDA, std::string("direct post-processing: ") + cudaGetErrorString(e));
    return EBEM_OK;
}

// ---------------------------------------------------------------------------
// time marching

// y += I_Gamma u: (3x+i) += area_x / 6 u(3s+i) for each vertex s of x
// (BEMenerg_dir_timeMarchingN.m:275, kron((indSM > 0) .* area / 6, eye(3))).
__global__ void mass_apply_kernel(const DirTri* __restrict__ tri, const int32_t* __restrict__ tris, int N,
                                  const double* __restrict__ u, double* __restrict__ y) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= N) return;
    const double c = tri[x].area / 6;
    for (int i = 0; i < 3; i++) {
        double acc = 0.0;
        for (int k = 0; k < 3; k++) acc += u[3 * tris[3 * x + k] + i];
        y[3 * x + i] += c * acc;
    }
}

// A += I_Gamma (A: 3N x 3Nv column-major).
__global__ void mass_add_kernel(const DirTri* __restrict__ tri, const int32_t* __restrict__ tris, int N,
                                double* __restrict__ A) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= N) return;
    const double c = tri[x].area / 6;
    const size_t ld = 3 * (size_t)N;
    for (int k = 0; k < 3; k++) {
        const int s = tris[3 * x + k];
        for (int i = 0; i < 3; i++) A[(3 * (size_t)s + i) * ld + 3 * (size_t)x + i] += c;
    }
}

__global__ void copy_cols_rev_kernel(const double* __restrict__ src, double* __restrict__ dst, int n, int nT, int to_rev) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)n * nT) return;
    const int r = (int)(idx % n), c = (int)(idx / n);
    if (to_rev) dst[(size_t)(nT - 1 - c) * n + r] = src[idx];
    else dst[idx] = src[(size_t)(nT - 1 - c) * n + r];
}

// beta (rows x nT) += sum_l B_l * shift(g, l), B_l rows x cols per lag.
static int beta_gemm(cublasHandle_t hb, const double* dB, int L, int rows, int cols, const double* dg, int nT,
                     double* dbeta) {
    const double one = 1.0;
    for (int l = 0; l < L && l < nT; l++) {
        const double* Bl = dB + (size_t)l * rows * cols;
        cublasStatus_t st = cublasDgemm(hb, CUBLAS_OP_N, CUBLAS_OP_N, rows, nT - l, cols, &one, Bl, rows, dg, cols, &one,
                                        dbeta + (size_t)l * rows, rows);
        if (st != CUBLAS_STATUS_SUCCESS) return fail(EBEM_ERR_CUDA, "cublasDgemm failed in the data convolution");
    }
    return EBEM_OK;
}

int march_dn_device(const MeshData& m, const double* dV, int LV, const double* dK, int LK, const double* d_gV, int nT,
                    double* d_u, cudaStream_t s) {
    const int R = 3 * m.nt, Cn = 3 * m.nv;
    if (R < Cn) return fail(EBEM_ERR_INVALID, "least-squares system needs 3N >= 3Nv");
    int rc = EBEM_OK, dev = 0, sms = 148, lwork = 0, lw2 = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cusolverDnHandle_t hs = nullptr;
    cublasHandle_t hb = nullptr;
    double *A = nullptr, *Q = nullptr, *X = nullptr, *tau = nullptr, *work = nullptr, *beta = nullptr, *rev = nullptr;
    int* info = nullptr;
    const double one = 1.0, zero = 0.0;
    auto cu = [&](cudaError_t e, const char* what) {
        if (e != cudaSuccess && rc == EBEM_OK) rc = fail(EBEM_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
        return rc == EBEM_OK;
    };
    auto blas_ok = [&](cublasStatus_t st, const char* what) {
        if (st != CUBLAS_STATUS_SUCCESS && rc == EBEM_OK)
            rc = fail(EBEM_ERR_CUDA, std::string(what) + " failed (cuBLAS status " + std::to_string((int)st) + ")");
        return rc == EBEM_OK;
    };
    auto sol_ok = [&](cusolverStatus_t st, const char* what) {
        if (st != CUSOLVER_STATUS_SUCCESS && rc == EBEM_OK)
            rc = fail(EBEM_ERR_CUDA, std::string(what) + " failed (cuSOLVER status " + std::to_string((int)st) + ")");
        return rc == EBEM_OK;
    };
    const size_t RC = (size_t)R * Cn;
    if (!cu(ws_malloc(&A, sizeof(double) * RC, s), "alloc") || !cu(ws_malloc(&Q, sizeof(double) * RC, s), "alloc") ||
        !cu(ws_malloc(&X, sizeof(double) * RC, s), "alloc") || !cu(ws_malloc(&tau, sizeof(double) * Cn, s), "alloc") ||
        !cu(ws_malloc(&beta, sizeof(double) * (size_t)R * nT, s), "alloc") ||
        !cu(ws_malloc(&rev, sizeof(double) * (size_t)Cn * nT, s), "alloc") ||
        !cu(ws_malloc(&info, sizeof(int), s), "alloc")) {
        rc = fail(EBEM_ERR_NOMEM, "direct time-marching workspace allocation failed");
        goto done;
    }
    if ((rc = solver_handle(s, &hs)) || (rc = blas_handle(s, &hb))) goto done;
    // beta_V,n = sum_j V_{n-j} g_j
    if (!cu(cudaMemsetAsync(beta, 0, sizeof(double) * (size_t)R * nT, s), "memset")) goto done;
    if ((rc = beta_gemm(hb, dV, LV, R, R, d_gV, nT, beta))) goto done;
    // A = K_0 + I_Gamma = Q_1 R_1 (thin QR, once); the least-squares solution
    // of every step is u = X y with X = R_1^{-1} Q_1^T (Cn x R), formed once
    // (the reference solves (K_0 + I_Gamma) \ y densely at every step)
    if (!cu(cudaMemcpyAsync(A, dK, sizeof(double) * RC, cudaMemcpyDeviceToDevice, s), "copy")) goto done;
    mass_add_kernel<<<(m.nt + 127) / 128, 128, 0, s>>>(m.d_dir, m.d_tris, m.nt, A);
    if (!cu(cudaGetLastError(), "mass matrix")) goto done;
    if (!sol_ok(cusolverDnDgeqrf_bufferSize(hs, R, Cn, A, R, &lwork), "QR workspace query") ||
        !sol_ok(cusolverDnDorgqr_bufferSize(hs, R, Cn, Cn, A, R, tau, &lw2), "Q workspace query"))
        goto done;
    lwork = std::max(lwork, lw2);
    if (!cu(ws_malloc(&work, sizeof(double) * (size_t)std::max(lwork, 1), s), "alloc")) goto done;
    if (!sol_ok(cusolverDnDgeqrf(hs, R, Cn, A, R, tau, work, lwork, info), "QR factorisation")) goto done;
    if (!cu(cudaMemcpyAsync(Q, A, sizeof(double) * RC, cudaMemcpyDeviceToDevice, s), "copy")) goto done;
    if (!sol_ok(cusolverDnDorgqr(hs, R, Cn, Cn, Q, R, tau, work, lwork, info), "forming Q_1")) goto done;
    // X = Q_1^T (transpose; X zeroed first although geam reads no B when
    // beta = 0), then R_1 X = Q_1^T in place
    if (!cu(cudaMemsetAsync(X, 0, sizeof(double) * RC, s), "memset")) goto done;
    if (!blas_ok(cublasDgeam(hb, CUBLAS_OP_T, CUBLAS_OP_N, Cn, R, &one, Q, R, &zero, X, Cn, X, Cn), "transpose"))
        goto done;
    if (!blas_ok(cublasDtrsm(hb, CUBLAS_SIDE_LEFT, CUBLAS_FILL_MODE_UPPER, CUBLAS_OP_N, CUBLAS_DIAG_NON_UNIT, Cn, R, &one,
                             A, R, X, Cn),
                 "triangular solve for X"))
        goto done;
    // u in reversed time order: u_n at column nT-1-n
    if (!cu(cudaMemsetAsync(rev, 0, sizeof(double) * (size_t)Cn * nT, s), "memset")) goto done;
    // steps in blocks of kHistBlock, as march_device: beta's columns collect the
    // right-hand sides
    for (int n = 0; n < nT; n++) {
        const int i = n % kHistBlock, M = std::min(i, LK - 1);          // K_1 .. K_M inside the block
        double *un = rev + (size_t)(nT - 1 - n) * Cn, *y = beta + (size_t)n * R;
        if (i == 0 && (rc = launch_hist_block(dK + RC, R, Cn, LK - 1, rev, nT, n, beta, sms, s))) goto done;
        if (n > 0) {
            mass_apply_kernel<<<(m.nt + 127) / 128, 128, 0, s>>>(m.d_dir, m.d_tris, m.nt, un + Cn, y);
            if (!cu(cudaGetLastError(), "mass apply")) goto done;
        }
        if (M > 0 && (rc = launch_hist_gemv(dK + RC, R, (long long)Cn * M, un + Cn, y, sms, s))) goto done;
        if ((rc = launch_gemv_add(X, Cn, R, y, un, sms, s))) goto done;
    }
    {
        const long long tot = (long long)Cn * nT;
        copy_cols_rev_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(rev, d_u, Cn, nT, 0);
        cu(cudaGetLastError(), "copy");
    }
    cu(cudaStreamSynchronize(s), "direct time marching");
done:
    ws_free(A, s); ws_free(Q, s); ws_free(X, s); ws_free(tau, s); ws_free(work, s); ws_free(beta, s); ws_free(rev, s);
    ws_free(info, s);
    return rc;
}

__global__ void half_add_kernel(const double* __restrict__ rhs, double* __restrict__ out, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] += rhs[i] / 2;
}

int march_dd_device(const MeshData& m, const double* dV, int LV, const double* dK, int LK, const double* d_rhs,
                    const double* d_gK, int nT, double* d_phi, cudaStream_t s) {
    const int R = 3 * m.nt, Cn = 3 * m.nv;
    double* b = nullptr;
    cublasHandle_t hb = nullptr;
    int rc = EBEM_OK;
    if (int e = blas_handle(s, &hb)) return e;
    if (ws_malloc(&b, sizeof(double) * (size_t)R * nT, s) != cudaSuccess)
        return fail(EBEM_ERR_NOMEM, "right-hand side allocation failed");
    // b = rhs / 2 + beta_K, beta_K,n = sum_j K_{n-j} gK_j
    if (cudaMemsetAsync(b, 0, sizeof(double) * (size_t)R * nT, s) != cudaSuccess) rc = fail(EBEM_ERR_CUDA, "memset failed");
    if (!rc) rc = beta_gemm(hb, dK, LK, R, Cn, d_gK, nT, b);
    if (!rc) {
        const long long n = (long long)R * nT;
        half_add_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d_rhs, b, n);
        if (cudaGetLastError() != cudaSuccess) rc = fail(EBEM_ERR_CUDA, "rhs combination failed");
    }
    if (!rc) rc = march_device(dV, R, LV, b, nT, d_phi, s);
    cudaStreamSynchronize(s);
    ws_free(b, s);
    return rc;
}

}  // namespace ebem
