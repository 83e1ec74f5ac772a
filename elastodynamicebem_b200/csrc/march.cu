// Right-hand side, time marching and post-processing on the device.
//
// Reference (paths relative to the reference project root;
// "CORE/" = functions/BEMenerg_indir/BEMenerg_core/):
//   right-hand side   CORE/BEMenerg_core_calcTn/BEMenerg_core_calcTnBlock.m:28-58,
//                     CORE/BEMenerg_core_calcTn/BEMenerg_core_calcNucleoTn.m:196-244
//   time marching     CORE/BEMenerg_coreGPU/BEMenerg_coreGPU_timeMarching.m:151-169
//                     (LU of E_0 once; phi_n = E_0^{-1}(b_n - sum_l E_l phi_{n-l}))
//   post-processing   functions/BEMenerg_indir/BEMenerg_postProc/BEMenerg_postProcA/
//                     BEMenerg_postProcA_singlePoint.m:21-61, _calcMatrix.m, _calcMatrixBlock.m
#include "ebem_internal.h"
#include "sa_group.cuh"

#include <cublas_v2.h>
#include <cusolverDn.h>

#include <algorithm>
#include <cmath>

namespace ebem {

// ---------------------------------------------------------------------------
// Dirichlet data g(x, t).  Ids 2..7 are the reference's cases
// (BEMenerg_core_calcNucleoTn.m:199-237); 0 and 1 are the data of the screen
// and sphere benchmark problems.
__device__ void datum_value(int id, double velP, double Tfin, const double x[3], double t, double g[3]) {
    g[0] = g[1] = g[2] = 0.0;
    switch (id) {
    case 0: g[2] = t * t * t * t * exp(-2 * t); break;
    case 1: {
        double s = (t > 0) ? sin(2 * kPi * t) : 0.0;
        g[0] = x[0] * s; g[1] = x[1] * s; g[2] = x[2] * s;
    } break;
    case 2: g[2] = 0.5 * t; break;
    case 3: {
        double f = 1.0;
        if (t < kPi / 2) { double s = sin(t); f = s * s * s * s * s; }
        g[2] = f * (x[0] * x[0]);
    } break;
    case 4: case 5: {
        double h = (id == 4) ? 1.0 : 3.0;
        int hat_k = (int)ceil((velP * Tfin) / (2 * h)) - 1;
        double s = 0.0;
        for (int k = 0; k <= hat_k; k++) {
            double a1 = velP * t - 2 * h * k - (h - x[2]);
            double a2 = velP * t - 2 * h * (k + 1) + (h - x[2]);
            double term = a1 * (a1 > 0) - a2 * (a2 > 0);
            s += ((k & 1) ? -1.0 : 1.0) * term;
        }
        g[2] = s;
    } break;
    case 6: { double u = x[0] - 2 + velP * t - 0.475; g[0] = -exp(-20 * u * u); } break;
    case 7: { double u = x[2] + 1 - velP * t; g[2] = -exp(-20 * u * u); } break;
    default: break;
    }
}

__global__ void rhs_kernel(const NodeW* __restrict__ nodes, int N, int n_gh, int datum, double dt, int nT,
                           double velP, double Tfin, double* __restrict__ rhs) {
    long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)N * nT) return;
    int t = (int)(idx % N), n = (int)(idx / N);
    double t0 = dt * n, t1 = dt * (n + 1);
    double ris[3] = {0, 0, 0};
    for (int g = 0; g < n_gh; g++) {
        NodeW p = nodes[(size_t)t * n_gh + g];
        double x[3] = {p.x, p.y, p.z}, g1[3], g0[3];
        datum_value(datum, velP, Tfin, x, t1, g1);
        datum_value(datum, velP, Tfin, x, t0, g0);
        for (int c = 0; c < 3; c++) ris[c] = ris[c] + (g1[c] - g0[c]) * p.w;
    }
    for (int c = 0; c < 3; c++) rhs[(size_t)n * 3 * N + 3 * t + c] = (fabs(ris[c]) < 1.0e-14) ? 0.0 : ris[c];
}

// ---------------------------------------------------------------------------
// Datum 8, the reference's manufactured case 'TEST'
// (BEMenerg_core_calcNucleoTn.m:13-132): the boundary value on the screen
// [-1, 1]^2 (z = 0) whose solution is the constant density (1, 1, 1).  The
// reference integrates nucl_1..3 over the square with integral2 for each pair
// of instants (BEMenerg_core_TnTest_classic.m:11-13).  Regrouped by instant,
// nucl_c = f_c(t1) - f_c(t0) with (r = |y - x|, c, s the direction cosines)
//   f_1 = A c^2 + B (3 c^2 - 1) + S + c s (A + 3 B),
//   f_2 = A s^2 + B (3 s^2 - 1) + S + c s (A + 3 B),   f_3 = S - B,
//   A = J_P - J_S, B = I_P - I_S, S = J_S, J_v = H(t - r/v)/(v^2 r),
//   I_v = H(t - r/v)(t^2 - r^2/v^2)/(2 r^3),
// so F_c(x, t) = int f_c(t) dy / (4 pi rho) is computed per instant and the
// right-hand side takes F(t1) - F(t0).  In polar coordinates about x the
// radial integrals are closed forms (a = min(R, c_S t), b = min(R, c_P t)):
//   int_0^R r A = b/c_P^2 - a/c_S^2,   int_0^R r S = a/c_S^2,
//   int_0^R r B = (1/c_S^2 - 1/c_P^2) a/2 + t^2/2 (1/a - 1/b) - (b - a)/(2 c_P^2),
// and the angle is integrated along each side of the square: with d the
// distance of x from the side's line and u the signed position along it from
// the foot of the perpendicular, R = sqrt(d^2 + u^2) and dtheta = d du / R^2.
// The u-range is cut at the foot, at +-d 2^j (geometric grading: the
// integrand's singularities sit at u = +-i d) and where r = c_S t or r = c_P t
// crosses the side; 16-point Gauss-Legendre on each piece.
__constant__ double c_gl16[2][16];      // 16-point Gauss-Legendre on (-1, 1): nodes, weights
constexpr int kTestCuts = 64;

__device__ void test_level(double x1, double x2, double t, double cP, double cS, double F[3]) {
    F[0] = F[1] = F[2] = 0.0;
    if (t <= 0) return;
    const double iP2 = 1 / (cP * cP), iS2 = 1 / (cS * cS), rS = cS * t, rP = cP * t;
    const double cx[4] = {-1, 1, 1, -1}, cy[4] = {-1, -1, 1, 1};
    for (int k = 0; k < 4; k++) {
        const double ax = cx[k] - x1, ay = cy[k] - x2;                 // corner k - x; the side runs to corner k+1
        const double ex = 0.5 * (cx[(k + 1) & 3] - cx[k]), ey = 0.5 * (cy[(k + 1) & 3] - cy[k]);   // unit, length 2
        const double s0 = -(ax * ex + ay * ey);                         // foot at corner + s0 e
        const double fx = ax + s0 * ex, fy = ay + s0 * ey;              // foot - x, perpendicular to e
        const double d = fx * ey - fy * ex;                             // > 0: the square runs counterclockwise about x
        const double ulo = -s0, uhi = 2 - s0;
        double cut[kTestCuts];
        int nc = 0;
        auto add = [&](double u) {
            if (u > ulo && u < uhi && nc < kTestCuts - 1) cut[nc++] = u;
        };
        cut[nc++] = ulo;
        add(0.0);
        for (int q = 0; q < 2; q++) {
            const double rho = q ? rP : rS;
            if (rho > d) {
                const double w = sqrt((rho - d) * (rho + d));
                add(-w);
                add(w);
            }
        }
        const double umax = fmax(-ulo, uhi);
        for (int j = 0; j < 26 && d * (double)(1 << j) < umax; j++) {
            add(-d * (double)(1 << j));
            add(d * (double)(1 << j));
        }
        cut[nc++] = uhi;
        for (int i = 1; i < nc; i++)                                   // insertion sort
            for (int j = i; j > 0 && cut[j] < cut[j - 1]; j--) {
                const double tmp = cut[j];
                cut[j] = cut[j - 1];
                cut[j - 1] = tmp;
            }
        for (int q = 0; q + 1 < nc; q++) {
            const double h = 0.5 * (cut[q + 1] - cut[q]), mid = 0.5 * (cut[q + 1] + cut[q]);
            if (h <= 0) continue;
            for (int ia = 0; ia < 16; ia++) {
                const double u = mid + h * c_gl16[0][ia];
                const double R2 = d * d + u * u, R = sqrt(R2);
                const double w = h * c_gl16[1][ia] * d / R2;           // dtheta
                const double cs = (fx + u * ex) / R, sn = (fy + u * ey) / R;
                const double a = fmin(R, rS), b = fmin(R, rP);
                const double RS = a * iS2, RA = b * iP2 - a * iS2;
                double RB = 0.5 * (iS2 - iP2) * a;
                if (b > a) RB += 0.5 * t * t * (1 / a - 1 / b) - 0.5 * (b - a) * iP2;
                const double mixd = cs * sn * (RA + 3 * RB);
                F[0] += w * (cs * cs * RA + (3 * cs * cs - 1) * RB + RS + mixd);
                F[1] += w * (sn * sn * RA + (3 * sn * sn - 1) * RB + RS + mixd);
                F[2] += w * (RS - RB);
            }
        }
    }
}

// S_k[t] = sum_g w_g F(x_g, t_k) / (4 pi rho), k = 0..nT, one thread per (triangle, level).
__global__ void rhs_test_level_kernel(const NodeW* __restrict__ nodes, int N, int n_gh, double dt, int nT, double cP,
                                      double cS, double c4pirho, double* __restrict__ S) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)N * (nT + 1)) return;
    const int t = (int)(idx % N), k = (int)(idx / N);
    double acc[3] = {0, 0, 0};
    for (int g = 0; g < n_gh; g++) {
        const NodeW p = nodes[(size_t)t * n_gh + g];
        double F[3];
        test_level(p.x, p.y, dt * k, cP, cS, F);
        for (int c = 0; c < 3; c++) acc[c] += F[c] * p.w;
    }
    for (int c = 0; c < 3; c++) S[((size_t)k * N + t) * 3 + c] = acc[c] / c4pirho;
}

// b_n = S_{n+1} - S_n, entries below 1e-14 set to 0 (BEMenerg_core_calcTnBlock.m:50-51).
__global__ void rhs_test_diff_kernel(const double* __restrict__ S, int N, int nT, double* __restrict__ rhs) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= 3LL * N * nT) return;
    const int n = (int)(idx / (3LL * N));
    const size_t e = (size_t)(idx % (3LL * N));
    const double v = S[(size_t)(n + 1) * 3 * N + e] - S[(size_t)n * 3 * N + e];
    rhs[idx] = (fabs(v) < 1.0e-14) ? 0.0 : v;
}

static void gauss_legendre16(double x[16], double w[16]) {
    // Newton's iteration on P_16 from cos(pi (i + 3/4) / (n + 1/2)).
    const int n = 16;
    for (int i = 0; i < n; i++) {
        double z = cos(kPi * (i + 0.75) / (n + 0.5)), dp = 1;
        for (int it = 0; it < 100; it++) {
            double p0 = 1, p1 = z;
            for (int k = 2; k <= n; k++) {
                const double p2 = ((2 * k - 1) * z * p1 - (k - 1) * p0) / k;
                p0 = p1;
                p1 = p2;
            }
            dp = n * (z * p1 - p0) / (z * z - 1);
            const double dz = p1 / dp;
            z -= dz;
            if (fabs(dz) < 1e-16) break;
        }
        x[i] = z;
        w[i] = 2 / ((1 - z * z) * dp * dp);
    }
}

static int launch_rhs_test(const MeshData& m, const PhysParams& P, int n_gh, double* d_rhs, cudaStream_t s) {
    double gl[2][16];
    gauss_legendre16(gl[0], gl[1]);
    EBEM_CUDA_TRY(cudaMemcpyToSymbolAsync(c_gl16, gl, sizeof gl, 0, cudaMemcpyHostToDevice, s));
    double* d_S = nullptr;
    const size_t nS = 3 * (size_t)m.nt * (P.nT + 1);
    EBEM_CUDA_TRY(ws_malloc(&d_S, nS * sizeof(double), s));
    const int threads = 128;
    const long long lv = (long long)m.nt * (P.nT + 1), nb = 3LL * m.nt * P.nT;
    rhs_test_level_kernel<<<(unsigned)((lv + threads - 1) / threads), threads, 0, s>>>(
        m.d_nodes, m.nt, n_gh, P.dt, P.nT, P.velP, P.velS, 4 * kPi * P.rho, d_S);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) {
        rhs_test_diff_kernel<<<(unsigned)((nb + threads - 1) / threads), threads, 0, s>>>(d_S, m.nt, P.nT, d_rhs);
        e = cudaGetLastError();
    }
    ws_free(d_S, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail(EBEM_ERR_CUDA, std::string("TEST right-hand side: ") + cudaGetErrorString(e));
    return EBEM_OK;
}

int launch_rhs(const MeshData& m, const PhysParams& P, int n_gh, int datum, double* d_rhs, cudaStream_t s) {
    if (datum == 8) return launch_rhs_test(m, P, n_gh, d_rhs, s);
    long long total = (long long)m.nt * P.nT;
    int threads = 128;
    rhs_kernel<<<(unsigned)((total + threads - 1) / threads), threads, 0, s>>>(m.d_nodes, m.nt, n_gh, datum, P.dt,
                                                                              P.nT, P.velP, P.dt * P.nT, d_rhs);
    EBEM_CUDA_TRY(cudaGetLastError());
    return EBEM_OK;
}

// ---------------------------------------------------------------------------
// Products with column-major matrices of the marching, HBM-bound: for B
// consecutive steps n0 .. n0 + B - 1 at once
//   Y_i += alpha sum_k A(:, k) x_i(k),   i < B,
// A = [E_1 E_2 ...] (rows x K, `cols` columns per lag) and x_i the density in
// reversed time order from step n0 + i - 1 back (contiguous: x_i = x0 - i
// cols), of which only steps 0 .. n0 - 1 count: columns k < i cols are step n0
// or later (zero in the reversed storage when the product runs), k >= kmax0 + i
// cols would be before step 0.  Each matrix is read once for B steps instead of
// once per step.  A product with such a zero adds nothing unless the matrix
// entry is an infinity or NaN, which must not reach a step before the first of
// its lag: a block whose sum for a step is not finite takes that sum again over
// the step's own columns.
// A block takes 64 rows and a range of columns, its 8 warps every eighth
// column (two 256-byte runs each, 16 loads in flight per lane), the x_i of 128
// columns at a time in shared memory; the warps' sums are added in shared
// memory and then to Y with one atomic per row, step and block.  (One block
// per 2048 rows left the second block of a 2100-row matrix 97 % idle: 3.9
// TB/s on the history of the 700-triangle prism, 48 steps of 2100 unknowns:
// 10.3 ms; now 1.1 ms for what precedes the blocks of 8 steps and 0.8 ms for
// the lags inside them.)
constexpr int kToepRows = 64, kToepCols = 128;

template <int B>
__global__ void __launch_bounds__(256, B > 4 ? 3 : 5)
toeplitz_kernel(const double* __restrict__ A, int rows, long long K, int cols, long long cols_per_block,
                const double* __restrict__ x0, long long kmax0, double alpha, double* __restrict__ Y, long long ldy) {
    __shared__ double xs[kToepCols * B];
    __shared__ double red[8][kToepRows];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int row0 = blockIdx.y * kToepRows;
    const int r0 = min(row0 + lane, rows - 1), r1 = min(row0 + lane + 32, rows - 1);
    const long long k0 = (long long)blockIdx.x * cols_per_block, k1 = min(k0 + cols_per_block, K);
    double acc[2][B];
#pragma unroll
    for (int i = 0; i < B; i++) acc[0][i] = acc[1][i] = 0.0;
    for (long long kk = k0; kk < k1; kk += kToepCols) {
        __syncthreads();
        for (int t = threadIdx.x; t < kToepCols * B; t += 256) {
            const int i = t / kToepCols, c = t - i * kToepCols;
            const long long k = kk + c;
            xs[c * B + i] = (k < k1 && k < kmax0 + (long long)i * cols) ? x0[k - (long long)i * cols] : 0.0;
        }
        __syncthreads();
#pragma unroll 1
        for (int h = 0; h < 2; h++) {
            double a[8][2];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                // columns past the range read its last one (their x is zero)
                const long long k = min(kk + w + 8 * (8 * h + j), k1 - 1);
                const double* col = A + k * (long long)rows;
                a[j][0] = __ldg(col + r0);
                a[j][1] = __ldg(col + r1);
            }
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const double* x = xs + (w + 8 * (8 * h + j)) * B;
#pragma unroll
                for (int i = 0; i < B; i++) {
                    acc[0][i] += a[j][0] * x[i];
                    acc[1][i] += a[j][1] * x[i];
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < B; i++) {
        __syncthreads();
        red[w][lane] = acc[0][i];
        red[w][lane + 32] = acc[1][i];
        __syncthreads();
        const bool out = threadIdx.x < kToepRows && row0 + (int)threadIdx.x < rows;
        auto total = [&]() {
            double v = 0.0;
#pragma unroll
            for (int q = 0; q < 8; q++) v += red[q][threadIdx.x];
            return v;
        };
        double v = out ? total() : 0.0;
        if (__syncthreads_or(!isfinite(v))) {
            const long long shift = (long long)i * cols, end = min(k1, kmax0 + shift);
            double s0 = 0.0, s1 = 0.0;
            for (long long k = max(k0, shift) + w; k < end; k += 8) {
                const double x = x0[k - shift];
                s0 += A[k * rows + r0] * x;
                s1 += A[k * rows + r1] * x;
            }
            red[w][lane] = s0;
            red[w][lane + 32] = s1;
            __syncthreads();
            if (out) v = total();
        }
        if (out && v != 0.0) atomicAdd(Y + i * ldy + row0 + threadIdx.x, alpha * v);
    }
}

template <int B>
static int launch_toeplitz(const double* A, int rows, long long K, int cols, const double* x0, long long kmax0, double alpha,
                           double* Y, long long ldy, int sm_count, cudaStream_t s) {
    if (K <= 0) return EBEM_OK;
    const int tiles = (rows + kToepRows - 1) / kToepRows;
    // about six blocks per SM, at least 128 columns each
    const long long want = std::max<long long>(1, (long long)sm_count * 6 / tiles);
    long long cpb = (K + want - 1) / want;
    cpb = (cpb + kToepCols - 1) / kToepCols * kToepCols;
    const dim3 grid((unsigned)((K + cpb - 1) / cpb), (unsigned)tiles);
    toeplitz_kernel<B><<<grid, 256, 0, s>>>(A, rows, K, cols, cpb, x0, kmax0, alpha, Y, ldy);
    EBEM_CUDA_TRY(cudaGetLastError());
    return EBEM_OK;
}

int launch_hist_gemv(const double* A, int rows, long long K, const double* x, double* y, int sm_count, cudaStream_t s) {
    return launch_toeplitz<1>(A, rows, K, 0, x, K, -1.0, y, 0, sm_count, s);
}

int launch_gemv_add(const double* A, int rows, int K, const double* x, double* y, int sm_count, cudaStream_t s) {
    return launch_toeplitz<1>(A, rows, K, 0, x, K, 1.0, y, 0, sm_count, s);
}

// Steps n0 .. n0 + kHistBlock - 1: Y(:, n0 + i) -= sum_l E_l phi_{n0 + i - l}
// over the steps before n0 (E1: first of M lags, rows x cols each; rev: cols x
// nT, step n at column nT - 1 - n, zero from step n0 on; Y: rows x nT).
int launch_hist_block(const double* E1, int rows, int cols, int M, const double* rev, int nT, int n0, double* Y, int sm_count,
                      cudaStream_t s) {
    const int nb = std::min(kHistBlock, nT - n0), lags = std::min(M, n0 + nb - 1);
    if (n0 <= 0 || lags <= 0) return EBEM_OK;
    const double* x0 = rev + (size_t)(nT - n0) * cols;
    const long long K = (long long)lags * cols, kmax0 = (long long)n0 * cols;
    double* y = Y + (size_t)n0 * rows;
    switch (nb) {
    case 1: return launch_toeplitz<1>(E1, rows, K, cols, x0, kmax0, -1.0, y, rows, sm_count, s);
    case 2: return launch_toeplitz<2>(E1, rows, K, cols, x0, kmax0, -1.0, y, rows, sm_count, s);
    case 3: return launch_toeplitz<3>(E1, rows, K, cols, x0, kmax0, -1.0, y, rows, sm_count, s);
    case 4: return launch_toeplitz<4>(E1, rows, K, cols, x0, kmax0, -1.0, y, rows, sm_count, s);
    case 5: return launch_toeplitz<5>(E1, rows, K, cols, x0, kmax0, -1.0, y, rows, sm_count, s);
    case 6: return launch_toeplitz<6>(E1, rows, K, cols, x0, kmax0, -1.0, y, rows, sm_count, s);
    case 7: return launch_toeplitz<7>(E1, rows, K, cols, x0, kmax0, -1.0, y, rows, sm_count, s);
    default: return launch_toeplitz<8>(E1, rows, K, cols, x0, kmax0, -1.0, y, rows, sm_count, s);
    }
}

// dst(:, n) = src(:, nT - 1 - n), n3 x nT.
__global__ void copy_reverse_kernel(const double* __restrict__ src, double* __restrict__ dst, int n3, int nT) {
    long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)n3 * nT) return;
    int r = (int)(idx % n3), n = (int)(idx / n3);
    dst[idx] = src[(size_t)(nT - 1 - n) * n3 + r];
}

#define CUSOLVER_TRY(expr)                                                                        \
    do {                                                                                          \
        cusolverStatus_t _st = (expr);                                                            \
        if (_st != CUSOLVER_STATUS_SUCCESS) {                                                     \
            rc = fail(EBEM_ERR_CUDA, std::string(#expr) + " failed with status " + std::to_string((int)_st)); \
            goto done;                                                                            \
        }                                                                                         \
    } while (0)

// ---------------------------------------------------------------------------
// Library handles per host thread and device.  A thread-local table of plain
// pointers: nothing is destroyed at thread or process exit (the driver
// reclaims the handles with the context), so no handle outlives its CUDA
// context in a destructor.
namespace {
constexpr int kHandleDevices = 64;
struct ThreadHandles {
    cusolverDnHandle_t sol[kHandleDevices];
    cublasHandle_t blas[kHandleDevices];
    unsigned sol_gen[kHandleDevices], blas_gen[kHandleDevices];   // device generation at creation
};
thread_local ThreadHandles t_handles = {};

int handle_device(int* dev) {
    if (cudaGetDevice(dev) != cudaSuccess || *dev < 0 || *dev >= kHandleDevices) {
        cudaGetLastError();
        return fail(EBEM_ERR_CUDA, "no usable current device for a library handle");
    }
    return EBEM_OK;
}
}  // namespace

int solver_handle(cudaStream_t s, cusolverDnHandle_t* h) {
    int dev = 0;
    if (int rc = handle_device(&dev)) return rc;
    cusolverDnHandle_t& c = t_handles.sol[dev];
    const unsigned gen = device_generation(dev);
    if (c && t_handles.sol_gen[dev] != gen) c = nullptr;      // released device state: abandoned
    if (!c) {
        if (cusolverDnCreate(&c) != CUSOLVER_STATUS_SUCCESS) {
            c = nullptr;
            return fail(EBEM_ERR_CUDA, "cuSOLVER handle creation failed");
        }
        t_handles.sol_gen[dev] = gen;
    }
    if (cusolverDnSetStream(c, s) != CUSOLVER_STATUS_SUCCESS) return fail(EBEM_ERR_CUDA, "cuSOLVER stream binding failed");
    *h = c;
    return EBEM_OK;
}

int blas_handle(cudaStream_t s, cublasHandle_t* h) {
    int dev = 0;
    if (int rc = handle_device(&dev)) return rc;
    cublasHandle_t& c = t_handles.blas[dev];
    const unsigned gen = device_generation(dev);
    if (c && t_handles.blas_gen[dev] != gen) c = nullptr;     // released device state: abandoned
    if (!c) {
        if (cublasCreate(&c) != CUBLAS_STATUS_SUCCESS) {
            c = nullptr;
            return fail(EBEM_ERR_CUDA, "cuBLAS handle creation failed");
        }
        t_handles.blas_gen[dev] = gen;
    }
    if (cublasSetStream(c, s) != CUBLAS_STATUS_SUCCESS) return fail(EBEM_ERR_CUDA, "cuBLAS stream binding failed");
    *h = c;
    return EBEM_OK;
}

void release_thread_handles(int dev) {
    if (dev < 0 || dev >= kHandleDevices) return;
    if (!t_handles.sol[dev] && !t_handles.blas[dev]) return;
    int prev = -1;
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    cudaSetDevice(dev);
    if (t_handles.sol[dev]) cusolverDnDestroy(t_handles.sol[dev]);
    if (t_handles.blas[dev]) cublasDestroy(t_handles.blas[dev]);
    t_handles.sol[dev] = nullptr;
    t_handles.blas[dev] = nullptr;
    if (prev >= 0) cudaSetDevice(prev);
    cudaGetLastError();
}

// phi (device, column-major n3 x nT) from E (device, n3 x n3 x L) and rhs
// (device, n3 x nT): E_0^{-1} once, then per step the history product and
// one product with E_0^{-1}.
int march_device(const double* dE, int n3, int L, const double* drhs, int nT, double* dphi, cudaStream_t s,
                 int factor) {
    int rc = EBEM_OK, dev = 0, sms = 148;
    double *rev = nullptr, *Y = nullptr;
    LuPlan lu;
    const size_t nn = (size_t)n3 * n3, tot = (size_t)n3 * nT;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (ws_malloc(&rev, 2 * tot * sizeof(double), s) != cudaSuccess)
        return fail(EBEM_ERR_NOMEM, "time-marching workspace allocation failed");
    Y = rev + tot;
    rc = lu_plan_create(dE, n3, s, &lu, true, factor == EBEM_FACTOR_CHOLESKY);
    if (!rc) {
        // density in reversed time order: phi_n at column nT-1-n, so that
        // phi_{n-1}, phi_{n-2}, ... are contiguous for the history product;
        // right-hand sides in time order.  The steps go in blocks of
        // kHistBlock: what the steps before the block contribute to all of
        // them in one product, the lags inside the block step by step.
        if (cudaMemsetAsync(rev, 0, tot * sizeof(double), s) != cudaSuccess ||
            cudaMemcpyAsync(Y, drhs, tot * sizeof(double), cudaMemcpyDeviceToDevice, s) != cudaSuccess)
            rc = fail(EBEM_ERR_CUDA, "rhs copy failed");
        for (int n = 0; n < nT && !rc; n++) {
            const int i = n % kHistBlock, M = std::min(i, L - 1);
            double *y = Y + (size_t)n * n3, *phi = rev + (size_t)(nT - 1 - n) * n3;
            if (i == 0) rc = launch_hist_block(dE + nn, n3, n3, L - 1, rev, nT, n, Y, sms, s);
            if (!rc && M > 0) rc = launch_hist_gemv(dE + nn, n3, (long long)n3 * M, phi + n3, y, sms, s);
            if (!rc) rc = launch_gemv_add(lu.inv, n3, n3, y, phi, sms, s);
        }
        if (!rc) {
            copy_reverse_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(rev, dphi, n3, nT);
            if (cudaGetLastError() != cudaSuccess) rc = fail(EBEM_ERR_CUDA, "density copy failed");
        }
        if (!rc && cudaStreamSynchronize(s) != cudaSuccess) rc = fail(EBEM_ERR_CUDA, "time marching failed");
    }
    lu_plan_destroy(&lu);
    ws_free(rev, s);
    return rc;
}

// ---------------------------------------------------------------------------
// A^{-1} of one matrix kept on the device (the E_0 solve of the marching,
// also for callers that drive the steps themselves): Gauss-Jordan elimination
// with partial pivoting; past its size, or where the device has no room for
// its cluster or buffers, LU (getrf) and getrs on the identity, whose n
// right-hand sides run as matrix-matrix triangular solves.
__global__ void set_identity_kernel(double* __restrict__ a, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[(size_t)i * n + i] = 1.0;
}

// (A + A^T) / 2 in place (column-major n x n).
__global__ void symmetrize_kernel(double* __restrict__ a, int n) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(idx % n), j = (int)(idx / n);
    if (idx >= (long long)n * n || i >= j) return;
    const double v = 0.5 * (a[(size_t)j * n + i] + a[(size_t)i * n + j]);
    a[(size_t)j * n + i] = v;
    a[(size_t)i * n + j] = v;
}

int lu_plan_create(const double* dA, int n, cudaStream_t s, LuPlan* plan, bool pooled, bool cholesky) {
    int rc = EBEM_OK;
    int lwork = 0, hinfo = 0;
    double *lu = nullptr, *work = nullptr;
    int *ipiv = nullptr, *info = nullptr;
    const size_t nn = (size_t)n * n;
    cusolverDnHandle_t h = nullptr;
    plan->n = n;
    plan->pooled = pooled;
    plan->st = s;
    cudaError_t e = pooled ? ws_malloc(&plan->inv, nn * sizeof(double), s) : cudaMalloc(&plan->inv, nn * sizeof(double));
    if (e != cudaSuccess) {
        cudaGetLastError();
        plan->inv = nullptr;
        return fail(EBEM_ERR_NOMEM, "inverse allocation failed");
    }
    if (!cholesky && n <= gj_max_n()) {
        // Gauss-Jordan elimination (inverse.cu): its panel is one row per thread of
        // one cluster, 4096 rows at most.  n = 4096 with one marching step: 17.5 ms
        // against 24.6 ms for the library's LU and triangular solves, which larger
        // matrices take.
        bool placed = false;
        rc = gj_inverse(dA, n, plan->inv, &hinfo, &placed, s);
        if (!rc && hinfo != 0) rc = fail(EBEM_ERR_SINGULAR, "matrix is singular (zero pivot " + std::to_string(hinfo) + ")");
        if (rc || placed) return rc;
    }
    if ((rc = solver_handle(s, &h))) return rc;
    if (ws_malloc(&lu, nn * sizeof(double), s) != cudaSuccess || ws_malloc(&ipiv, n * sizeof(int), s) != cudaSuccess ||
        ws_malloc(&info, sizeof(int), s) != cudaSuccess) {
        rc = fail(EBEM_ERR_NOMEM, "LU workspace allocation failed");
        goto done;
    }
    if (cudaMemcpyAsync(lu, dA, nn * sizeof(double), cudaMemcpyDeviceToDevice, s) != cudaSuccess) {
        rc = fail(EBEM_ERR_CUDA, "matrix copy failed");
        goto done;
    }
    if (cholesky) {
        symmetrize_kernel<<<(unsigned)(((long long)n * n + 255) / 256), 256, 0, s>>>(lu, n);
        CUSOLVER_TRY(cusolverDnDpotrf_bufferSize(h, CUBLAS_FILL_MODE_LOWER, n, lu, n, &lwork));
    } else {
        CUSOLVER_TRY(cusolverDnDgetrf_bufferSize(h, n, n, lu, n, &lwork));
    }
    if (ws_malloc(&work, (size_t)(lwork > 0 ? lwork : 1) * sizeof(double), s) != cudaSuccess) {
        rc = fail(EBEM_ERR_NOMEM, "LU workspace allocation failed");
        goto done;
    }
    if (cholesky) CUSOLVER_TRY(cusolverDnDpotrf(h, CUBLAS_FILL_MODE_LOWER, n, lu, n, work, lwork, info));
    else CUSOLVER_TRY(cusolverDnDgetrf(h, n, n, lu, n, work, ipiv, info));
    if (cudaMemcpyAsync(&hinfo, info, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess) {
        rc = fail(EBEM_ERR_CUDA, "LU factorisation failed");
        goto done;
    }
    if (hinfo != 0) {
        rc = cholesky ? fail(EBEM_ERR_SINGULAR, "the symmetric part of the matrix is not positive definite (leading "
                                                "minor " + std::to_string(hinfo) + ")")
                      : fail(EBEM_ERR_SINGULAR, "matrix is singular (zero pivot " + std::to_string(hinfo) + ")");
        goto done;
    }
    if (cudaMemsetAsync(plan->inv, 0, nn * sizeof(double), s) != cudaSuccess) {
        rc = fail(EBEM_ERR_CUDA, "inverse initialisation failed");
        goto done;
    }
    set_identity_kernel<<<(n + 255) / 256, 256, 0, s>>>(plan->inv, n);
    if (cudaGetLastError() != cudaSuccess) {
        rc = fail(EBEM_ERR_CUDA, "inverse initialisation failed");
        goto done;
    }
    if (cholesky) CUSOLVER_TRY(cusolverDnDpotrs(h, CUBLAS_FILL_MODE_LOWER, n, n, lu, n, plan->inv, n, info));
    else CUSOLVER_TRY(cusolverDnDgetrs(h, CUBLAS_OP_N, n, n, lu, n, ipiv, plan->inv, n, info));
done:
    ws_free(lu, s);
    ws_free(work, s);
    ws_free(ipiv, s);
    ws_free(info, s);
    return rc;
}

// b (n x nrhs, device, overwritten) = A^{-1} b.
int lu_plan_solve(LuPlan* plan, double* db, int nrhs, cudaStream_t s) {
    cublasHandle_t hb = nullptr;
    if (int rc = blas_handle(s, &hb)) return rc;
    const int n = plan->n;
    const size_t cnt = (size_t)n * nrhs;
    double* tmp = nullptr;
    if (ws_malloc(&tmp, cnt * sizeof(double), s) != cudaSuccess) return fail(EBEM_ERR_NOMEM, "solve workspace allocation failed");
    const double one = 1.0, zero = 0.0;
    const cublasStatus_t st =
        nrhs == 1 ? cublasDgemv(hb, CUBLAS_OP_N, n, n, &one, plan->inv, n, db, 1, &zero, tmp, 1)
                  : cublasDgemm(hb, CUBLAS_OP_N, CUBLAS_OP_N, n, nrhs, n, &one, plan->inv, n, db, n, &zero, tmp, n);
    cudaError_t e = st == CUBLAS_STATUS_SUCCESS ? cudaMemcpyAsync(db, tmp, cnt * sizeof(double), cudaMemcpyDeviceToDevice, s)
                                                : cudaSuccess;
    ws_free(tmp, s);
    if (st != CUBLAS_STATUS_SUCCESS) return fail(EBEM_ERR_CUDA, "product with the inverse failed (cuBLAS status " + std::to_string((int)st) + ")");
    if (e != cudaSuccess) return fail(EBEM_ERR_CUDA, std::string("solve copy: ") + cudaGetErrorString(e));
    return EBEM_OK;
}

void lu_plan_destroy(LuPlan* plan) {
    if (plan->inv) {
        if (plan->pooled) ws_free(plan->inv, plan->st);
        else cudaFree(plan->inv);
    }
    plan->inv = nullptr;
}

// ---------------------------------------------------------------------------
// Post-processing (closed form): u(x, t) = sum_{k=1}^{nHat} (M(t - (k-1) dt)
// - M(t - k dt)) phi_k + M(t - nHat dt) phi_{nHat+1}, nHat = ceil(t/dt) - 1,
// M(tau) the single-point combined kernel integral over each triangle
// (BEMenerg_postProcA_singlePoint.m:21-61), divided by 4 pi rho and cleaned
// below 1e-14 (BEMenerg_postProcA_calcMatrix.m:103).
__device__ __forceinline__ void sym_mv_add(double acc[3], const double M[6], const double* ph, double sgn) {
    acc[0] += sgn * (M[0] * ph[0] + M[1] * ph[1] + M[2] * ph[2]);
    acc[1] += sgn * (M[1] * ph[0] + M[3] * ph[1] + M[4] * ph[2]);
    acc[2] += sgn * (M[2] * ph[0] + M[4] * ph[1] + M[5] * ph[2]);
}

// The instants at which M(tau) of triangle F seen from x is zero without
// evaluating it: the P front (radius velP tau) has not reached the triangle.
// M is zero when the closed form's case split finds no front at the node
// (T_NONE), which needs velP tau <= sqrt(zeta^2 + dMIN^2) as the
// projection computes them; that is at least the distance from x to the
// triangle less the projection's tolerances (the plane distance snapped to
// 0 below 1e-6, the inside test's 1e-6 on the barycentrics, the edge foot
// tests' 1e-6, which can take a foot up to 1e-6 / |edge| <= 1e-6 maxL / (2
// area) beyond an end), and that distance is at least the centroid distance
// less the longest edge.  pp_reach returns that bound less a margin of half
// the longest edge on top of the tolerances; an instant with velP tau below
// it is skipped.  Rounded explicitly (no contraction): the evaluation pass
// and the contraction must take the same decision for every instant.
__device__ __forceinline__ double pp_reach(const TriGeom& F, const NodeW& x) {
    const double d0 = __dsub_rn(x.x, F.ctr[0]), d1 = __dsub_rn(x.y, F.ctr[1]), d2 = __dsub_rn(x.z, F.ctr[2]);
    const double r = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2)));
    const double tol = __dadd_rn(__dadd_rn(__dmul_rn(0.5, F.maxL), 1.0e-5),
                                 __dadd_rn(__ddiv_rn(__dmul_rn(1.0e-6, F.maxL), F.area), __dmul_rn(1.0e-12, r)));
    return __dsub_rn(__dsub_rn(r, F.maxL), tol);     // a degenerate triangle (area 0) gives -inf: never skipped
}

__device__ __forceinline__ bool pp_before_front(double reach, double velP, double tau) {
    return __dmul_rn(velP, tau) < reach;
}

// By parts the sum above is
//   u(x, t_q) = M(t_q) phi_0 + sum_{k=1}^{nHat} M(t_q - k dt) (phi_k - phi_{k-1}),
// and for output times on the time grid the instants t_q - k dt of different
// (q, k) coincide.  The instants are formed on the host as k dt rounded, then
// subtracted from t_q (no fused multiply-add: the closed form's case
// selection is discontinuous where a front radius equals the point's distance
// from the plane, so an instant one unit in the last place off can change M
// there) and deduplicated by value; pp_front_kernel evaluates M once per
// (triangle, point, distinct instant that the P front has reached);
// pp_inst_sum_kernel contracts, one block per (time, point).
//
// pp_front_kernel: one warp per (point, 10 consecutive triangles), their 30
// children on the lanes (sa_group.cuh), so that what does not depend on the
// instant is formed once.  Then per triangle the instants run over the lanes:
// those at which no side is partly covered (zero, or the whole triangle: a +
// tau^2 b) are finished at once; the others, (triangle, instant) cells with
// one to six (front, child) items, are queued and evaluated 32 at a time, a
// lane walking its cell's items.  1280 triangles, 256 points, 40 grid times:
// 0.47 ms, against 9.4 ms for one thread per (triangle, point, instant) with
// the edge pieces by Gauss-Legendre (the whole call 9.9 -> 1.2 ms).
struct PPShared {
    FrontGroup W;
    double C[kGroupNodes][9];
    double near[kSlots], all[kGroupNodes];
    int first[kGroupNodes];
    int2 queue[64];                // (triangle of the group, instant)
};

// M of the cell, cleaned, to the buffer.
__device__ __forceinline__ void pp_store(double* dst, const double T[7], const double* C, double ic4) {
    double Fk[6];
    front_rotate(Fk, T, C);
#pragma unroll
    for (int e = 0; e < 6; e++) {
        const double v = Fk[e] * ic4;
        Fk[e] = (fabs(v) < 1.0e-14) ? 0.0 : v;
    }
    double2* d2 = reinterpret_cast<double2*>(dst);
    d2[0] = make_double2(Fk[0], Fk[1]);
    d2[1] = make_double2(Fk[2], Fk[3]);
    d2[2] = make_double2(Fk[4], Fk[5]);
}

constexpr int kPPWarps = 4;
__global__ void __launch_bounds__(32 * kPPWarps, 4) pp_front_kernel(const TriGeom* __restrict__ geo, int N,
                                                                    const double* __restrict__ pts, int p0, int np, int nu,
                                                                    const double* __restrict__ taus, double velP,
                                                                    double velS, double ic4, double* __restrict__ Mbuf) {
    extern __shared__ __align__(16) unsigned char pp_smem[];
    const int lane = threadIdx.x & 31;
    PPShared& S = reinterpret_cast<PPShared*>(pp_smem)[threadIdx.x >> 5];
    const int groups = (N + kGroupNodes - 1) / kGroupNodes;
    const long long tasks = (long long)groups * np, nwarps = (long long)gridDim.x * kPPWarps;
    const double k1 = 1.0 / (velP * velP), ks = 1.0 / (velS * velS);
    const int g = lane / 3, c = lane - 3 * g;
    for (long long t = (long long)blockIdx.x * kPPWarps + (threadIdx.x >> 5); t < tasks; t += nwarps) {
        const int pl = (int)(t / groups), j0 = (int)(t - (long long)pl * groups) * kGroupNodes;
        const int gn = min(kGroupNodes, N - j0), p = p0 + pl;
        NodeW x;
        x.x = pts[3 * p]; x.y = pts[3 * p + 1]; x.z = pts[3 * p + 2]; x.w = 1.0;
        const TriGeom* F = geo + j0 + min(g, gn - 1);
        __syncwarp();
        int first = nu;
        if (g < gn) {
            // the skip test is monotone in the sorted instants: first instant not skipped
            const double reach = pp_reach(*F, x);
            int lo = 0, hi = nu;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (pp_before_front(reach, velP, taus[mid])) lo = mid + 1;
                else hi = mid;
            }
            first = lo;
        }
        if (__ballot_sync(0xffffffffu, first < nu) == 0u) continue;
        FrontLane L;
        group_geometry(L, g < gn, &x, F, lane);
        const unsigned circ = group_fields(S.W, L, lane), split = __ballot_sync(0xffffffffu, L.split);
        auto add_split = [&](double T[7], int gg, bool cP, bool cS, double rP, double rS, double t2) {
            for (unsigned m = (split >> (3 * gg)) & 7u; m; m &= m - 1) {
                const int slot = 3 * gg + __ffs(m) - 1;
                if ((cP || rP > S.near[slot]) && !(cS || rS > S.near[slot])) group_foot(T, S.W, slot, t2);
            }
        };
        if (L.child) {
            S.near[lane] = L.live ? L.near : INFINITY;
            if (c == 0) {
                S.all[g] = L.all;
                S.first[g] = first;
            }
#pragma unroll
            for (int e = 0; e < 3; e++) S.C[g][3 * c + e] = F->C[3 * c + e];
        }
        __syncwarp();
        int queued = 0;
        for (int gg = 0; gg <= gn; gg++) {
            const int u0 = gg < gn ? S.first[gg] : nu - 1;          // one step past the last triangle empties the queue
            for (int ub = u0; ub < nu; ub += 32) {
                const int ui = ub + lane;
                bool ask = false;
                if (gg < gn && ui < nu) {
                    const double tau = taus[ui], rP = velP * tau, rS = velS * tau, z = S.W.zeta[gg], all = S.all[gg];
                    const bool front = z == 0.0 || z != rS;        // c_S tau == zeta: no front
                    const bool cP = front && rP > all, cS = front && rS > all;
                    if (front)
#pragma unroll
                        for (int k = 0; k < 3; k++)
                            ask = ask || (!cP && rP > S.near[3 * gg + k]) || (!cS && rS > S.near[3 * gg + k]);
                    if (!ask) {
                        double T[7] = {0, 0, 0, 0, 0, 0, 0};
                        group_node(T, S.W, gg, cP, cS, (circ >> (3 * gg)) & 1u, rP, rS, tau * tau, k1, ks);
                        if (cP && !cS) add_split(T, gg, cP, cS, rP, rS, tau * tau);
                        pp_store(Mbuf + (((size_t)pl * nu + ui) * N + j0 + gg) * 6, T, S.C[gg], ic4);
                    }
                }
                const unsigned asking = __ballot_sync(0xffffffffu, ask);
                if (ask) S.queue[queued + __popc(asking & ((1u << lane) - 1u))] = make_int2(gg, ui);
                queued += __popc(asking);
                __syncwarp();
                if (queued >= 32 || (gg == gn && queued > 0)) {
                    const int n = min(queued, 32);
                    if (lane < n) {
                        const int2 cell = S.queue[lane];
                        const double tau = taus[cell.y], rP = velP * tau, rS = velS * tau, all = S.all[cell.x];
                        const bool cP = rP > all, cS = rS > all;
                        unsigned m = 0;
#pragma unroll
                        for (int k = 0; k < 3; k++) {
                            if (!cP && rP > S.near[3 * cell.x + k]) m |= 1u << k;
                            if (!cS && rS > S.near[3 * cell.x + k]) m |= 8u << k;
                        }
                        double T[7] = {0, 0, 0, 0, 0, 0, 0};
                        group_node(T, S.W, cell.x, cP, cS, (circ >> (3 * cell.x)) & 1u, rP, rS, tau * tau, k1, ks);
                        add_split(T, cell.x, cP, cS, rP, rS, tau * tau);
                        while (m) {
                            const int k = __ffs(m) - 1;
                            m &= m - 1;
                            const bool isP = k < 3;
                            const int slot = 3 * cell.x + (isP ? k : k - 3);
                            group_item(T, S.W, slot, !((split >> slot) & 1u), isP, isP ? rP : rS, isP ? k1 : ks);
                        }
                        pp_store(Mbuf + (((size_t)pl * nu + cell.y) * N + j0 + cell.x) * 6, T, S.C[cell.x], ic4);
                    }
                    const int2 rest = S.queue[32 + lane];
                    __syncwarp();
                    queued -= n;
                    if (lane < queued) S.queue[lane] = rest;
                    __syncwarp();
                }
            }
        }
    }
}

// Blocks of 128 threads, or of 1024 when there are too few (time, point)
// pairs to fill the GPU.
__global__ void __launch_bounds__(1024) pp_inst_sum_kernel(const double* __restrict__ Mbuf, const TriGeom* __restrict__ geo,
                                                          int N, const double* __restrict__ pts, int p0, int np, int nu,
                                                          const double* __restrict__ taus, double velP,
                                                          const int* __restrict__ tab, int kmax,
                                                          const int* __restrict__ nhat, int npts,
                                                          const double* __restrict__ phi, double* __restrict__ u) {
    const int q = blockIdx.x / np, pl = blockIdx.x - q * np;
    const int nh = nhat[q];
    const int* tq = tab + (size_t)q * kmax;
    const size_t n3 = 3 * (size_t)N;
    const int p = p0 + pl;
    NodeW x;
    x.x = pts[3 * p]; x.y = pts[3 * p + 1]; x.z = pts[3 * p + 2]; x.w = 1.0;
    double acc[3] = {0, 0, 0};
    for (int j = threadIdx.x; j < N; j += blockDim.x) {
        const double reach = pp_reach(geo[j], x);
        for (int k = 0; k <= nh; k++) {
            if (pp_before_front(reach, velP, taus[tq[k]])) break;       // M = 0 from here on (instants fall with k), not stored
            const double* Mv = Mbuf + (((size_t)pl * nu + tq[k]) * N + j) * 6;
            const double* pk = phi + (size_t)k * n3 + 3 * (size_t)j;
            double d[3] = {pk[0], pk[1], pk[2]};
            if (k > 0) {
                d[0] -= pk[-(long long)n3];
                d[1] -= pk[1 - (long long)n3];
                d[2] -= pk[2 - (long long)n3];
            }
            double Ml[6];
#pragma unroll
            for (int e = 0; e < 6; e++) Ml[e] = Mv[e];
            sym_mv_add(acc, Ml, d, 1.0);
        }
    }
    __shared__ double red[3][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        double v = acc[c];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[c][w] = v;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double v = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) v += red[threadIdx.x][i];
        u[((size_t)q * npts + p0 + pl) * 3 + threadIdx.x] = v;
    }
}

void form_instants(const double* times, int ntimes, double dt, int nT, Instants* out) {
    Instants& I = *out;
    I.nh.assign(ntimes, -1);
    I.kmax = 1;
    size_t total = 0;
    for (int q = 0; q < ntimes; q++) {
        if (times[q] > 0) I.nh[q] = std::min((int)std::ceil(times[q] / dt) - 1, nT - 1);
        I.kmax = std::max(I.kmax, I.nh[q] + 1);
        total += I.nh[q] + 1;
    }
    auto instant = [&](int q, int k) {
        volatile double a = (double)k * dt;        // rounded product, then the difference
        return times[q] - a;
    };
    I.tab.assign((size_t)ntimes * I.kmax, 0);
    // The n-th smallest instants of all times lie within one dt of each other: in
    // ascending order as they are visited here unless times differ by whole steps
    // (on the time grid), where the rounding of a step decides the order.
    std::vector<std::pair<double, int>> runs;      // smallest instant of each time
    for (int q = 0; q < ntimes; q++)
        if (I.nh[q] >= 0) runs.emplace_back(instant(q, I.nh[q]), q);
    std::sort(runs.begin(), runs.end());
    I.uniq.clear();
    I.uniq.reserve(total);
    bool sorted = true;
    for (int n = 0; n < I.kmax && sorted; n++)
        for (const auto& r : runs) {
            const int q = r.second, k = I.nh[q] - n;
            if (k < 0) continue;
            const double t = instant(q, k);
            if (!I.uniq.empty() && !(t >= I.uniq.back())) {
                sorted = false;
                break;
            }
            if (I.uniq.empty() || t != I.uniq.back()) I.uniq.push_back(t);
            I.tab[(size_t)q * I.kmax + k] = (int)I.uniq.size() - 1;
        }
    if (sorted) return;
    I.uniq.clear();
    for (int q = 0; q < ntimes; q++)
        for (int k = 0; k <= I.nh[q]; k++) I.uniq.push_back(instant(q, k));
    const std::vector<double> taus(I.uniq);
    std::sort(I.uniq.begin(), I.uniq.end());
    I.uniq.erase(std::unique(I.uniq.begin(), I.uniq.end()), I.uniq.end());
    size_t c = 0;
    for (int q = 0; q < ntimes; q++)
        for (int k = 0; k <= I.nh[q]; k++)
            I.tab[(size_t)q * I.kmax + k] = (int)(std::lower_bound(I.uniq.begin(), I.uniq.end(), taus[c++]) - I.uniq.begin());
}

int launch_pp_sa(const MeshData& m, const PhysParams& P, const double* d_phi, const double* d_pts, int npts,
                       const double* h_times, int ntimes, double* d_u, cudaStream_t s) {
    Instants I;
    form_instants(h_times, ntimes, P.dt, P.nT, &I);
    const int nu = (int)I.uniq.size(), kmax = I.kmax;
    if (nu == 0) {
        // no instant: u = 0
        EBEM_CUDA_TRY(cudaMemsetAsync(d_u, 0, sizeof(double) * 3 * (size_t)npts * ntimes, s));
        return EBEM_OK;
    }
    const size_t per_point = (size_t)nu * m.nt * 6 * sizeof(double);
    auto by_halves = [&]() {
        const int half = ntimes / 2;
        if (int rc = launch_pp_sa(m, P, d_phi, d_pts, npts, h_times, half, d_u, s)) return rc;
        return launch_pp_sa(m, P, d_phi, d_pts, npts, h_times + half, ntimes - half, d_u + 3 * (size_t)npts * half, s);
    };
    // times off the grid have their own instants each
    if (per_point > ((size_t)1 << 30) && ntimes > 1) return by_halves();
    // up to 1 GiB of M at a time.  1280 triangles, 256 points, 40 grid times (114
    // distinct instants, 7 MB a point): 1.18 ms; 512 MB 1.35, 192 MB 1.88, 96 MB
    // 2.98 (a chunk of 14 points has fewer warps than the GPU holds).
    int chunk = (int)std::max<size_t>(1, std::min<size_t>((size_t)npts, ((size_t)1 << 30) / per_point));
    // the tables in one upload: instants, index table, nHat
    HostPack pk;
    const size_t o_taus = pk.add(I.uniq.data(), nu * sizeof(double));
    const size_t o_tab = pk.add(I.tab.data(), I.tab.size() * sizeof(int));
    const size_t o_nh = pk.add(I.nh.data(), ntimes * sizeof(int));
    unsigned char* d_pack = nullptr;
    double* Mbuf = nullptr;
    if (pk.upload(&d_pack, s) != cudaSuccess) {
        cudaGetLastError();
        ws_free(d_pack, s);
        return fail(EBEM_ERR_NOMEM, "post-processing workspace allocation failed");
    }
    while (ws_malloc(&Mbuf, per_point * chunk, s) != cudaSuccess) {
        // a device with less to spare: fewer points, then fewer times at a time
        if (chunk == 1) {
            ws_free(d_pack, s);
            return ntimes > 1 ? by_halves() : fail(EBEM_ERR_NOMEM, "post-processing workspace allocation failed");
        }
        chunk = (chunk + 1) / 2;
    }
    const double* d_taus = reinterpret_cast<const double*>(d_pack + o_taus);
    const int* d_tab = reinterpret_cast<const int*>(d_pack + o_tab);
    const int* d_nh = reinterpret_cast<const int*>(d_pack + o_nh);
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m.device);
    const size_t smem = sizeof(PPShared) * kPPWarps;
    cudaError_t e = cudaFuncSetAttribute(pp_front_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    for (int p0 = 0; p0 < npts && e == cudaSuccess; p0 += chunk) {
        const int np = std::min(chunk, npts - p0);
        const long long tasks = (long long)((m.nt + kGroupNodes - 1) / kGroupNodes) * np;
        const long long want = (tasks + kPPWarps - 1) / kPPWarps, cap = 64LL * sms;
        pp_front_kernel<<<(unsigned)std::min(want, cap), 32 * kPPWarps, smem, s>>>(
            m.d_geo, m.nt, d_pts, p0, np, nu, d_taus, P.velP, P.velS, 1.0 / (4 * kPi * P.rho), Mbuf);
        const int sum_threads = ((long long)ntimes * np < 2LL * sms) ? 1024 : 128;
        pp_inst_sum_kernel<<<(unsigned)((long long)ntimes * np), sum_threads, 0, s>>>(
            Mbuf, m.d_geo, m.nt, d_pts, p0, np, nu, d_taus, P.velP, d_tab, kmax, d_nh, npts, d_phi, d_u);
        e = cudaGetLastError();
    }
    ws_free(Mbuf, s);
    ws_free(d_pack, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail(EBEM_ERR_CUDA, std::string("post-processing kernels: ") + cudaGetErrorString(e));
    return EBEM_OK;
}

}  // namespace ebem
