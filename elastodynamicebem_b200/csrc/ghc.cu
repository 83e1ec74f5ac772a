// Numerical-inner assembly of E_l: outer Gauss-Hammer rule on the source
// triangle, composite Gauss-Hammer rule on the field triangle, the Lamé kernel
// integrated twice in time with separate P and S Heaviside fronts.
//
// Reference: functions/BEMenerg_indir/BEMenerg_core/BEMenerg_coreGPU/CUDAkernels/
// kernelGHC.cu:5-259 (identical copies: BEMenerg_coreFN/CUDAkernels/kernelGHC.cu,
// functions/BEMenerg_dir/CUDAkernels/kernelV.cu), launched by
// BEMenerg_coreGPU_launchKernel.m:11 with grid (N, N, lags) and one thread
// per inner node.  Semantics kept: off-diagonal pairs only (the diagonal
// comes from the semi-analytic path, BEMenerg_coreGPU_timeMarching.m:101-131),
// the null test (lag-1) c_S dt > max vertex distance (kernelGHC.cu:171-201),
// instants dt (lag + {-1, 0, 1}) with weights (1, -2, 1) and t >= 0
// (:88-99), entries written only when |value| > 1e-14 before the division by
// 4 pi rho (:164-165), accumulated into the output (+=).
//
// B200 design: the lag combination E_l = K_{l+1} - 2 K_l + K_{l-1} is taken per
// node pair and front, where it is non-zero in two lags and a constant after
// them; a warp per (source, field) pair sorts its node pairs by the level of
// the arrival and evaluates each once per front (the reference evaluates every
// node pair at every instant of every lag and reduces through shared memory).
#include "ebem_internal.h"
#include "sa_pair.cuh"

#include "front_bins.cuh"
#include "sa_math.cuh"

namespace ebem {

struct GHCArgs {
    const double* coords;
    const int32_t* tris;
    const TriGeom* geo;
    const double* outer;    // n_out x 3 barycentric
    const double* wout;     // n_out
    const double* inner;    // n_in x 3 barycentric (n_sub sub-triangles x n_sing nodes)
    const double* win;      // n_sing
    int n_out, n_sub, n_sing;
    int N;
    double velP, velS, dt, c4pirho;
    int lag0, nlag;
    double* E;
    size_t ld, ld_lag;
};

// Second difference over the window of lag l (levels l-1, l, l+1 of t_k =
// k dt, kernelGHC.cu:88-99) of the time functions of one front X of the
// kernel kernelGHC.cu:204-259 (nucleo): H = [t - r/c > 0] and
// Q = (c^2 t^2 - r^2) / c^2 H.  Before the front both vanish; with the whole
// window after it H is constant and Q = t^2 - r^2/c^2, so the differences
// are exactly (0, 2 dt^2).
struct Win2 {
    double H, Q;
};

// t: the three levels, rounded products.
__device__ __forceinline__ Win2 ghc_window2(double r, double c, int l, const double t[3], double dt) {
    Win2 d = {0.0, 0.0};
    const double tX = r / c;
    if (t[2] - tX <= 0) return d;
    if (l >= 1 && t[0] - tX > 0) {
        d.Q = 2 * dt * dt;
        return d;
    }
    const double w[3] = {1.0, -2.0, 1.0};
#pragma unroll
    for (int j = 0; j < 3; j++) {
        if (l - 1 + j < 0) continue;
        if (t[j] - tX > 0) {
            d.H += w[j];
            d.Q += w[j] * ((c * c * t[j] * t[j] - r * r) / (c * c));
        }
    }
    return d;
}

// One node pair's share of the lag-l second difference of nucleo, symmetric
// entries (11,12,13,22,23,33): with dQ = dQ_P - dQ_S,
//   out_ij = g1 x_i x_j + g2 delta_ij,
//   g1 = ir^3 (dH_P/c_P^2 - dH_S/c_S^2) + 3/2 ir^5 dQ,  g2 = ir dH_S/c_S^2 - 1/2 ir^3 dQ.
__host__ __device__ __forceinline__ void ghc_pair(double nu[6], const double x[3], double ir, double dHP, double dHS,
                                                  double dQ, double icP2, double icS2) {
    const double ir2 = ir * ir, ir3 = ir2 * ir, ir5 = ir3 * ir2;
    const double g1 = ir3 * (dHP * icP2 - dHS * icS2) + 1.5 * ir5 * dQ;
    const double g2 = ir * dHS * icS2 - 0.5 * ir3 * dQ;
    nu[0] = g1 * x[0] * x[0] + g2;
    nu[1] = g1 * x[0] * x[1];
    nu[2] = g1 * x[0] * x[2];
    nu[3] = g1 * x[1] * x[1] + g2;
    nu[4] = g1 * x[1] * x[2];
    nu[5] = g1 * x[2] * x[2] + g2;
}

// Thread per pair, for rules of few node pairs on many pairs (see the launch).
// 80 registers: bound by the latency of its FP64 chains (157 without the cap:
// bar of 2800 triangles, rule 7/4/3 188 ms against 137).
__global__ void __launch_bounds__(128, 6) ghc_assemble_thread_kernel(GHCArgs A) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (long long)A.N * A.N) return;
    const int i = (int)(p % A.N);          // source (outer rule)
    const int j = (int)(p / A.N);          // field (inner rule)
    if (i == j) return;
    double VS[3][3], VF[3][3];
    for (int v = 0; v < 3; v++)
        for (int c = 0; c < 3; c++) {
            VS[v][c] = A.coords[3 * A.tris[3 * i + v] + c];
            VF[v][c] = A.coords[3 * A.tris[3 * j + v] + c];
        }
    double distMax = 0;
    for (int a = 0; a < 3; a++)
        for (int b = 0; b < 3; b++) {
            double d0 = VS[a][0] - VF[b][0], d1 = VS[a][1] - VF[b][1], d2 = VS[a][2] - VF[b][2];
            distMax = fmax(distMax, sqrt(d0 * d0 + d1 * d1 + d2 * d2));
        }
    // lags computed: not null, i.e. (l-1) c_S dt <= distMax
    int lhi = A.lag0 + A.nlag - 1;
    while (lhi >= A.lag0 && (lhi - 1) * A.velS * A.dt > distMax) lhi--;
    if (lhi < A.lag0) return;
    const double aS = A.geo[i].area, aF = A.geo[j].area;
    const double cP = A.velP, cS = A.velS, dt = A.dt;
    const double icP2 = 1 / (cP * cP), icS2 = 1 / (cS * cS);
    const size_t n3 = A.ld;
    const int map[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
    // the node pairs' exact distance range (one pass): a lag whose window lies
    // before the P front or after the S front for all of them adds nothing
    // (the null test above bounds the lags by vertex distances only)
    double r2min = 1e300, r2max = 0.0;
    for (int q = 0; q < A.n_sub * A.n_sing; q++) {
        const double* bq = A.inner + 3 * q;
        double y[3];
        for (int c = 0; c < 3; c++) y[c] = bq[0] * VF[0][c] + bq[1] * VF[1][c] + bq[2] * VF[2][c];
        for (int o = 0; o < A.n_out; o++) {
            const double* bl = A.outer + 3 * o;
            double x[3];
            for (int c = 0; c < 3; c++) x[c] = y[c] - (bl[0] * VS[0][c] + bl[1] * VS[1][c] + bl[2] * VS[2][c]);
            const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
            r2min = fmin(r2min, r2);
            r2max = fmax(r2max, r2);
        }
    }
    for (int l = A.lag0; l <= lhi; l++) {
        const double tl[3] = {level_time(l - 1, dt), level_time(l, dt), level_time(l + 1, dt)};
        const double skipP2 = (cP * tl[2]) * (cP * tl[2]) * (1 + 1e-12);
        const double skipS2 = (l >= 1) ? (cS * tl[0]) * (cS * tl[0]) * (1 - 1e-12) : -1.0;
        if (r2min > skipP2 || r2max < skipS2) continue;
        double K[6] = {0, 0, 0, 0, 0, 0};
        for (int q = 0; q < A.n_sub * A.n_sing; q++) {
            const double* bq = A.inner + 3 * q;
            double y[3];
            for (int c = 0; c < 3; c++) y[c] = bq[0] * VF[0][c] + bq[1] * VF[1][c] + bq[2] * VF[2][c];
            const double wq = A.win[q % A.n_sing] * aF;
            for (int o = 0; o < A.n_out; o++) {
                const double* bl = A.outer + 3 * o;
                double x[3];
                for (int c = 0; c < 3; c++) x[c] = y[c] - (bl[0] * VS[0][c] + bl[1] * VS[1][c] + bl[2] * VS[2][c]);
                const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
                if (r2 > skipP2 || r2 < skipS2) continue;
                const double r = sqrt(r2);
                const Win2 P = ghc_window2(r, cP, l, tl, dt), S = ghc_window2(r, cS, l, tl, dt);
                const double w = (A.wout[o] * aS) * wq;
                double nu[6];
                ghc_pair(nu, x, 1 / r, P.H, S.H, P.Q - S.Q, icP2, icS2);
#pragma unroll
                for (int e = 0; e < 6; e++) K[e] += w * nu[e];
            }
        }
        double* base = A.E + (size_t)(l - A.lag0) * A.ld_lag + (3 * (size_t)j) * n3 + 3 * (size_t)i;
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int r = 0; r < 3; r++) {
                const double v = K[map[3 * c + r]];
                if (fabs(v) > 1.0e-14) base[c * n3 + r] += v / A.c4pirho;
            }
    }
}

// Warp per (source, field) pair.  Bound by instruction issue: 8200 warp
// instructions a pair at 336 node pairs, of which the items 3200, the arrival
// levels and the sort 1600, the reductions and sums per lag 2500; 57 % of the
// issue slots are used with 16 warps an SM (126 registers; 80 registers and 24
// warps: 1.23 ms against 0.99 for 4 blocks at rule 7/4/3, 12 warps 1.14).  The
// form before evaluated every node pair in every lag between its P and S
// arrival.  Sphere of 320 triangles, 40 lags, rule 7/16/3: 6.6 -> 1.3 ms,
// 7/4/3: 2.4 -> 0.92; sphere of 1280, 7/16/3: 76 -> 16.5 ms; bar of 2800,
// lags 40..59, 7/4/3: 96 -> 42 ms.
//
// Node pair (inner node q, outer node o) at
// distance r meets front X (P, S) at the first level k with t_k > r / c_X.  The
// second difference (levels l-1, l, l+1 of t_k = k dt, kernelGHC.cu:88-99) of
// the kernel kernelGHC.cu:204-259 (nucleo), H = [t > r/c] and Q = (t^2 -
// r^2/c^2) H per front, is then, with sigma = 1 for P and -1 for S,
//   lag k - 1:   Hm + Q_k T,      lag k:  -Hm + ((2k + 1) dt^2 - Q_k) T,
//   lags > k:    2 dt^2 T,
//   T = sigma (3/2 ir^5 x x^T - 1/2 ir^3 I),
//   Hm = sigma ir^3/c^2 x x^T (+ ir/c^2 I for S),
// and zero before.  The items (node pair, front) are sorted by k
// (front_bins.cuh) and evaluated once each; cur and nxt collect the lags k - 1
// and k, run every lag from k - 1 on, which the other two take back where the
// constant does not hold yet.  A warp reduction per lag adds into the pair's
// sums in shared memory (node pairs beyond kBinChunk in further chunks).
constexpr int kGHCWarps = 4;
constexpr size_t kGHCSmem = 200 * 1024;    // of a block at most; the opt-in of every launch, so that threads' calls do not lower each other's

inline __host__ __device__ int ghc_chunk(int n_in, int n_out) {        // inner nodes of one chunk
    const int q = kBinChunk / n_out;
    return q < n_in ? q : n_in;
}
inline __host__ __device__ size_t ghc_warp_bytes(int n_in, int n_out, int lag0, int nlag) {
    const size_t b = (size_t)(4 * (ghc_chunk(n_in, n_out) + n_out) + 6 * ((nlag + 1) / 2 * 2)) * sizeof(double) + front_bins_bytes(bin_window(lag0, nlag).bins);
    return (b + 15) / 16 * 16;
}

__global__ void __launch_bounds__(32 * kGHCWarps, 4) ghc_assemble_kernel(GHCArgs A) {
    extern __shared__ __align__(16) unsigned char ghc_smem[];
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    const int n_in = A.n_sub * A.n_sing, chunk = ghc_chunk(n_in, A.n_out);
    const int lend = A.lag0 + A.nlag - 1;
    const BinWindow win = bin_window(A.lag0, A.nlag);
    // nodes (x, y, z, weight), sums (6 per lag), bins
    double* ys = reinterpret_cast<double*>(ghc_smem + (threadIdx.x >> 5) * ghc_warp_bytes(n_in, A.n_out, A.lag0, A.nlag));
    double* xs = ys + 4 * chunk;
    double* acc = xs + 4 * A.n_out;
    FrontBins B = front_bins_at(reinterpret_cast<unsigned char*>(acc + 6 * ((A.nlag + 1) / 2 * 2)), win.bins);
    const float iout = 1.0f / (float)A.n_out;          // (np + 1/2) iout: exact quotient for np < kBinChunk
    const double cP = A.velP, cS = A.velS, dt = A.dt, dt2 = dt * dt;
    const double icdtP = 1 / (cP * dt), icdtS = 1 / (cS * dt);
    const double icP2 = 1 / (cP * cP), icS2 = 1 / (cS * cS), ic4 = 1 / A.c4pirho;
    const size_t n3 = A.ld;
    for (long long p = warp; p < (long long)A.N * A.N; p += nwarps) {
        const int j = (int)((p <= 0xffffffffLL) ? (long long)((unsigned)p / (unsigned)A.N) : p / A.N);      // field (inner rule)
        const int i = (int)(p - (long long)j * A.N);                                                    // source (outer rule)
        if (i == j) continue;
        // before the P front in every lag: nodes lie within 2/3 of the longest side from the centroid
        const TriGeom &GS = A.geo[i], &GF = A.geo[j];
        const double e0 = GS.ctr[0] - GF.ctr[0], e1 = GS.ctr[1] - GF.ctr[1], e2 = GS.ctr[2] - GF.ctr[2];
        const double reach = (lend + 1) * dt * cP + 0.66667 * (GS.maxL + GF.maxL);
        if (reach * reach * (1 + 1e-9) < e0 * e0 + e1 * e1 + e2 * e2) continue;
        double VS[3][3], VF[3][3];
        for (int v = 0; v < 3; v++)
            for (int c = 0; c < 3; c++) {
                VS[v][c] = A.coords[3 * A.tris[3 * i + v] + c];
                VF[v][c] = A.coords[3 * A.tris[3 * j + v] + c];
            }
        double distMax = 0;
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++) {
                double d0 = VS[a][0] - VF[b][0], d1 = VS[a][1] - VF[b][1], d2 = VS[a][2] - VF[b][2];
                distMax = fmax(distMax, d0 * d0 + d1 * d1 + d2 * d2);
            }
        distMax = sqrt(distMax);
        // lags computed: not null, i.e. (l-1) c_S dt <= distMax
        int lhi = lend;
        while (lhi >= A.lag0 && (lhi - 1) * A.velS * A.dt > distMax) lhi--;
        if (lhi < A.lag0) continue;
        const double aS = A.geo[i].area, aF = A.geo[j].area;
        __syncwarp();
        for (int o = lane; o < A.n_out; o += 32) {
            const double* b = A.outer + 3 * o;
#pragma unroll
            for (int c = 0; c < 3; c++) xs[4 * o + c] = b[0] * VS[0][c] + b[1] * VS[1][c] + b[2] * VS[2][c];
            xs[4 * o + 3] = A.wout[o] * aS;
        }
        for (int t = lane; t < 6 * A.nlag; t += 32) acc[t] = 0.0;
        __syncwarp();
        bool any = false;
        for (int q0 = 0; q0 < n_in; q0 += chunk) {
            const int nq = min(chunk, n_in - q0), n = nq * A.n_out;
            for (int q = lane; q < nq; q += 32) {
                const double* b = A.inner + 3 * (size_t)(q0 + q);
#pragma unroll
                for (int c = 0; c < 3; c++) ys[4 * q + c] = b[0] * VF[0][c] + b[1] * VF[1][c] + b[2] * VF[2][c];
                ys[4 * q + 3] = A.win[(q0 + q) % A.n_sing] * aF;
            }
            __syncwarp();
            bool late = false, met = false;
            for (int t = lane; t < n; t += 32) {
                const int q = (int)(((float)t + 0.5f) * iout), o = t - q * A.n_out;
                const double x0 = ys[4 * q] - xs[4 * o], x1 = ys[4 * q + 1] - xs[4 * o + 1], x2 = ys[4 * q + 2] - xs[4 * o + 2];
                const double r2 = x0 * x0 + x1 * x1 + x2 * x2, r = q_sqrt(r2);
                unsigned bP = front_bin(r2, r, cP, icdtP, dt, win);
                unsigned bS = front_bin(r2, r, cS, icdtS, dt, win);
                if (bS == 0) bP = bS = kNoBin;                    // past both fronts before the window: the constants cancel
                else late = late || bS == kNoBin;
                met = met || bP != kNoBin;
                B.bin[t] = make_ushort2((unsigned short)bP, (unsigned short)bS);
            }
            if (!__any_sync(0xffffffffu, met)) continue;            // both fronts miss the window
            late = __any_sync(0xffffffffu, late);
            any = true;
            const int total = bins_sort(B, n, win.bins, lane);
            double cur[6] = {0, 0, 0, 0, 0, 0}, nxt[6] = {0, 0, 0, 0, 0, 0}, run[6] = {0, 0, 0, 0, 0, 0};
            double last = 0.0;                        // this lane's reduced entry of the lag before
            const double tail = 2 * dt2;
            int first = B.off[0], idle = 0;           // idle: bins without items up to this one
            for (int t = lane; t < first; t += 32) {  // bin 0: the constant only
                const unsigned it = B.list[t];
                const int np = (int)(it & 0x7fffffffu), q = (int)(((float)np + 0.5f) * iout), o = np - q * A.n_out;
                const double x0 = ys[4 * q] - xs[4 * o], x1 = ys[4 * q + 1] - xs[4 * o + 1], x2 = ys[4 * q + 2] - xs[4 * o + 2];
                const double r2 = x0 * x0 + x1 * x1 + x2 * x2, ir = q_rcp(q_sqrt(r2)), ir3 = ir * ir * ir;
                const double w = xs[4 * o + 3] * ys[4 * q + 3], sw = it >> 31 ? -w : w;
                const double fT = sw * 1.5 * ir3 * ir * ir, dT = -0.5 * sw * ir3;
                const double xx[6] = {x0 * x0, x0 * x1, x0 * x2, x1 * x1, x1 * x2, x2 * x2};
                if (r2 > 0)
#pragma unroll
                    for (int e = 0; e < 6; e++) run[e] += tail * (fT * xx[e] + ((e == 0 || e == 3 || e == 5) ? dT : 0.0));
            }
            for (int b = 1; b < win.bins; b++) {
                const int k = win.kbase + b - 1, lastitem = B.off[b], items = lastitem - first;
                if (items == 0 && first == 0) continue;                 // before the first arrival
                idle = items ? 0 : idle + 1;
                const double tk2 = (k * dt) * (k * dt), step = (2 * k + 1) * dt2;
                for (int t = first + lane; t < lastitem; t += 32) {
                    const unsigned it = B.list[t];
                    const bool isS = it >> 31;
                    const int np = (int)(it & 0x7fffffffu), q = (int)(((float)np + 0.5f) * iout), o = np - q * A.n_out;
                    const double x0 = ys[4 * q] - xs[4 * o], x1 = ys[4 * q + 1] - xs[4 * o + 1], x2 = ys[4 * q + 2] - xs[4 * o + 2];
                    const double r2 = x0 * x0 + x1 * x1 + x2 * x2, ir = q_rcp(q_sqrt(r2));
                    const double w = xs[4 * o + 3] * ys[4 * q + 3], ic2 = isS ? icS2 : icP2;
                    const double ir3 = ir * ir * ir, sw = isS ? -w : w;
                    const double Q = tk2 - r2 * ic2;
                    // entries 11, 12, 13, 22, 23, 33 of x x^T times f plus I times d
                    const double fT = sw * 1.5 * ir3 * ir * ir, dT = -0.5 * sw * ir3;
                    const double fH = sw * ir3 * ic2, dH = isS ? w * ir * ic2 : 0.0;
                    const double xx[6] = {x0 * x0, x0 * x1, x0 * x2, x1 * x1, x1 * x2, x2 * x2};
                    const double e1 = Q - tail, e2 = step - Q - tail;
#pragma unroll
                    for (int e = 0; e < 6; e++) {
                        const bool diag = e == 0 || e == 3 || e == 5;
                        const double T = fT * xx[e] + (diag ? dT : 0.0), H = fH * xx[e] + (diag ? dH : 0.0);
                        cur[e] += H + e1 * T;
                        nxt[e] += e2 * T - H;
                        if (r2 > 0) run[e] += tail * T;       // r = 0: both fronts here at once, no constant remains
                    }
                }
                const int l = k - 1;
                if (l >= A.lag0 && l <= lhi) {
                    if (idle < 3 || l == A.lag0) {
                        double v[8];
#pragma unroll
                        for (int e = 0; e < 6; e++) v[e] = cur[e] + run[e];
                        v[6] = v[7] = 0.0;
                        last = warp_reduce_scatter8(v, lane);
                    }
                    const int e = scatter8_entry(lane);
                    if ((lane & 3) == 0 && e < 6) acc[(l - A.lag0) * 6 + e] += last;
                }
                first = lastitem;
#pragma unroll
                for (int e = 0; e < 6; e++) {
                    cur[e] = nxt[e];
                    nxt[e] = 0.0;
                }
                if (!late && first == total && items == 0) break;       // every node pair is past both fronts
            }
            __syncwarp();
        }
        if (!any) continue;
        const int map[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
        double* base = A.E + (3 * (size_t)j) * n3 + 3 * (size_t)i;
        for (int t = lane; t < 9 * (lhi - A.lag0 + 1); t += 32) {
            const int l = t / 9, e = t - 9 * l, c = e / 3, r = e - 3 * c;
            const double v = acc[6 * l + map[e]];
            if (fabs(v) > 1.0e-14) base[(size_t)l * A.ld_lag + c * n3 + r] += v * ic4;
        }
    }
}

int launch_ghc_assemble(const MeshData& m, const PhysParams& P, int n_gh, int n_sub, int n_sing, int lag0, int nlag,
                        double* d_E, size_t ld, size_t ld_lag, cudaStream_t s) {
    double ob[28 * 3], ow[28];
    if (gh_composite(n_gh, 1, ob, ow)) return fail(EBEM_ERR_INVALID, "unsupported outer rule");
    std::vector<double> ib((size_t)3 * n_sub * n_sing), iw(n_sing);
    if (gh_composite(n_sing, n_sub, ib.data(), iw.data())) return fail(EBEM_ERR_INVALID, "unsupported inner rule");
    size_t nb = 3 * n_gh + n_gh + ib.size() + iw.size();
    std::vector<double> tab(nb);
    size_t o = 0;
    for (int k = 0; k < 3 * n_gh; k++) tab[o++] = ob[k];
    for (int k = 0; k < n_gh; k++) tab[o++] = ow[k];
    for (double v : ib) tab[o++] = v;
    for (double v : iw) tab[o++] = v;
    double* d_tab = nullptr;
    EBEM_CUDA_TRY(ws_malloc(&d_tab, nb * sizeof(double), s));
    if (cudaError_t e = cudaMemcpyAsync(d_tab, tab.data(), nb * sizeof(double), cudaMemcpyHostToDevice, s)) {
        ws_free(d_tab, s);
        return fail(EBEM_ERR_CUDA, std::string("rule table upload: ") + cudaGetErrorString(e));
    }
    GHCArgs A;
    A.coords = m.d_coords;
    A.tris = m.d_tris;
    A.geo = m.d_geo;
    A.outer = d_tab;
    A.wout = d_tab + 3 * n_gh;
    A.inner = d_tab + 4 * n_gh;
    A.win = d_tab + 4 * n_gh + ib.size();
    A.n_out = n_gh;
    A.n_sub = n_sub;
    A.n_sing = n_sing;
    A.N = m.nt;
    A.velP = P.velP;
    A.velS = P.velS;
    A.dt = P.dt;
    A.c4pirho = 4 * kPi * P.rho;
    A.lag0 = lag0;
    A.nlag = nlag;
    A.E = d_E;
    A.ld = ld;
    A.ld_lag = ld_lag;
    const long long NN = (long long)m.nt * m.nt;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m.device);
    cudaError_t e = cudaSuccess;
    const long long np = (long long)n_gh * n_sub * n_sing;
    // A pair costs the thread kernel time in proportion to the node pairs, the
    // warp kernel mostly the lags: equal at about 20 node pairs on 700 triangles
    // and 1280 (9 node pairs: 1.9 against 3.2 ms and 4.3 against 8.8; 36: 5.8
    // against 3.5 and 13.7 against 9.6).  Below 48 pairs an SM and node pair
    // the threads do not fill the chip (3 node pairs: 80 triangles 0.15 ms
    // against 0.08, 252 triangles 0.28 against 0.42).
    // On windows of few lags the threads' time falls with the lags and the sort of
    // the node pairs stays: 36 node pairs, lags from the middle of the run, 1 and 4
    // of them 3.2 and 10.4 ms by threads against 12.6 and 16.9 on 2800 triangles
    // (12 lags 28.5 against 27.0), 0.57 and 1.80 against 1.28 and 1.98 on 1280,
    // 0.11 and 0.29 against 0.16 and 0.23 on 320; 84 node pairs, 1 lag 6.3 against
    // 14.6, 1.10 against 1.46 and 0.19 against 0.18.
    const bool byThread = (np <= 24 && NN >= 48LL * sms * np) ||
                          (NN >= 256LL * sms && nlag * (np * (1 + 3.0 * sms / m.nt) - 20) < 190);
    if (byThread) {
        ghc_assemble_thread_kernel<<<(unsigned)((NN + 127) / 128), 128, 0, s>>>(A);
        e = cudaGetLastError();
    }
    for (int l0 = 0; !byThread && l0 < nlag && e == cudaSuccess; l0 += kBinLags) {
        A.lag0 = lag0 + l0;
        A.nlag = nlag - l0 < kBinLags ? nlag - l0 : kBinLags;
        A.E = d_E + (size_t)l0 * ld_lag;
        const size_t each = ghc_warp_bytes(n_sub * n_sing, n_gh, A.lag0, A.nlag);
        int warps = kGHCWarps;
        while (warps > 1 && warps * each > kGHCSmem) warps--;
        const size_t smem = warps * each;
        e = cudaFuncSetAttribute(ghc_assemble_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGHCSmem);
        if (e != cudaSuccess) break;
        const long long want = (NN + warps - 1) / warps, cap = (long long)sms * 64;
        ghc_assemble_kernel<<<(unsigned)(want < cap ? want : cap), 32 * warps, smem, s>>>(A);
        e = cudaGetLastError();
    }
    ws_free(d_tab, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail(EBEM_ERR_CUDA, std::string("numerical-inner assembly: ") + cudaGetErrorString(e));
    return EBEM_OK;
}

}  // namespace ebem
