// Inverse of a dense matrix for the marching (E_0^{-1}): blocked Gauss-Jordan
// elimination with partial pivoting, in place of the LU factors and n
// triangular solves of the reference's lu(sparse(matrix))
// (f/BEMenerg_indir/BEMenerg_core/BEMenerg_coreSA/BEMenerg_coreSA_timeMarching.m:46,59).
//
// A panel of 64 columns K is eliminated over all n rows by one thread-block
// cluster (gj_panel_kernel), each thread one row in registers: per column the
// largest entry of the rows not yet used is the pivot, found by warp
// reductions, one exchange of the blocks' candidates (value and row) through
// distributed shared memory and one cluster barrier.  Rows are not swapped: the
// pivot rows P are remembered.  The panel then holds C = A(:,K) A(P,K)^{-1}
// (negated off the rows P, the inverse on them), and every other column
// follows with one product (gj_update_kernel):
//   A'(:, o) = A(:, o) [rows P: 0] + C A(P, o),
// out of place between two buffers that stay in L2.  After the last panel row
// p holds the unknown k(p) and column k the right-hand side entry p(k):
//   inverse(k(p), p(k')) = A'(p, k').
//
// Bound: the serial chain of n pivots, 1.3 us each whatever the number of
// blocks (of it, per ncu, block and cluster barriers and the release of the
// remote stores about 40 %); 64 columns move A half as often as 32 (n = 2100:
// 4.6 against 4.7 ms).  Against the library's LU and n triangular solves (one
// marching step each): n = 258 0.90 -> 0.52 ms, 858 3.1 -> 1.5, 1440 5.2 -> 2.7,
// 2100 9.3 -> 4.7, 3840 22.9 -> 15.3.
#include "ebem_internal.h"
#include "sa_math.cuh"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace ebem {

constexpr int kGJCols = 64, kGJThreads = 256, kGJMaxCluster = 16;

struct GJSlot {
    double row[kGJCols];
    unsigned hi, r;             // upper half of |pivot candidate|, its row
};

__global__ void __launch_bounds__(kGJThreads, 1) gj_panel_kernel(const double* __restrict__ A, int n, int k0, int nb,
                                                                 double* __restrict__ Pn, int* __restrict__ piv,
                                                                 int* __restrict__ used, int* __restrict__ info) {
    __shared__ GJSlot slot[2][kGJMaxCluster];
    __shared__ GJSlot mine;
    __shared__ unsigned whi[kGJThreads / 32], wrow[kGJThreads / 32];
    cg::cluster_group cl = cg::this_cluster();
    const int cr = (int)cl.block_rank(), cs = (int)cl.num_blocks();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int row = cr * kGJThreads + (int)threadIdx.x;
    const bool valid = row < n;
    double a[kGJCols];
#pragma unroll
    for (int c = 0; c < kGJCols; c++) a[c] = (valid && c < nb) ? A[(size_t)(k0 + c) * n + row] : 0.0;
    bool open = valid && used[valid ? row : 0] < 0;
    int col = -1, bad = 0;
    cl.sync();          // every block has started before another writes to it
#pragma unroll 1
    for (int j = 0; j < nb; j++) {
        // the current column is a[0]; the columns rotate by one per pivot
        const unsigned hi = open ? (unsigned)__double2hiint(fabs(a[0])) + 1u : 0u;     // 0: no candidate
        const unsigned m = __reduce_max_sync(0xffffffffu, hi);
        const int win = __ffs(__ballot_sync(0xffffffffu, hi == m)) - 1;
        if (lane == win) {
            whi[w] = m;
            wrow[w] = (unsigned)row;
        }
        __syncthreads();
        const unsigned v = lane < kGJThreads / 32 ? whi[lane] : 0u;
        const unsigned M = __reduce_max_sync(0xffffffffu, v);
        const int bw = __ffs(__ballot_sync(0xffffffffu, lane < kGJThreads / 32 && v == M)) - 1;
        const unsigned R = wrow[bw];
        if (row == (int)R) {
#pragma unroll
            for (int c = 0; c < kGJCols; c++) mine.row[c] = a[c];
            mine.hi = M;
            mine.r = R;
        }
        __syncthreads();
        GJSlot* buf = slot[j & 1];
        for (int t = w; t < cs; t += kGJThreads / 32) {
            GJSlot* to = cl.map_shared_rank(buf, t) + cr;
#pragma unroll
            for (int c = 0; c < kGJCols; c += 32) to->row[c + lane] = mine.row[c + lane];
            if (lane == 0) {
                to->hi = mine.hi;
                to->r = mine.r;
            }
        }
        cl.sync();
        const unsigned g = lane < cs ? buf[lane].hi : 0u;
        const unsigned G = __reduce_max_sync(0xffffffffu, g);
        const int who = __ffs(__ballot_sync(0xffffffffu, lane < cs && g == G)) - 1;
        const double* p = buf[who].row;
        const int R2 = (int)buf[who].r;
        const double q = q_rcp(p[0]);
        if (row == R2) {
            if (p[0] == 0.0 && bad == 0) bad = k0 + j + 1;
#pragma unroll
            for (int c = 0; c < kGJCols - 1; c++) a[c] = p[c + 1] * q;
            a[kGJCols - 1] = q;
            open = false;
            col = k0 + j;
        } else {
            const double f = -a[0] * q;
#pragma unroll
            for (int c = 0; c < kGJCols - 1; c++) a[c] = fma(f, p[c + 1], a[c + 1]);
            a[kGJCols - 1] = f;
        }
    }
    if (valid) {
        // (no global stores inside the loop: the cluster barrier would wait for them)
        if (col >= 0) {
            used[row] = col;
            piv[col] = row;
        }
        if (bad) atomicMin(info, bad);
        // after nb rotations column b is a[kGJCols - nb + b]
#pragma unroll
        for (int c = 0; c < kGJCols; c++)
            if (c >= kGJCols - nb) Pn[(size_t)(c - (kGJCols - nb)) * n + row] = a[c];
    }
    cl.sync();          // no block leaves while another may still write to it
}

constexpr int kGJTileR = 128, kGJTileC = 64, kGJStep = 32;
__global__ void __launch_bounds__(256, 2) gj_update_kernel(const double* __restrict__ A, double* __restrict__ B, int n, int k0,
                                                           int nb, const double* __restrict__ Pn, const int* __restrict__ piv,
                                                           const int* __restrict__ used) {
    __shared__ double sp[kGJStep][kGJTileR];
    __shared__ double sr[kGJStep][kGJTileC];
    const int r0 = blockIdx.x * kGJTileR, c0 = blockIdx.y * kGJTileC;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    // The panel's products are summed by themselves and added to A once: its entries
    // are rounded n / 64 times, not n times (n = 1500, a diagonal of size 1 beside small
    // entries: solutions 2.0e-15 off -> below 9e-16).  A read after the products,
    // 16 loads in flight, instead of before them also leaves the block a shorter
    // start (n = 3840 15.56 -> 15.28 ms; one load at a time 20.4).
    double acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.0;
    for (int b0 = 0; b0 < nb; b0 += kGJStep) {
        __syncthreads();
        for (int t = threadIdx.x; t < kGJStep * kGJTileR; t += 256) {
            const int b = t / kGJTileR, r = t - b * kGJTileR;
            sp[b][r] = (b0 + b < nb && r0 + r < n) ? Pn[(size_t)(b0 + b) * n + r0 + r] : 0.0;
        }
        for (int t = threadIdx.x; t < kGJStep * kGJTileC; t += 256) {
            const int c = t / kGJStep, b = t - c * kGJStep;
            sr[b][c] = (b0 + b < nb && c0 + c < n) ? A[(size_t)(c0 + c) * n + piv[k0 + b0 + b]] : 0.0;
        }
        __syncthreads();
#pragma unroll 4
        for (int b = 0; b < kGJStep; b++) {
            double x[8], y[4];
#pragma unroll
            for (int i = 0; i < 8; i++) x[i] = sp[b][tx + 16 * i];
#pragma unroll
            for (int j = 0; j < 4; j++) y[j] = sr[b][ty + 16 * j];
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fma(x[i], y[j], acc[i][j]);
        }
    }
    unsigned open = 0;                                 // rows but this panel's pivots, which start from 0
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int r = r0 + tx + 16 * i;
        if (r < n && used[r] < k0) open |= 1u << i;
    }
#pragma unroll
    for (int h = 0; h < 4; h += 2) {                   // 16 loads in flight
        double base[2][8];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int c = c0 + ty + 16 * (h + j), b = c - k0;
            const bool panel = b >= 0 && b < nb;
            const double* from = panel ? Pn + (size_t)b * n : A + (size_t)c * n;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int r = r0 + tx + 16 * i;
                base[j][i] = (c < n && r < n && (panel || (open >> i & 1u))) ? from[r] : 0.0;
            }
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int c = c0 + ty + 16 * (h + j), b = c - k0;
            if (c >= n) continue;
            const bool panel = b >= 0 && b < nb;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int r = r0 + tx + 16 * i;
                if (r < n) B[(size_t)c * n + r] = panel ? base[j][i] : base[j][i] + acc[i][h + j];
            }
        }
    }
}

// inverse(k(p), p(k')) = M(p, k'): thread per (p, k'), p fastest.
__global__ void gj_unscramble_kernel(const double* __restrict__ M, int n, const int* __restrict__ piv,
                                     const int* __restrict__ used, double* __restrict__ inv) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
    if (p < n) inv[(size_t)piv[k] * n + used[p]] = M[(size_t)k * n + p];
}

int gj_max_n() { return kGJThreads * kGJMaxCluster; }

// d_inv = A^{-1} (device, column-major n x n, n <= gj_max_n()); *singular: the
// number of the first zero pivot, 0 for none.  Waits for the stream.  *placed is
// false, and nothing has run, when the device cannot hold the panel's cluster
// (more than 8 blocks are not portable, and a context may be given a part of the
// SMs) or the two buffers (LU needs one).
int gj_inverse(const double* dA, int n, double* d_inv, int* singular, bool* placed, cudaStream_t s) {
    const size_t nn = (size_t)n * n;
    const unsigned cluster = (unsigned)((n + kGJThreads - 1) / kGJThreads);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(cluster);
    cfg.blockDim = dim3(kGJThreads);
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int resident = 0;
    *placed = (cluster <= 8 || cudaFuncSetAttribute(gj_panel_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
              cudaOccupancyMaxActiveClusters(&resident, gj_panel_kernel, &cfg) == cudaSuccess && resident > 0;
    if (!*placed) {
        cudaGetLastError();
        return EBEM_OK;
    }
    double* buf = nullptr;
    int* idx = nullptr;
    if (ws_malloc(&buf, (2 * nn + (size_t)n * kGJCols) * sizeof(double), s) != cudaSuccess ||
        ws_malloc(&idx, (2 * (size_t)n + 1) * sizeof(int), s) != cudaSuccess) {
        cudaGetLastError();
        ws_free(buf, s);
        *placed = false;
        return EBEM_OK;
    }
    double* Pn = buf + 2 * nn;
    int *piv = idx, *used = idx + n, *info = idx + 2 * n;
    cudaError_t e = cudaMemsetAsync(idx, 0xff, 2 * (size_t)n * sizeof(int), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(info, 0x7f, sizeof(int), s);      // 0x7f7f7f7f: none
    const dim3 tiles((unsigned)((n + kGJTileR - 1) / kGJTileR), (unsigned)((n + kGJTileC - 1) / kGJTileC));
    const double* cur = dA;
    for (int k0 = 0, t = 0; k0 < n && e == cudaSuccess; k0 += kGJCols, t ^= 1) {
        const int nb = n - k0 < kGJCols ? n - k0 : kGJCols;
        e = cudaLaunchKernelEx(&cfg, gj_panel_kernel, cur, n, k0, nb, Pn, piv, used, info);
        if (e != cudaSuccess) break;
        double* nxt = buf + (size_t)t * nn;
        gj_update_kernel<<<tiles, 256, 0, s>>>(cur, nxt, n, k0, nb, Pn, piv, used);
        e = cudaGetLastError();
        cur = nxt;
    }
    if (e == cudaSuccess) {
        gj_unscramble_kernel<<<dim3((unsigned)((n + 255) / 256), (unsigned)n), 256, 0, s>>>(cur, n, piv, used, d_inv);
        e = cudaGetLastError();
    }
    int h = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, info, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    ws_free(buf, s);
    ws_free(idx, s);
    if (e != cudaSuccess) return fail(EBEM_ERR_CUDA, std::string("matrix inverse: ") + cudaGetErrorString(e));
    *singular = h == 0x7f7f7f7f ? 0 : h;
    return EBEM_OK;
}

}  // namespace ebem
