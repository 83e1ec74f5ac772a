// Semi-analytic assembly of dense outputs in two passes.
//
// Pass 1 (sa_level_kernel with block records, sa_assemble.cu): one warp per
// (source, field) pair walks the pair's time levels and stores the 6
// symmetric entries of
//   E_l = (F_{l+1} - 2 F_l + F_{l-1}) / (4 pi rho), clean-up |x| < 1e-14 -> 0
// (calcMatrixSubBlock.m:15,23,101-104,111; calcMatrixBlock.m:77) at its
// non-null lags, and those lags (llo, lhi; the null test of
// BEMenerg_coreSA_calcMatrixBlock.m:57-61).
//
// Pass 2 (sa_emit_kernel): every entry of the window's blocks, zero outside
// the pair's non-null lags, written (or added) one thread per block with
// consecutive threads on consecutive sources: the output is written in whole
// sectors, zeros included.  Written by the level kernel itself, each block is
// 24-byte column pieces scattered 3N doubles apart.
//
// The record buffer holds, per chunk of field columns, (columns) x (lags) x
// (sources) x 6 doubles plus one int2 per pair; the columns are split into
// equal chunks that keep it in L2.
#include "ebem_internal.h"

#include <algorithm>
#include <atomic>
#include <mutex>

namespace ebem {

namespace {
// Per-pass device times of the two-pass assembly (ebem_profile_*): CUDA
// events around each launch on the call's stream, read at the end of the call.
std::atomic<int> g_profile{0};
std::mutex g_prof_mu;
double g_prof_ms[2] = {0.0, 0.0};        // pass 1 (levels), pass 2 (emission)
long long g_prof_n[2] = {0, 0};
}  // namespace

void profile_enable(int on) { g_profile.store(on ? 1 : 0); }

void profile_read(double ms[2], long long n[2], int reset) {
    std::lock_guard<std::mutex> lock(g_prof_mu);
    for (int k = 0; k < 2; k++) {
        ms[k] = g_prof_ms[k];
        n[k] = g_prof_n[k];
        if (reset) { g_prof_ms[k] = 0.0; g_prof_n[k] = 0; }
    }
}

// The window's blocks from the records of one chunk of field columns: one
// thread per (source, field, lag) block, consecutive threads on consecutive
// sources of one field column, so each of the 9 stores of a warp covers one
// contiguous 768-byte run of a column (the three row stores of a column fill
// it completely); the records are read as 16-byte pairs.
__global__ void __launch_bounds__(128) sa_emit_kernel(const double* __restrict__ rec, const int2* __restrict__ band,
                                                      int nsrc, int j0, int lag0, int nlag, double* __restrict__ E,
                                                      size_t ld, size_t ld_lag, int accumulate) {
    const int ii = blockIdx.x * blockDim.x + threadIdx.x;
    if (ii >= nsrc) return;
    const int jj = blockIdx.y, q = blockIdx.z, l = lag0 + q;
    const int2 b = band[(long long)jj * nsrc + ii];
    double v[6] = {0, 0, 0, 0, 0, 0};
    if (b.x >= 0 && l >= b.x && l <= b.y) {
        const double2* p = reinterpret_cast<const double2*>(rec + (((long long)jj * nlag + q) * nsrc + ii) * 6);
#pragma unroll
        for (int h = 0; h < 3; h++) { const double2 t = p[h]; v[2 * h] = t.x; v[2 * h + 1] = t.y; }
    }
    // (r, c) -> symmetric entry 11, 12, 13, 22, 23, 33
    const int sym[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
    double* base = E + (size_t)q * ld_lag + 3 * (size_t)(j0 + jj) * ld + 3 * (size_t)ii;
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int r = 0; r < 3; r++) {
            double* dst = base + (size_t)c * ld + r;
            const double x = v[sym[3 * c + r]];
            if (accumulate) *dst += x;
            else *dst = x;
        }
}

int launch_sa_twopass(const MeshData& m, const PhysParams& P, int n_gh, int lag0, int nlag, int src0, int nsrc,
                      double* d_E, size_t ld, size_t ld_lag, int accumulate, unsigned long long* d_count,
                      cudaStream_t s, const unsigned char* cls, const ClassTable* classes) {
    if (classes && (src0 != 0 || nsrc != m.nt)) return fail(EBEM_ERR_INVALID, "a class array needs all source rows");
    if (m.nt > 65535 || nlag > 65535) return fail(EBEM_ERR_INVALID, "mesh or lag window too large for one launch");
    const size_t fbytes = (size_t)nlag * nsrc * 6 * sizeof(double);
    const size_t per_col = fbytes + (size_t)nsrc * sizeof(int2);
    // equal chunks of field columns whose records stay in L2 (126 MB) until the
    // emission pass reads them: sphere of 1280 triangles, L = 40, GH7, in MB
    // of records: 64 11.9 ms, 96 11.6, 128 11.4, 256 11.8, 512 12.3, 1536
    // 12.9 (below 128 the launches' tails cost what L2 gains)
    const size_t budget = (size_t)128 << 20;
    const int most = (int)std::max<size_t>(1, std::min<size_t>((size_t)m.nt, budget / per_col));
    const int chunks = (m.nt + most - 1) / most;
    int cols = (m.nt + chunks - 1) / chunks;
    double* Fb = nullptr;
    while (ws_malloc(&Fb, per_col * cols, s) != cudaSuccess) {
        // a device with less to spare: fewer columns at a time
        if (cols == 1) return fail(EBEM_ERR_NOMEM, "assembly workspace allocation failed");
        cols = (cols + 1) / 2;
    }
    int2* band = reinterpret_cast<int2*>(reinterpret_cast<unsigned char*>(Fb) + fbytes * cols);
    const bool prof = g_profile.load() != 0;
    std::vector<cudaEvent_t> ev;
    auto mark = [&]() {
        if (!prof) return;
        cudaEvent_t e = nullptr;
        if (cudaEventCreate(&e) == cudaSuccess && cudaEventRecord(e, s) == cudaSuccess) ev.push_back(e);
        else if (e) cudaEventDestroy(e);
    };
    int rc = EBEM_OK;
    mark();
    for (int j0 = 0; j0 < m.nt && rc == EBEM_OK; j0 += cols) {
        const int nj = std::min(cols, m.nt - j0);
        rc = launch_sa_records(m, P, n_gh, lag0, nlag, src0, nsrc, j0, nj, Fb, band, d_count, s, cls, classes);
        if (rc) break;
        mark();
        dim3 grid((unsigned)((nsrc + 127) / 128), (unsigned)nj, (unsigned)nlag);
        sa_emit_kernel<<<grid, 128, 0, s>>>(Fb, band, nsrc, j0, lag0, nlag, d_E, ld, ld_lag, accumulate);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) rc = fail(EBEM_ERR_CUDA, std::string("emission kernel: ") + cudaGetErrorString(e));
        mark();
    }
    ws_free(Fb, s);
    if (prof) {
        // events alternate: start, after pass 1, after pass 2, after pass 1, ...
        double add[2] = {0.0, 0.0};
        long long cnt[2] = {0, 0};
        if (rc == EBEM_OK && !ev.empty() && cudaEventSynchronize(ev.back()) == cudaSuccess) {
            for (size_t k = 1; k < ev.size(); k++) {
                float ms = 0.0f;
                if (cudaEventElapsedTime(&ms, ev[k - 1], ev[k]) == cudaSuccess) {
                    add[(k - 1) & 1] += ms;
                    cnt[(k - 1) & 1]++;
                }
            }
        }
        for (cudaEvent_t e : ev) cudaEventDestroy(e);
        cudaGetLastError();
        std::lock_guard<std::mutex> lock(g_prof_mu);
        for (int k = 0; k < 2; k++) {
            g_prof_ms[k] += add[k];
            g_prof_n[k] += cnt[k];
        }
    }
    return rc;
}

}  // namespace ebem
