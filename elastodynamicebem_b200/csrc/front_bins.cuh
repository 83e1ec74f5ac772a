// Node pairs of one (row, column) pair of triangles sorted by the time level at
// which a front reaches them, for the window differences of the numerical
// assemblies (ghc.cu, direct.cu).
//
// The lag-l entry of those operators is a second or third difference of
// functions of t that vanish before a front's arrival at t = r / c and are
// polynomials after it.  So a node pair contributes through each front to two
// or three lags next to the first level k with t_k > r / c, and a constant to
// every later lag.  A warp finds k for every (node pair, front), sorts them by
// k (a counting sort with __match_any, so the order and with it the sums are
// the same in every run) and takes the items level by level, 32 at a time:
// each item is evaluated once, where an evaluation per lag repeats it for every
// lag between the P and the S arrival.
#pragma once

#include "sa_device.cuh"

namespace ebem {

constexpr int kBinChunk = 512;              // node pairs sorted at a time
constexpr int kBinLags = 512;               // lags of one launch at most (the host goes on with the next ones)
constexpr unsigned kNoBin = 0xffffu;

// Bins of a window of nlag lags from lag0 on.  Bin b >= 1 holds the items of
// level k = kbase + b - 1, kbase = max(lag0 - 1, 0); bin 0 those of earlier
// levels, which reach the window with their constant only.  Levels past the
// window have none.
struct BinWindow {
    int kbase, bins;                        // bins 0 .. bins - 1
};
__host__ __device__ inline BinWindow bin_window(int lag0, int nlag) {
    BinWindow w;
    w.kbase = lag0 > 0 ? lag0 - 1 : 0;
    w.bins = lag0 + nlag - w.kbase + 2;     // up to level lag0 + nlag
    return w;
}

// t_k = k dt, rounded before anything is subtracted from it or it from anything:
// contracted to a fused multiply-add the difference would be the product's
// rounding error where a front meets a distance exactly at a level, and the front
// one level early.
__device__ __forceinline__ double level_time(int k, double dt) { return __dmul_rn((double)k, dt); }

// Bin of the first level k >= 0 with k dt - r / c > 0, as the reference tests it
// in IEEE arithmetic (sqrt, quotient, product, difference).  r2 = r^2, icdt =
// 1 / (c dt).  Away from the whole numbers r icdt decides alone: its error is a
// few units in the last place, the margin 1e-9 of it; so the two quotients and
// the root in IEEE arithmetic are paid by one node pair in 1e8.
__device__ __forceinline__ unsigned front_bin(double r2, double r, double c, double icdt, double dt, const BinWindow& w) {
    const int most = w.kbase + w.bins - 2;
    const double g = r * icdt;
    if (!(g < (double)most + 1.0)) return kNoBin;
    int k = (int)g + 1;
    if (fabs(g - rint(g)) <= 1e-9 * g + 1e-12) {
        const double tX = sqrt(r2) / c;
        k = max(k - 3, 0);
        while (k <= most && !(level_time(k, dt) - tX > 0)) k++;
    }
    return k > most ? kNoBin : k < w.kbase ? 0u : (unsigned)(k - w.kbase + 1);
}

// Shared memory of one warp.
struct FrontBins {
    int* off;                   // per bin: count, then offset
    ushort2* bin;               // kBinChunk: P, S bin of a node pair
    unsigned* list;             // 2 kBinChunk items: node pair | front << 31 (S)
};

__host__ __device__ inline size_t front_bins_bytes(int bins) {
    return ((size_t)bins * sizeof(int) + 15) / 16 * 16 + kBinChunk * (sizeof(ushort2) + 2 * sizeof(unsigned));
}

__device__ __forceinline__ FrontBins front_bins_at(unsigned char* p, int bins) {
    FrontBins b;
    b.off = reinterpret_cast<int*>(p);
    p += ((size_t)bins * sizeof(int) + 15) / 16 * 16;
    b.bin = reinterpret_cast<ushort2*>(p);
    b.list = reinterpret_cast<unsigned*>(p + kBinChunk * sizeof(ushort2));
    return b;
}

// One front of 32 node pairs: count them per bin, or put them into the list
// (off then runs through each bin's items).
template <bool SCATTER>
__device__ __forceinline__ void bins_step(FrontBins& B, unsigned b, unsigned item, int lane) {
    const unsigned same = __match_any_sync(0xffffffffu, b);
    const int rank = __popc(same & ((1u << lane) - 1u));
    int at = 0;
    if (b != kNoBin) at = B.off[b];
    __syncwarp();
    if (b != kNoBin) {
        if (SCATTER) B.list[at + rank] = item;
        if (rank == 0) B.off[b] = at + __popc(same);
    }
    __syncwarp();
}

// Sorts the n <= kBinChunk node pairs whose bins are in B.bin; afterwards the
// items of bin b are list[(b ? off[b - 1] : 0) .. off[b]).  Returns their number.
__device__ __forceinline__ int bins_sort(FrontBins& B, int n, int bins, int lane) {
    for (int b = lane; b < bins; b += 32) B.off[b] = 0;
    __syncwarp();
    for (int q0 = 0; q0 < n; q0 += 32) {
        const int q = q0 + lane;
        const ushort2 v = q < n ? B.bin[q] : make_ushort2(kNoBin, kNoBin);
        bins_step<false>(B, v.x, 0, lane);
        bins_step<false>(B, v.y, 0, lane);
    }
    int total = 0;
    for (int b0 = 0; b0 < bins; b0 += 32) {
        const int b = b0 + lane;
        const int v = b < bins ? B.off[b] : 0;
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (b < bins) B.off[b] = total + x - v;
        total += __shfl_sync(0xffffffffu, x, 31);
    }
    __syncwarp();
    for (int q0 = 0; q0 < n; q0 += 32) {
        const int q = q0 + lane;
        const ushort2 v = q < n ? B.bin[q] : make_ushort2(kNoBin, kNoBin);
        bins_step<true>(B, v.x, (unsigned)q, lane);
        bins_step<true>(B, v.y, (unsigned)q | 0x80000000u, lane);
    }
    return total;
}

// Warp sums of 8 per-lane values with 9 shuffles: lane l returns the sum of
// value 4 b4 + 2 b3 + b2 (b: bits of l).
__device__ __forceinline__ double warp_reduce_scatter8(double v[8], int lane) {
#pragma unroll
    for (int h = 4; h > 0; h >>= 1) {
        const int m = 4 * h;
        const bool up = (lane & m) != 0;
#pragma unroll
        for (int k = 0; k < h; k++) {
            const double send = up ? v[k] : v[k + h], keep = up ? v[k + h] : v[k];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, m);
        }
    }
    double x = v[0];
    x += __shfl_xor_sync(0xffffffffu, x, 2);
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    return x;
}
__device__ __forceinline__ int scatter8_entry(int lane) {
    return ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
}

}  // namespace ebem
