// Device preparation of the mesh and the semi-analytic (SA) assembly kernel.
//
// Reference (paths relative to the reference project root; "SA/" =
// functions/BEMenerg_indir/BEMenerg_core/BEMenerg_coreSA/):
//   mesh fields      functions/utility/fileRead/readSpaceMesh.m:93-148
//   frame            SA/calcoloMatrice/operazioniGeometriche/calcoloSistemaRiferimento.m
//   Euler matrix     SA/calcoloMatrice/operazioniGeometriche/rotazioneInversaEulero.m:23-176
//   mapped nodes     SA/BEMenerg_coreSA_calcCostantData.m:8-23
//   null test        SA/calcoloMatrice/BEMenerg_coreSA_calcMatrixBlock.m:57-61, clean-up :77
//   sub-block        SA/calcoloMatrice/BEMenerg_coreSA_calcMatrixSubBlock.m:1-111
//   projection       SA/calcoloMatrice/operazioniGeometriche/preparazioneTriangolo.m:1-115
//   edge distance    SA/calcoloMatrice/operazioniGeometriche/calcoloDistanzaTriangolo.m
//   children         SA/calcoloMatrice/BEMenerg_coreSA_calcIntgInt_fieldTriangle.m:13-84
//
// Work decomposition (B200 design, not the reference's): one warp per
// (source i, field j) pair.  F(t_k), the combined kernel integral at one
// instant, depends on k only, so each level is evaluated once and E_l =
// F_{l+1} - 2 F_l + F_{l-1} is formed from three levels (the reference
// evaluates every instant three times, once per lag that uses it).  For dense
// outputs the blocks are kept as records and written in a second, coalesced pass
// (sa_twopass.cu); the other modes write them directly.
#include "ebem_internal.h"

#include <algorithm>
#include <mutex>
#include <type_traits>
#include "sa_group.cuh"

namespace ebem {

// ---------------------------------------------------------------------------
// mesh preparation

__global__ void prep_kernel(const double* __restrict__ coords, const int32_t* __restrict__ tris, int nt,
                            TriGeom* __restrict__ geo) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nt) return;
    double V[3][3];
    for (int v = 0; v < 3; v++) {
        int id = tris[3 * t + v];
        for (int c = 0; c < 3; c++) V[v][c] = coords[3 * id + c];
    }
    TriGeom g;
    tri_geom(V, g);
    geo[t] = g;
}

__global__ void map_nodes_kernel(const double* __restrict__ coords, const int32_t* __restrict__ tris, int nt,
                                 const TriGeom* __restrict__ geo, const double* __restrict__ bary,
                                 const double* __restrict__ w, int n_gh, NodeW* __restrict__ out) {
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nt * n_gh) return;
    int t = idx / n_gh, g = idx % n_gh;
    double V[3][3];
    for (int v = 0; v < 3; v++) {
        int id = tris[3 * t + v];
        for (int c = 0; c < 3; c++) V[v][c] = coords[3 * id + c];
    }
    double b0 = bary[3 * g], b1 = bary[3 * g + 1], b2 = bary[3 * g + 2];
    NodeW o;
    o.x = b0 * V[0][0] + b1 * V[1][0] + b2 * V[2][0];
    o.y = b0 * V[0][1] + b1 * V[1][1] + b2 * V[2][1];
    o.z = b0 * V[0][2] + b1 * V[1][2] + b2 * V[2][2];
    o.w = geo[t].area * w[g];
    out[idx] = o;
}

// Outer rule passed by value (no device table).
struct RuleParam {
    double b[28][3];
    double w[28];
};

__global__ void map_nodes_param_kernel(const double* __restrict__ coords, const int32_t* __restrict__ tris, int nt,
                                       const TriGeom* __restrict__ geo, RuleParam rule, int n_gh,
                                       NodeW* __restrict__ out) {
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nt * n_gh) return;
    int t = idx / n_gh, g = idx % n_gh;
    double V[3][3];
    for (int v = 0; v < 3; v++) {
        int id = tris[3 * t + v];
        for (int c = 0; c < 3; c++) V[v][c] = coords[3 * id + c];
    }
    const double b0 = rule.b[g][0], b1 = rule.b[g][1], b2 = rule.b[g][2];
    NodeW o;
    o.x = b0 * V[0][0] + b1 * V[1][0] + b2 * V[2][0];
    o.y = b0 * V[0][1] + b1 * V[1][1] + b2 * V[2][1];
    o.z = b0 * V[0][2] + b1 * V[1][2] + b2 * V[2][2];
    o.w = geo[t].area * rule.w[g];
    out[idx] = o;
}

int prep_mesh(MeshData& m, cudaStream_t s) {
    int threads = 128, blocks = (m.nt + threads - 1) / threads;
    prep_kernel<<<blocks, threads, 0, s>>>(m.d_coords, m.d_tris, m.nt, m.d_geo);
    EBEM_CUDA_TRY(cudaGetLastError());
    return EBEM_OK;
}

int map_nodes(MeshData& m, int n_gh, cudaStream_t s) {
    static const int kSlotRule[MeshData::kNodeRules] = {1, 3, 7, 12, 19, 28};
    int slot = -1;
    for (int k = 0; k < MeshData::kNodeRules; k++)
        if (kSlotRule[k] == n_gh) slot = k;
    if (slot < 0) return fail(EBEM_ERR_INVALID, "unsupported Gauss-Hammer rule");
    if (NodeW* t = m.d_node_tables[slot]) {
        m.d_nodes = t;
        m.nodes_rule = n_gh;
        return EBEM_OK;
    }
    RuleParam rule;
    if (int rc = gh_composite(n_gh, 1, &rule.b[0][0], rule.w)) return fail(rc, "unsupported Gauss-Hammer rule");
    // the table enters the cache only once the mapping has finished, so a
    // failed call leaves no half-built table behind
    NodeW* table = nullptr;
    if (store_malloc(&table, sizeof(NodeW) * (size_t)m.nt * n_gh, s) != cudaSuccess)
        return fail(EBEM_ERR_NOMEM, "outer-node table allocation failed");
    const int total = m.nt * n_gh;
    map_nodes_param_kernel<<<(total + 127) / 128, 128, 0, s>>>(m.d_coords, m.d_tris, m.nt, m.d_geo, rule, n_gh, table);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        ws_free(table, s);
        return fail(EBEM_ERR_CUDA, std::string("outer-node mapping: ") + cudaGetErrorString(e));
    }
    m.d_node_tables[slot] = table;
    m.d_nodes = table;
    m.nodes_rule = n_gh;
    return EBEM_OK;
}

int map_nodes_composite(MeshData& m, int n_gh, int n_sub, cudaStream_t s) {
    if (n_sub == 1) return map_nodes(m, n_gh, s);
    const int key = n_gh * 4096 + n_sub;
    for (int k = 0; k < MeshData::kCompRules; k++)
        if (m.d_comp_tables[k] && m.comp_key[k] == key) {
            m.d_nodes = m.d_comp_tables[k];
            m.nodes_rule = n_gh * n_sub;
            return EBEM_OK;
        }
    int slot = -1;
    for (int k = 0; k < MeshData::kCompRules && slot < 0; k++)
        if (!m.d_comp_tables[k]) slot = k;
    if (slot < 0) return fail(EBEM_ERR_INVALID, "too many composite outer rules cached on one mesh");
    if (n_sub < 1 || n_sub > 1024) return fail(EBEM_ERR_INVALID, "composite rule: n_sub out of range");
    const int nn = n_gh * n_sub;
    std::vector<double> bary(3 * (size_t)nn), w((size_t)nn), wb(n_gh);
    int rc = gh_composite(n_gh, n_sub, bary.data(), wb.data());
    if (rc) return fail(rc, "unsupported composite Gauss-Hammer rule (n_sub must be a square)");
    for (int q = 0; q < n_sub; q++)
        for (int g = 0; g < n_gh; g++) w[(size_t)q * n_gh + g] = wb[g];
    NodeW* table = nullptr;
    double* d_tab = nullptr;
    if (cudaMalloc(&table, sizeof(NodeW) * (size_t)m.nt * nn) != cudaSuccess ||
        cudaMalloc(&d_tab, sizeof(double) * 4 * (size_t)nn) != cudaSuccess) {
        cudaGetLastError();
        if (table) cudaFree(table);
        return fail(EBEM_ERR_NOMEM, "outer-node table allocation failed");
    }
    cudaError_t e = cudaMemcpyAsync(d_tab, bary.data(), sizeof(double) * 3 * nn, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(d_tab + 3 * (size_t)nn, w.data(), sizeof(double) * nn, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        const long long total = (long long)m.nt * nn;
        const int threads = 128;
        map_nodes_kernel<<<(unsigned)((total + threads - 1) / threads), threads, 0, s>>>(
            m.d_coords, m.d_tris, m.nt, m.d_geo, d_tab, d_tab + 3 * (size_t)nn, nn, table);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(d_tab);
    if (e != cudaSuccess) {
        cudaFree(table);
        return fail(EBEM_ERR_CUDA, std::string("outer-node mapping: ") + cudaGetErrorString(e));
    }
    m.d_comp_tables[slot] = table;
    m.comp_key[slot] = key;
    m.d_nodes = table;
    m.nodes_rule = nn;
    return EBEM_OK;
}

// ---------------------------------------------------------------------------
// assembly

struct SAArgs {
    const TriGeom* geo = nullptr;
    const NodeW* nodes = nullptr;
    int N = 0, n_gh = 0;
    double velP = 0, velS = 0, dt = 0, ic4 = 0;   // ic4 = 1 / (4 pi rho)
    int lag0 = 0, nlag = 0;
    int src0 = 0, nsrc = 0; // source rows [src0, src0 + nsrc) of the panel
    int j0 = 0, nj = 0;     // field columns [j0, j0 + nj)
    int diag_only = 0;      // 1: only the diagonal pairs (i, i), i in the panel
    const int2* pairs = nullptr;   // optional explicit (source, field) list (npairs entries)
    long long npairs = 0;
    unsigned long long* count = nullptr;
    // dense output, column-major 3 nsrc x 3N per lag
    double* E = nullptr;
    size_t ld = 0;          // leading dimension (>= 3 nsrc)
    size_t ld_lag = 0;      // doubles between consecutive lags
    int accumulate = 0;
    int zeros_written = 0;  // the buffer is zeroed already: only the band's blocks are written
    // banded output (instead of E): pair p = (i - src0) N + j owns the blocks
    // [boff[p], boff[p+1]) of Eb, one per lag of its band starting at blo[p],
    // 6 symmetric entries (11,12,13,22,23,33) each
    double* Eb = nullptr;
    const long long* boff = nullptr;
    const int* blo = nullptr;
    // block records (instead of E), written at the non-null lags only: the 6
    // entries of lag l of pair (i, j) at Lout[(((j - j0) nlag + l - lag0) nsrc
    // + i - src0) 6], of pair p of a list at Lout[(p nlag + l - lag0) 6]; the
    // non-null lags (llo, lhi) at band[(j - j0) nsrc + i - src0] when asked for
    double* Lout = nullptr;
    int2* band = nullptr;
    // classes of a per-(pair, lag) class array: cls[(j N + i) nlag + l - lag0]
    const unsigned char* cls = nullptr;
    // derived (sa_args_derive)
    double k1 = 0, ks = 0, icP = 0, icS = 0;   // 1 / c_P^2, 1 / c_S^2, 1 / (c_P dt), 1 / (c_S dt)
};

EBEM_HDI void sa_args_derive(SAArgs& A) {
    A.k1 = 1.0 / (A.velP * A.velP);
    A.ks = 1.0 / (A.velS * A.velS);
    A.icP = 1.0 / (A.velP * A.dt);
    A.icS = 1.0 / (A.velS * A.dt);
}

__device__ __forceinline__ void store_entry(const SAArgs& A, int q, int i, int j, int e, double v) {
    // entry e = 3 c + r of the column-major 3x3 block at (3(i - src0), 3j)
    const int c = e / 3, r = e - 3 * c;
    double* dst = A.E + (size_t)q * A.ld_lag + (3 * (size_t)j + c) * A.ld + 3 * (size_t)(i - A.src0) + r;
    if (A.accumulate) *dst += v;
    else *dst = v;
}


// ---------------------------------------------------------------------------
// Level kernel: F(t_k) of one (source, field) pair per warp, from the closed
// form of sa_front.cuh.
//
// * Lane = child of an outer node: level-independent data of the child
//   (fields in shared memory, one column per child) and the two level ranges
//   of each front, [kA, kN): from the first level at which the front meets
//   the side to the first at which it has passed the node's whole triangle.
// * Item = (level, front, child) with the level in that range: the children's
//   ranges become two bit masks per level (ballots), the masks' population
//   counts number the items level by level, and the 32 lanes take 32 items
//   at a time whatever their level, front or child, all on one path
//   (front_item).  On the sphere of 1280 triangles a pair has some 130
//   items, where the lanes of one level's children would be a third busy.
// * The items' seven values go through shared memory into per-level sums,
//   lane = (level, entry), always in item order: a level's sum does not
//   depend on where the 32-item rounds fall, so any lag window or row panel
//   gives the same bits.
// * Lane = level: the nodes a front has passed wholly add a + t^2 b, summed
//   over the node's children beforehand; split children add their constants
//   between the arrivals of P and S at the foot; nodes that project inside the
//   field triangle add V(rho) x (angle); then the rotation to global axes.
//   (The split costs 1 to 2 %, sphere of 1280 triangles 10.83 -> 10.94 ms, prism
//   of 252 with GH12 0.670 -> 0.684, for 2 to 4 times less rounding.)
// Outer rules with more than 10 nodes run in equal groups of at most 10; levels
// in chunks of 32.
//
// Bound: FP64 issue (an item's two logarithms, two arctangents, two square
// roots and one division, sa_math.cuh).  Sphere of 320 triangles, L = 40,
// GH7 (ncu): issue active 57 %, FP64 pipe 40 %, stalls per issued
// instruction 1.8 on fixed latencies and 0.3 on instruction fetch.  Per
// assembly, against the kernel that integrated the edge pieces by
// Gauss-Legendre and decided each child's pieces at each level (lane = child,
// FP64 pipe 22 %, 3 to 4 stalls on instruction fetch): sphere of 1280
// triangles 159.4 -> 10.8 ms, of 320 12.8 -> 0.93 ms, prism of 252 with GH12
// 8.9 -> 0.69 ms.  On the way (1280 triangles): closed form with the library's
// functions out of line 24.6 ms, inlined 29.4; sa_math.cuh, one division per
// evaluation and 32-bit pair indices 13.0; blocks as records that stay in L2
// (sa_twopass.cu) 11.1; the level masks by a bit transpose 10.8.  The IEEE
// divisions of the second difference alone cost 2.0 ms (their slow path's
// code), hence ic4.  Launch shape: 8 warps, 2 blocks per SM (128 registers);
// 4 x 4 13.3 against 13.0 ms, 4 x 3 13.5, 16 x 1 13.2, 12 x 1 13.1.
constexpr int kLevelChunk = 32;  // levels per chunk: one lane per level

#ifndef EBEM_LEVEL_WPB
#define EBEM_LEVEL_WPB 8
#endif
#ifndef EBEM_LEVEL_MINB
#define EBEM_LEVEL_MINB 2
#endif

struct LevelShared {
    FrontGroup W;
    double res[32][7];                       // the round's items
    double acc[kLevelChunk][7];              // per-level sums
    unsigned long long mask[kLevelChunk];    // items of a level: P children, S children << 32
    double carry[2][6];                      // direct output: F of the two levels before the chunk
    int kP[kGroupNodes], kS[kGroupNodes];    // first level at which the front has passed the whole triangle
    int2 kf[kSlots];                         // first levels at which P and S have passed the foot of a split child
    int off[kLevelChunk + 1];                // first item of each level
};

// Position of the n-th set bit (n counted from 0) of m.
EBEM_DI int nth_bit(unsigned m, int n) {
    int pos = 0;
#pragma unroll
    for (int h = 16; h > 0; h >>= 1) {
        const int c = __popc(m & ((1u << h) - 1u));
        if (n >= c) {
            n -= c;
            pos += h;
            m >>= h;
        }
    }
    return pos;
}

// pair_band by a warp, one lag per lane.
EBEM_DI void pair_band_warp(const TriGeom& F, const TriGeom& S, double velP, double velS, double dt, int lag0, int nlag,
                            int lane, int* llo, int* lhi) {
    const double v0 = F.ctr[0] - S.ctr[0], v1 = F.ctr[1] - S.ctr[1], v2 = F.ctr[2] - S.ctr[2];
    const double d = sqrt(v0 * v0 + v1 * v1 + v2 * v2);
    const double distMin = d - F.maxL - S.maxL;
    const double distMax = d + F.maxL + S.maxL;
    *llo = -1;
    *lhi = -2;
    for (int q0 = 0; q0 < nlag; q0 += 32) {
        const int l = lag0 + q0 + lane;
        const unsigned on = __ballot_sync(0xffffffffu, q0 + lane < nlag && lag_nonnull(l, velP, velS, dt, distMin, distMax));
        if (on) {
            if (*llo < 0) *llo = lag0 + q0 + __ffs(on) - 1;
            *lhi = lag0 + q0 + 31 - __clz(on);
        }
    }
}

// Bits [max(lo, 0), min(hi, 32)).
EBEM_DI unsigned level_bits(int lo, int hi) {
    lo = max(lo, 0);
    hi = min(hi, 32);
    return hi > lo ? (0xffffffffu >> (32 - (hi - lo))) << lo : 0u;
}

// 32 x 32 bit transpose over a warp: bit k of lane i becomes bit i of lane k.
EBEM_DI unsigned transpose32(unsigned x, int lane) {
    unsigned m = 0x0000ffffu;
#pragma unroll
    for (int j = 16; j > 0; j >>= 1, m ^= m << j) {
        const unsigned y = __shfl_xor_sync(0xffffffffu, x, j);
        x = (lane & j) ? ((x & ~m) | ((y >> j) & m)) : ((x & m) | ((y & m) << j));
    }
    return x;
}

// Whether level k is used by a lag of class c (lags k-1, k, k+1 of the pair's
// non-null range [llo, lhi]).
EBEM_DI bool level_wanted(const SAArgs& A, const unsigned char* cls, int c, int k, int llo, int lhi) {
    for (int l = max(k - 1, llo); l <= min(k + 1, lhi); l++)
        if (cls[l - A.lag0] == c) return true;
    return false;
}

// The dynamic shared memory opt-in of a kernel, before every launch that is
// not being captured: it belongs to the context, which a caller may have
// reset since the last call; a captured launch relies on the uncaptured one
// before it (the batch plan runs its launch before capturing it).
template <class K>
static int opt_in_smem(K kernel, size_t smem, cudaStream_t s) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &st) == cudaSuccess && st != cudaStreamCaptureStatusNone) return EBEM_OK;
    EBEM_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return EBEM_OK;
}

// Output of a launch: dense blocks, the banded layout, or block records.
enum : int { OUT_DENSE, OUT_BANDED, OUT_RECORDS };

// Pair p of the launch: (source i, field j).  With classes (CLS) the pair's
// levels are walked once for each class its lags have, with that class's
// rule.
template <int OUT, bool CLS>
__device__ __forceinline__ void level_pair(const SAArgs& A, const ClassTable* T, LevelShared& Ls, long long p, int i, int j,
                                           int lane, unsigned long long& my_count) {
    const TriGeom& F = A.geo[j];
    const TriGeom& Sg = A.geo[i];
    int llo = -1, lhi = -2;
    long long bbase = 0;
    if (OUT == OUT_BANDED) {
        // banded output: the band comes from the structure pass, so writes stay in the pair's blocks
        const long long pb = (long long)(i - A.src0) * A.N + j;
        bbase = A.boff[pb];
        const int nb = (int)(A.boff[pb + 1] - bbase);
        if (nb > 0) {
            llo = A.blo[pb];
            lhi = llo + nb - 1;
        }
    } else {
        pair_band_warp(F, Sg, A.velP, A.velS, A.dt, A.lag0, A.nlag, lane, &llo, &lhi);
    }
    if (OUT == OUT_RECORDS && A.band && lane == 0)
        A.band[(long long)(j - A.j0) * A.nsrc + (i - A.src0)] = make_int2(llo, lhi);
    // direct dense output: the zeros of the window's lags outside the band
    if (OUT == OUT_DENSE && !A.accumulate && !A.zeros_written) {
        for (int idx = lane; idx < A.nlag * 9; idx += 32) {
            const int q = idx / 9, e = idx - 9 * q, l = A.lag0 + q;
            if (llo < 0 || l < llo || l > lhi) store_entry(A, q, i, j, e, 0.0);
        }
    }
    if (llo < 0) return;
    if (lane == 0) my_count += (unsigned long long)(lhi - llo + 1);
    const long long rec = A.pairs ? p * A.nlag : (long long)(j - A.j0) * A.nlag * A.nsrc + (i - A.src0);
    const long long rstride = A.pairs ? 1 : A.nsrc;
    const unsigned char* cls = CLS ? A.cls + ((long long)j * A.N + i) * A.nlag : nullptr;
    const double k1 = A.k1, ks = A.ks;
    int klo = max(1, llo - 1), khi = lhi + 1;
    const int ncls = CLS ? T->n : 1;
    unsigned present = 1u;                     // classes of the pair's lags, class 31 and above in bit 31
    if (CLS) {
        present = 0u;
        for (int l = llo + lane; l <= lhi; l += 32) present |= 1u << min((int)cls[l - A.lag0], 31);
        present = __reduce_or_sync(0xffffffffu, present);
    }
    for (int ic = 0; ic < ncls; ic++) {
        const NodeW* nodes = A.nodes;
        int n_gh = A.n_gh;
        if (CLS) {
            if (!((present >> min(ic, 31)) & 1u)) continue;
            // the class's first and last lag bound its levels
            int first = -1, last = -1;
            for (int l0 = llo; l0 <= lhi; l0 += 32) {
                const unsigned on = __ballot_sync(0xffffffffu, l0 + lane <= lhi && cls[min(l0 + lane, lhi) - A.lag0] == ic);
                if (on) {
                    if (first < 0) first = l0 + __ffs(on) - 1;
                    last = l0 + 31 - __clz(on);
                }
            }
            if (first < 0) continue;
            klo = max(1, first - 1);
            khi = last + 1;
            nodes = T->nodes[ic];
            n_gh = T->n_gh[ic];
        }
        __syncwarp();
        if (lane < 12) (&Ls.carry[0][0])[lane] = 0.0;
        const int ngroups = (n_gh + kGroupNodes - 1) / kGroupNodes, gsize = (n_gh + ngroups - 1) / ngroups;
        // this lane's child: level ranges of its items, zeta; circ: nodes with an angle (bit 3 g)
        int kaP = 0, knP = 0, kaS = 0, knS = 0;
        double zeta = 0.0;
        bool work = false;
        unsigned circ = 0, split = 0;          // split: children whose constants are apart (bit 3 g + c)
        for (int kc0 = klo; kc0 <= khi; kc0 += kLevelChunk) {
            const int nk = min(khi - kc0 + 1, kLevelChunk);
            __syncwarp();
#pragma unroll
            for (int e = 0; e < 7; e++) Ls.acc[lane][e] = 0.0;
            const bool wanted = lane < nk && (!CLS || level_wanted(A, cls, ic, kc0 + lane, llo, lhi));
            for (int grp = 0; grp < ngroups; grp++) {
                const int g0 = gsize * grp, gn = min(gsize, n_gh - g0);
                if (ngroups > 1 || kc0 == klo) {
                    __syncwarp();
                    FrontLane C;
                    const int g = lane / 3, c = lane - 3 * g;
                    group_geometry(C, g < gn, nodes + (size_t)i * n_gh + g0 + min(g, gn - 1), &F, lane);
                    zeta = C.G.zeta;
                    kaP = C.live ? front_level(C.near, A.icP, khi + 1) : khi + 1;
                    kaS = C.live ? front_level(C.near, A.icS, khi + 1) : khi + 1;
                    knP = front_level(C.all, A.icP, khi + 1);
                    knS = front_level(C.all, A.icS, khi + 1);
                    const int k0 = C.maybe ? front_level(q_sqrt(C.G.dMIN * C.G.dMIN + zeta * zeta), A.icP, khi + 1) : kaP;
                    work = __ballot_sync(0xffffffffu, C.child && min(k0, kaP) <= khi) != 0u;
                    if (work) {
                        circ = group_fields(Ls.W, C, lane);
                        split = __ballot_sync(0xffffffffu, C.split);
                        if (C.split) Ls.kf[lane] = make_int2(min(kaP, knP), min(kaS, knS));
                        if (C.child && c == 0) {
                            Ls.kP[g] = knP;
                            Ls.kS[g] = knS;
                        }
                    }
                }
                if (!work) continue;
                // items of each level: this child's levels, transposed to the level's children
                unsigned mP = level_bits(kaP - kc0, knP - kc0), mS = level_bits(kaS - kc0, knS - kc0);
                unsigned odd = 0;                      // children with a level at which c_S t == zeta: no front
                if (zeta != 0.0) {
                    const int kd = (int)rint(zeta * A.icS), b = kd - kc0;
                    if (b >= 0 && b < 32 && A.velS * (kd * A.dt) == zeta) {
                        mP &= ~(1u << b);
                        odd = 1;
                    }
                }
                odd = __ballot_sync(0xffffffffu, odd);
                mP = transpose32(mP, lane);
                mS = transpose32(mS, lane);
                if (!wanted) mP = mS = 0;
                const int n = __popc(mP) + __popc(mS);
                int incl = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += y;
                }
                const int total = __shfl_sync(0xffffffffu, incl, 31);
                Ls.mask[lane] = (unsigned long long)mP | ((unsigned long long)mS << 32);
                Ls.off[lane] = incl - n;
                if (lane == 31) Ls.off[32] = total;
                __syncwarp();
                for (int base = 0; base < total; base += 32) {
                    const int idx = min(base + lane, total - 1);
                    int lev = 0;                                       // last level with off <= idx that has items
#pragma unroll
                    for (int h = 16; h > 0; h >>= 1)
                        if (Ls.off[lev + h] <= idx) lev += h;
                    const unsigned long long m = Ls.mask[lev];
                    int r = idx - Ls.off[lev];
                    const int np = __popc((unsigned)m);
                    const bool isP = r < np;
                    const int slot = nth_bit(isP ? (unsigned)m : (unsigned)(m >> 32), isP ? r : r - np);
                    {
                        const double t = (kc0 + lev) * A.dt;
                        double T[7] = {0, 0, 0, 0, 0, 0, 0};
                        group_item(T, Ls.W, slot, !((split >> slot) & 1u), isP, (isP ? A.velP : A.velS) * t, isP ? k1 : ks);
#pragma unroll
                        for (int e = 0; e < 7; e++) Ls.res[lane][e] = T[e];
                    }
                    const int l0 = __shfl_sync(0xffffffffu, lev, 0), l1 = __shfl_sync(0xffffffffu, lev, 31);
                    __syncwarp();
                    const int e = lane & 7;
                    for (int lv = l0 + (lane >> 3); lv <= l1; lv += 4) {
                        const int i0 = max(Ls.off[lv] - base, 0), i1 = min(Ls.off[lv + 1] - base, 32);
                        if (e < 7 && i0 < i1) {
                            double v = Ls.acc[lv][e];
                            for (int q = i0; q < i1; q++) v += Ls.res[q][e];
                            Ls.acc[lv][e] = v;
                        }
                    }
                    __syncwarp();
                }
                // nodes the fronts have passed wholly, nodes with an angle: lane = level
                if (wanted) {
                    const int k = kc0 + lane;
                    const double t = k * A.dt, t2 = t * t, rP = A.velP * t, rS = A.velS * t;
                    double T[7];
#pragma unroll
                    for (int e = 0; e < 7; e++) T[e] = Ls.acc[lane][e];
                    for (unsigned m = split; m; m &= m - 1) {
                        const int slot = __ffs(m) - 1;
                        const int2 kf = Ls.kf[slot];
                        if (k >= kf.x && k < kf.y && (!((odd >> slot) & 1u) || Ls.W.zeta[slot / 3] != rS)) group_foot(T, Ls.W, slot, t2);
                    }
                    for (int g = 0; g < gn; g++) {
                        const double zg = Ls.W.zeta[g];
                        const bool cP = k >= Ls.kP[g] && (zg == 0.0 || zg != rS);
                        group_node(T, Ls.W, g, cP, k >= Ls.kS[g], (circ >> (3 * g)) & 1u, rP, rS, t2, k1, ks);
                    }
#pragma unroll
                    for (int e = 0; e < 7; e++) Ls.acc[lane][e] = T[e];
                }
            }
            // F(t_k) = (S I + C^T M C) / 2 in global axes, one lane per level
            double Fk[6] = {0, 0, 0, 0, 0, 0};
            if (wanted) {
                double T[7];
#pragma unroll
                for (int e = 0; e < 7; e++) T[e] = Ls.acc[lane][e];
                front_rotate(Fk, T, F.C);
            }
            // E_l = (F_{l+1} - 2 F_l + F_{l-1}) / (4 pi rho) for the lags l = k - 1
            // completed by the chunk's levels k, clean-up |x| < 1e-14
            // (calcMatrixSubBlock.m:15,23,111; calcMatrixBlock.m:77); F_0 = 0
            const int map[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
            const int l = kc0 + lane - 1;
            double b[6];
#pragma unroll
            for (int e = 0; e < 6; e++) Ls.acc[lane][e] = Fk[e];
            __syncwarp();
            // rows -2 and -1: the two levels before the chunk
            const double* r1 = lane >= 1 ? Ls.acc[lane - 1] : Ls.carry[1];
            const double* r2 = lane >= 2 ? Ls.acc[lane - 2] : Ls.carry[lane];
#pragma unroll
            for (int e = 0; e < 6; e++) {
                const double v = ((Fk[e] + (-2.0) * r1[e]) + r2[e]) * A.ic4;
                b[e] = (fabs(v) < 1.0e-14) ? 0.0 : v;
            }
            __syncwarp();
            if (lane >= 30) {
                // a further chunk follows a full one only
#pragma unroll
                for (int e = 0; e < 6; e++) Ls.carry[lane - 30][e] = Fk[e];
            }
            if (lane < nk && l >= llo && l <= lhi && (!CLS || cls[l - A.lag0] == ic)) {
                if (OUT != OUT_DENSE) {
                    double* dst = OUT == OUT_RECORDS ? A.Lout + (rec + (long long)(l - A.lag0) * rstride) * 6 : A.Eb + (bbase + (l - llo)) * 6;
                    if ((reinterpret_cast<size_t>(dst) & 15) == 0) {
                        double2* d2 = reinterpret_cast<double2*>(dst);
                        d2[0] = make_double2(b[0], b[1]);
                        d2[1] = make_double2(b[2], b[3]);
                        d2[2] = make_double2(b[4], b[5]);
                    } else {
                        // a caller's buffer off a 16-byte boundary
#pragma unroll
                        for (int e = 0; e < 6; e++) dst[e] = b[e];
                    }
                } else {
#pragma unroll
                    for (int e9 = 0; e9 < 9; e9++) store_entry(A, l - A.lag0, i, j, e9, b[map[e9]]);
                }
            }
            __syncwarp();
        }
    }
    // a class without a rule: the block is zero
    if (CLS)
        for (int l = llo + lane; l <= lhi; l += 32)
            if (cls[l - A.lag0] >= ncls)
                for (int e = 0; e < 6; e++) A.Lout[(rec + (long long)(l - A.lag0) * rstride) * 6 + e] = 0.0;
}

// Table: ClassTable, or NoClasses for the one rule of the arguments.
struct NoClasses {};
EBEM_DI const ClassTable* class_table(const ClassTable& T) { return &T; }
EBEM_DI const ClassTable* class_table(const NoClasses&) { return nullptr; }

template <int WPB, int MINB, int OUT, class Table>
__global__ void __launch_bounds__(32 * WPB, MINB) sa_level_kernel(SAArgs A, const __grid_constant__ Table T) {
    extern __shared__ __align__(16) unsigned char level_smem[];
    LevelShared* Lsh = reinterpret_cast<LevelShared*>(level_smem);
    __shared__ unsigned long long blk_count;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    LevelShared& Ls = Lsh[wib];
    if (threadIdx.x == 0) blk_count = 0;
    __syncthreads();
    const long long NP = A.pairs ? A.npairs : A.diag_only ? (long long)A.nsrc : (long long)A.nsrc * A.nj;
    const long long nwarps = (long long)gridDim.x * WPB;
    unsigned long long my_count = 0;
    const bool small = NP <= 0xffffffffLL;
    for (long long p = (long long)blockIdx.x * WPB + wib; p < NP; p += nwarps) {
        int i, j;
        if (A.pairs) {
            const int2 pj = A.pairs[p];
            i = pj.x;
            j = pj.y;
        } else {
            const long long q = A.diag_only ? 0 : small ? (long long)((unsigned)p / (unsigned)A.nsrc) : p / A.nsrc;
            i = A.src0 + (int)(p - q * A.nsrc);
            j = A.diag_only ? i : A.j0 + (int)q;
        }
        level_pair<OUT, std::is_same<Table, ClassTable>::value>(A, class_table(T), Ls, p, i, j, lane, my_count);
    }
    if (A.count) {
        if (lane == 0 && my_count) atomicAdd(&blk_count, my_count);
        __syncthreads();
        if (threadIdx.x == 0 && blk_count) atomicAdd(A.count, blk_count);
    }
}

template <int OUT, class Table>
static int launch_level(SAArgs A, const Table& T, long long NN, int device, cudaStream_t s) {
    constexpr int WPB = EBEM_LEVEL_WPB, MINB = EBEM_LEVEL_MINB;
    sa_args_derive(A);
    const size_t smem = sizeof(LevelShared) * WPB;
    if (int rc = opt_in_smem(sa_level_kernel<WPB, MINB, OUT, Table>, smem, s)) return rc;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    long long want = (NN + WPB - 1) / WPB;
    long long cap = (long long)sms * MINB * 16;
    unsigned blocks = (unsigned)(want < cap ? want : cap);
    if (blocks == 0) blocks = 1;
    sa_level_kernel<WPB, MINB, OUT, Table><<<blocks, 32 * WPB, smem, s>>>(A, T);
    EBEM_CUDA_TRY(cudaGetLastError());
    return EBEM_OK;
}

// All source rows and field columns of a mesh at lags [lag0, lag0 + nlag); the
// caller picks the output.
static SAArgs sa_args(const MeshData& m, const PhysParams& P, int n_gh, int lag0, int nlag) {
    SAArgs A;
    A.geo = m.d_geo;
    A.nodes = m.d_nodes;
    A.N = m.nt;
    A.n_gh = n_gh;
    A.velP = P.velP;
    A.velS = P.velS;
    A.dt = P.dt;
    A.ic4 = 1.0 / (4 * kPi * P.rho);
    A.lag0 = lag0;
    A.nlag = nlag;
    A.nsrc = m.nt;
    A.nj = m.nt;
    return A;
}

int launch_sa_diagonal(const MeshData& m, const PhysParams& P, int n_gh, int lag0, int nlag, double* d_E, size_t ld,
                       size_t ld_lag, cudaStream_t s) {
    SAArgs A = sa_args(m, P, n_gh, lag0, nlag);
    A.diag_only = 1;
    A.E = d_E;
    A.ld = ld;
    A.ld_lag = ld_lag;
    return launch_level<OUT_DENSE>(A, NoClasses(), m.nt, m.device, s);
}

int launch_sa_records(const MeshData& m, const PhysParams& P, int n_gh, int lag0, int nlag, int src0, int nsrc, int j0,
                      int nj, double* d_rec, int2* d_band, unsigned long long* d_count, cudaStream_t s,
                      const unsigned char* cls, const ClassTable* classes) {
    SAArgs A = sa_args(m, P, n_gh, lag0, nlag);
    A.src0 = src0;
    A.nsrc = nsrc;
    A.j0 = j0;
    A.nj = nj;
    A.count = d_count;
    A.Lout = d_rec;
    A.band = d_band;
    A.cls = cls;
    const long long NN = (long long)nsrc * nj;
    return classes ? launch_level<OUT_RECORDS>(A, *classes, NN, m.device, s)
                   : launch_level<OUT_RECORDS>(A, NoClasses(), NN, m.device, s);
}

// Blocks of an explicit list of (source, field) pairs at every lag [0, nlag)
// with the outer rule in m.d_nodes (n_gh nodes per triangle, composite or
// not): out[(p nlag + l) 6 + e], the 6 symmetric entries (11, 12, 13, 22, 23,
// 33) of E_l, zero outside the pair's non-null lags.
int launch_sa_pair_blocks(const MeshData& m, const PhysParams& P, int n_gh, const int2* d_pairs, long long npairs,
                          int nlag, double* d_out, cudaStream_t s) {
    if (npairs <= 0) return EBEM_OK;
    EBEM_CUDA_TRY(cudaMemsetAsync(d_out, 0, (size_t)npairs * nlag * 6 * sizeof(double), s));
    SAArgs A = sa_args(m, P, n_gh, 0, nlag);
    A.pairs = d_pairs;
    A.npairs = npairs;
    A.Lout = d_out;
    return launch_level<OUT_RECORDS>(A, NoClasses(), npairs, m.device, s);
}

// Banded output: all lags [0, L) of every pair, written into the band
// layout that band_structure() built.
int launch_sa_assemble_banded(const MeshData& m, const PhysParams& P, int n_gh, int L, double* d_Eb,
                              const long long* d_boff, const int* d_blo, cudaStream_t s) {
    SAArgs A = sa_args(m, P, n_gh, 0, L);
    A.Eb = d_Eb;
    A.boff = d_boff;
    A.blo = d_blo;
    return launch_level<OUT_BANDED>(A, NoClasses(), (long long)m.nt * m.nt, m.device, s);
}

// ---------------------------------------------------------------------------
// Assembly without device allocations (ebem_assemble_sa_noalloc).
//
// The ordinary assembly allocates two small device buffers of its own: the
// mapped outer nodes of the mesh (cached per rule) and, when the caller asks
// for the non-null count, an 8-byte counter.  This variant keeps both in one
// statically allocated device array, so that a call allocates nothing.  The
// array belongs to every GPU that loads the library until the process exits.
//
// Layout (bytes): [0, 8) counter, zeroed by each call that counts; from
// byte 256 on, the mapped node table, rewritten by each call.  Every call on
// a device shares the array: calls whose work overlaps on the GPU race.

constexpr size_t kNoAllocScratchBytes = size_t(1) << 20;        // 1 MiB per device
constexpr size_t kNoAllocNodeOffset = 256;
constexpr size_t kNoAllocMaxNodes = (kNoAllocScratchBytes - kNoAllocNodeOffset) / sizeof(NodeW);

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

size_t noalloc_max_nodes() { return kNoAllocMaxNodes; }

// Device address of the scratch array on the current device, looked up once
// per device (the host-side name of the array is not a device address) and
// again after ebem_device_release, whose caller may reset the device (a new
// context may place the array elsewhere).
static int noalloc_scratch(int device, unsigned char** out) {
    constexpr int kMaxDevices = 64;
    static unsigned char* addr[kMaxDevices] = {};
    static unsigned gen[kMaxDevices] = {};
    static std::mutex mu;
    if (device < 0 || device >= kMaxDevices) return fail(EBEM_ERR_INVALID, "device ordinal beyond the supported range");
    std::lock_guard<std::mutex> lock(mu);
    const unsigned g = device_generation(device);
    if (!addr[device] || gen[device] != g) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p)
            return fail(EBEM_ERR_CUDA, std::string("scratch address lookup failed: ") + cudaGetErrorString(e));
        addr[device] = (unsigned char*)p;
        gen[device] = g;
    }
    *out = addr[device];
    return EBEM_OK;
}

int launch_sa_assemble_noalloc(const MeshData& m, const PhysParams& P, int n_gh, int lag0, int nlag, double* d_E,
                               int accumulate, bool count, unsigned long long* host_count, cudaStream_t s) {
    if ((size_t)m.nt * n_gh > kNoAllocMaxNodes)
        return fail(EBEM_ERR_INVALID, "mesh too large for the allocation-free assembly: N x n_gh = " +
                                          std::to_string((long long)m.nt * n_gh) + " outer nodes, at most " +
                                          std::to_string(kNoAllocMaxNodes) + " fit in its 1 MiB scratch array");
    if (3 * n_gh > 64) return fail(EBEM_ERR_INVALID, "outer rule must have 3, 7, 12 or 19 nodes");
    unsigned char* base = nullptr;
    if (int rc = noalloc_scratch(m.device, &base)) return rc;
    unsigned long long* d_count = (unsigned long long*)base;
    NodeW* d_nodes = (NodeW*)(base + kNoAllocNodeOffset);
    RuleParam rule;
    if (int rc = gh_composite(n_gh, 1, &rule.b[0][0], rule.w)) return fail(rc, "unsupported Gauss-Hammer rule");
    const int total = m.nt * n_gh;
    map_nodes_param_kernel<<<(total + 127) / 128, 128, 0, s>>>(m.d_coords, m.d_tris, m.nt, m.d_geo, rule, n_gh, d_nodes);
    EBEM_CUDA_TRY(cudaGetLastError());
    if (count) EBEM_CUDA_TRY(cudaMemsetAsync(d_count, 0, sizeof(unsigned long long), s));
    SAArgs A = sa_args(m, P, n_gh, lag0, nlag);
    A.nodes = d_nodes;
    A.E = d_E;
    A.ld = 3 * (size_t)m.nt;
    A.ld_lag = A.ld * A.ld;
    A.accumulate = accumulate;
    A.count = count ? d_count : nullptr;
    int rc = launch_level<OUT_DENSE>(A, NoClasses(), (long long)m.nt * m.nt, m.device, s);
    if (rc) return rc;
    if (count) {
        EBEM_CUDA_TRY(cudaMemcpyAsync(host_count, d_count, sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
        EBEM_CUDA_TRY(cudaStreamSynchronize(s));
    }
    return EBEM_OK;
}

// ---------------------------------------------------------------------------
// Batched assembly: many meshes (instances) in one persistent launch.  Each
// warp grabs `chunk` consecutive pairs of the concatenated pair space
// (instance b owns pairs [pair_begin[b], pair_begin[b] + N_b^2)) from a global
// counter and assembles them with level_pair's per-pair walk (direct output),
// so a batch result equals the single-mesh results to rounding: per pair the
// per-level sums of level_pair, one lane per level forming F(t_k) and writing
// the blocks of the lags it completes.
template <int WPB, int MINB>
__global__ void __launch_bounds__(32 * WPB, MINB)
sa_batch_level_kernel(const BatchInst* __restrict__ insts, int ninst, long long total, int n_gh, int chunk,
                      unsigned long long* next) {
    extern __shared__ __align__(16) unsigned char batch_smem[];
    LevelShared* Lsh = reinterpret_cast<LevelShared*>(batch_smem);
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    LevelShared& Ls = Lsh[wib];
    __syncthreads();
    unsigned long long unused = 0;
    while (true) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(next, (unsigned long long)chunk);
        base = __shfl_sync(0xffffffffu, base, 0);
        if ((long long)base >= total) break;
        const long long end = min((long long)base + chunk, total);
        for (long long p = (long long)base; p < end; p++) {
            int lo = 0, hi = ninst - 1;                 // last instance with pair_begin <= p
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (insts[mid].pair_begin <= p) lo = mid;
                else hi = mid - 1;
            }
            const BatchInst& I = insts[lo];
            SAArgs A;
            A.geo = I.geo;
            A.nodes = I.nodes;
            A.N = I.N;
            A.n_gh = n_gh;
            A.velP = I.velP;
            A.velS = I.velS;
            A.dt = I.dt;
            A.ic4 = 1.0 / I.c4pirho;
            A.nlag = I.nlag;
            A.nsrc = I.N;
            A.nj = I.N;
            A.E = I.E;
            A.ld = 3 * (size_t)I.N;
            A.ld_lag = A.ld * A.ld;
            A.zeros_written = 1;
            sa_args_derive(A);
            const long long q = p - I.pair_begin;
            level_pair<OUT_DENSE, false>(A, nullptr, Ls, q, (int)(q % I.N), (int)(q / I.N), lane, unused);
        }
    }
}

template <int WPB, int MINB>
static int launch_batch_level(const BatchInst* d_insts, int ninst, long long total, int n_gh, int chunk,
                              unsigned long long* d_next, int device, cudaStream_t s) {
    const size_t smem = sizeof(LevelShared) * WPB;
    if (int rc = opt_in_smem(sa_batch_level_kernel<WPB, MINB>, smem, s)) return rc;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const unsigned blocks = (unsigned)(sms * MINB);       // one resident wave: persistent
    sa_batch_level_kernel<WPB, MINB><<<blocks, 32 * WPB, smem, s>>>(d_insts, ninst, total, n_gh, chunk, d_next);
    EBEM_CUDA_TRY(cudaGetLastError());
    return EBEM_OK;
}

// Zeros of every instance's output (the output pointers read from the device
// table at run time, as the assembly reads them): blockIdx.y = instance,
// 16-byte stores over its 9 N^2 nlag doubles.  The assembly then writes only
// the blocks of each pair's non-null lags; zeroing the whole buffer at copy
// bandwidth costs less than the scattered zero blocks of the direct output.
__global__ void batch_zero_kernel(const BatchInst* __restrict__ insts) {
    const BatchInst& I = insts[blockIdx.y];
    const long long n = 9LL * I.N * I.N * I.nlag;
    const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
    if ((reinterpret_cast<size_t>(I.E) & 15) == 0) {
        double2* E2 = reinterpret_cast<double2*>(I.E);
        const double2 z = make_double2(0.0, 0.0);
        for (long long k = t0; k < n / 2; k += stride) E2[k] = z;
        if ((n & 1) && t0 == 0) I.E[n - 1] = 0.0;
    } else {
        // an output that starts off a 16-byte boundary: 8-byte stores
        for (long long k = t0; k < n; k += stride) I.E[k] = 0.0;
    }
}

int launch_sa_batch(const BatchInst* d_insts, int ninst, long long total, int n_gh, int wpb, int chunk,
                    unsigned long long* d_next, int device, cudaStream_t s) {
    (void)n_gh;
    if (ninst > 65535) return fail(EBEM_ERR_INVALID, "too many batch instances for one launch");
    batch_zero_kernel<<<dim3(148, (unsigned)ninst), 256, 0, s>>>(d_insts);
    EBEM_CUDA_TRY(cudaGetLastError());
    if (wpb == 2) return launch_batch_level<2, 8>(d_insts, ninst, total, n_gh, chunk, d_next, device, s);
    return launch_batch_level<4, 4>(d_insts, ninst, total, n_gh, chunk, d_next, device, s);
}

}  // namespace ebem
