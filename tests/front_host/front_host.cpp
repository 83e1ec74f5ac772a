// Host build of the device algebra of the semi-analytic blocks: F(t_k) of one
// (source, field) pair from the closed form of sa_front.cuh, the levels,
// children and fronts walked one after the other, and from the edge
// quadrature of edge_quadrature.hpp (level_value).
#include <cmath>
#include <vector>

#include "edge_quadrature.hpp"
#include "sa_front.cuh"

using namespace ebem;

static void level_front(double Fk[6], int k, double cP, double cS, double dt, const TriGeom& F, const NodeW* nodes,
                        int n_gh) {
    const double k1 = 1 / (cP * cP), ks = 1 / (cS * cS), t = k * dt, t2 = t * t, rP = cP * t, rS = cS * t;
    double T[7] = {0, 0, 0, 0, 0, 0, 0};
    for (int g = 0; g < n_gh; g++) {
        NodeGeo G;
        node_geo(G, nodes[g], F);
        double rhoP, rhoS;
        const int type = classify(G.zeta, rP, rS, G.dMIN, rhoP, rhoS);
        if (type == T_NONE) continue;
        const double z2 = G.zeta * G.zeta, zs = G.zeta * G.sigma;
        double fields[3][FC_N];
        FrontSide side[3];
        bool live[3];
        double all = 0.0, w[3];
        for (int c = 0; c < 3; c++) {
            live[c] = front_side(side[c], G, c);
            if (!live[c]) continue;
            w[c] = nodes[g].w * side[c].sgnC;
            front_fields(fields[c], 1, side[c], G.zeta, G.sigma, w[c]);
            all = std::fmax(all, std::fmax(std::fmax(side[c].R1s, side[c].R2s), side[c].F * side[c].F + 1e-6));
        }
        double ang[6] = {0, 0, 0, 0, 0, 0};
        for (int c = 0; c < 3; c++) {
            if (!live[c]) continue;
            double a[6], p[7] = {0, 0, 0, 0, 0, 0, 0};
            front_angles(a, FrontView{fields[c], 1});
            const double h[7] = {a[0], a[1], a[2], a[3], a[4], a[5], 0.0};
            front_to_plane(p, h, side[c].ux, side[c].uy, -1.0, w[c], w[c]);
            for (int e = 0; e < 6; e++) ang[e] += p[e];
        }
        const bool fullP = cP * (k * dt) > std::sqrt(all + z2), fullS = type == T_SP_SP && cS * (k * dt) > std::sqrt(all + z2);
        if (std::fabs(ang[0]) > 1e-12 * nodes[g].w)
            front_node_terms(T, ang, G.zeta, zs, type, rP, rS, rhoP, rhoS, !fullP, !fullS, t2, k1, ks);
        for (int c = 0; c < 3; c++) {
            if (!live[c]) continue;
            const FrontView C{fields[c], 1};
            const bool foot = side[c].x1 >= 0 && side[c].x2 < 0;
            const double F2 = side[c].F * side[c].F;
            const double near2 = std::fmax(F2 + 1e-6, foot ? 0.0 : std::fmin(side[c].R1s, side[c].R2s));
            double a[7], b[7];
            for (int f = 0; f < 2; f++) {
                const bool isP = f == 0;
                const double r = isP ? rP : rS, kk = isP ? k1 : ks;
                if (!isP && type != T_SP_SP) continue;
                if (isP ? fullP : fullS) {
                    front_full(a, b, C);
                    double h[7];
                    for (int e = 0; e < 7; e++) h[e] = kk * a[e] + ((e == 0 && !isP) ? -t2 : t2) * b[e];
                    front_to_plane(T, h, side[c].ux, side[c].uy, zs, w[c], isP ? -w[c] : w[c]);
                } else if (r > std::sqrt(near2 + z2)) {
                    double h[7];
                    front_item(h, C, r, isP);
                    front_to_plane(T, h, side[c].ux, side[c].uy, zs, kk * w[c], isP ? -kk * w[c] : kk * w[c]);
                }
            }
        }
    }
    const double M[3][3] = {{T[1], T[2], T[4]}, {T[2], T[3], T[5]}, {T[4], T[5], T[6]}};
    double R[3][3];
    for (int r = 0; r < 3; r++)
        for (int c = 0; c < 3; c++) {
            R[r][c] = 0;
            for (int p = 0; p < 3; p++)
                for (int q = 0; q < 3; q++) R[r][c] += F.C[3 * p + r] * M[p][q] * F.C[3 * q + c];
        }
    Fk[0] = 0.5 * (T[0] + R[0][0]); Fk[1] = 0.5 * R[0][1]; Fk[2] = 0.5 * R[0][2];
    Fk[3] = 0.5 * (T[0] + R[1][1]); Fk[4] = 0.5 * R[1][2]; Fk[5] = 0.5 * (T[0] + R[2][2]);
}

// Blocks of the listed (source, field, lag) triples: out[9 q + 3 r + c].
extern "C" void front_blocks(const double* coords, const int* tris, const double* bary, const double* wout, int n_gh,
                             double rho, double cP, double cS, double dt, int n, const int* src, const int* fld,
                             const int* lag, int closed, double* out) {
    const int sym[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
#pragma omp parallel for schedule(dynamic)
    for (int q = 0; q < n; q++) {
        TriGeom S, F;
        double V[3][3], VS[3][3];
        for (int v = 0; v < 3; v++)
            for (int c = 0; c < 3; c++) {
                VS[v][c] = coords[3 * tris[3 * src[q] + v] + c];
                V[v][c] = coords[3 * tris[3 * fld[q] + v] + c];
            }
        tri_geom(VS, S);
        tri_geom(V, F);
        std::vector<NodeW> nodes(n_gh);
        for (int g = 0; g < n_gh; g++) {
            double p[3];
            for (int c = 0; c < 3; c++) p[c] = bary[3 * g] * VS[0][c] + bary[3 * g + 1] * VS[1][c] + bary[3 * g + 2] * VS[2][c];
            nodes[g] = {p[0], p[1], p[2], S.area * wout[g]};
        }
        double E[6] = {0, 0, 0, 0, 0, 0};
        for (int w = -1; w <= 1; w++) {
            const int k = lag[q] + w;
            if (k < 1) continue;
            double Fk[6];
            if (closed) level_front(Fk, k, cP, cS, dt, F, nodes.data(), n_gh);
            else level_value(Fk, k, cP, cS, dt, F, nodes.data(), n_gh);
            for (int e = 0; e < 6; e++) E[e] += (w == 0 ? -2.0 : 1.0) * Fk[e];
        }
        for (int e = 0; e < 9; e++) {
            const double v = E[sym[e]] / (4 * kPi * rho);
            out[9 * q + e] = std::fabs(v) < 1.0e-14 ? 0.0 : v;
        }
    }
}

// q_log(x[k]) and q_atan2(y[k], x[k]) of sa_math.cuh.
extern "C" void front_math(int n, const double* y, const double* x, double* lg, double* at) {
    for (int k = 0; k < n; k++) {
        lg[k] = q_log(x[k]);
        at[k] = q_atan2(y[k], x[k]);
    }
}
