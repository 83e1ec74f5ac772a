// A group of up to 10 (node, field triangle) projections on the lanes of one
// warp: lane 3 g + c owns child c of projection g.  Shared by the assembly's
// level kernel (the outer nodes of one source triangle seen from one field
// triangle) and the closed-form post-processing (one point seen from
// consecutive triangles).
#pragma once

#include "sa_front.cuh"

namespace ebem {

constexpr int kGroupNodes = 10;  // projections per group: 30 children on 32 lanes
constexpr int kSlots = 3 * kGroupNodes;

// Level-independent data of the group in shared memory.
struct FrontGroup {
    double f[FC_N * kSlots];                 // children, field-major
    double full[kGroupNodes][14];            // a, b of the whole triangle (plane frame, weighted)
    double ang[kGroupNodes][6];              // its angle moments around the node
    double zeta[kGroupNodes], zs[kGroupNodes], dmin[kGroupNodes];
};

// This lane's child.
struct FrontLane {
    FrontSide s;
    NodeGeo G;
    double w;                   // node weight
    double near, all;           // a front of larger radius meets the side / has passed the whole triangle
    bool child, live, maybe;    // maybe: the node can have an angle (inside the triangle, or next to a skipped child)
    bool split;                 // the side's foot is near: its constants apart (group_foot)
};

EBEM_DI double shfl3_sum(double v, int lane) {
    return v + __shfl_sync(0xffffffffu, v, lane + 1) + __shfl_sync(0xffffffffu, v, lane + 2);
}

EBEM_DI void group_geometry(FrontLane& L, bool child, const NodeW* node, const TriGeom* F, int lane) {
    const int g = lane / 3, c = lane - 3 * g;
    L.child = child;
    L.live = L.split = false;
    L.w = 0.0;
    L.G.zeta = L.G.sigma = L.G.dMIN = 0.0;
    L.G.inside = false;
    if (child) {
        node_project(L.G, *node, *F);
        L.live = front_side(L.s, L.G, c);
        L.w = node->w;
    }
    const double z2 = L.G.zeta * L.G.zeta;
    double all = 0.0, near = 0.0;
    if (L.live) {
        const double F2 = L.s.F * L.s.F + 1.0e-6;
        L.split = L.s.x1 >= 0 && L.s.x2 < 0;
        all = fmax(fmax(L.s.R1s, L.s.R2s), F2);
        near = L.split ? F2 : fmax(F2, fmin(L.s.R1s, L.s.R2s));
    }
    // the whole triangle is passed when every live child is
    const int b3 = 3 * g;
    const double a1 = __shfl_sync(0xffffffffu, all, b3), a2 = __shfl_sync(0xffffffffu, all, b3 + 1);
    const double a3 = __shfl_sync(0xffffffffu, all, (b3 + 2) & 31);
    L.all = q_sqrt(fmax(a1, fmax(a2, a3)) + z2);
    L.near = q_sqrt(near + z2);
    // Up to 6 times the foot's distance r0 the constants, r^2 2 / r0, are no more than
    // twice the 2 pi r of the terms beside them.  Rounding of the blocks in the mean
    // square (sphere of 80 triangles, 200 levels): nothing apart 1.7e-13 of the
    // largest block, a line at 4, 6 and 12 4.8e-14, 4.9e-14 and 8.0e-14; the time
    // does not depend on the line.
    L.split = L.split && L.all > 6.0 * L.near;
    L.maybe = child && (L.G.inside || !L.live);
    if (L.maybe && !L.G.inside) L.G.dMIN = edge_distance(L.G.tri);
}

// Fields of the children, whole-triangle terms and angles; returns the
// projections with an angle (bit 3 g).
EBEM_DI unsigned group_fields(FrontGroup& W, const FrontLane& L, int lane) {
    const int g = lane / 3, c = lane - 3 * g;
    const FrontView view{W.f + (lane < kSlots ? lane : 0), kSlots};
    const double w = L.w;
    if (L.live) front_fields(W.f + lane, kSlots, L.s, L.G.zeta, L.G.sigma, w * L.s.sgnC);
    // angle of the triangle around the node
    unsigned circ = 0;
    if (__ballot_sync(0xffffffffu, L.maybe) != 0u) {
        double ag[6] = {0, 0, 0, 0, 0, 0};
        if (L.live) front_angles(ag, view);
        const double a0 = shfl3_sum(L.live ? L.s.sgnC * ag[0] : 0.0, lane);
        circ = __ballot_sync(0xffffffffu, L.child && c == 0 && fabs(a0) > 1.0e-12);
        if (circ) {
            double T[7] = {0, 0, 0, 0, 0, 0, 0};
            if (L.live) {
                const double h[7] = {ag[0], ag[1], ag[2], ag[3], ag[4], ag[5], 0.0};
                front_to_plane(T, h, L.s.ux, L.s.uy, -1.0, w * L.s.sgnC, w * L.s.sgnC);
            }
#pragma unroll
            for (int e = 0; e < 6; e++) {
                const double v = shfl3_sum(T[e], lane);
                if (L.child && c == 0) W.ang[g][e] = v;
            }
            // d_min of the node is known to the lanes that asked for it
            if (L.maybe) W.dmin[g] = L.G.dMIN;
        }
    }
    // whole triangle: a + t^2 b
    double a[7] = {0, 0, 0, 0, 0, 0, 0}, b[7] = {0, 0, 0, 0, 0, 0, 0};
    if (L.live) {
        double fa[7], fb[7];
        front_full(fa, fb, view, !L.split);
        const double ws = w * L.s.sgnC, zs = L.G.zeta * L.G.sigma;
        front_to_plane(a, fa, L.s.ux, L.s.uy, zs, ws, ws);
        front_to_plane(b, fb, L.s.ux, L.s.uy, zs, ws, ws);
    }
#pragma unroll
    for (int e = 0; e < 7; e++) {
        const double va = shfl3_sum(a[e], lane), vb = shfl3_sum(b[e], lane);
        if (L.child && c == 0) {
            W.full[g][e] = va;
            W.full[g][7 + e] = vb;
        }
    }
    if (L.child && c == 0) {
        W.zeta[g] = L.G.zeta;
        W.zs[g] = L.G.zeta * L.G.sigma;
    }
    return circ;
}

// Projection g at one instant: its whole triangle where a front has passed it
// (cP, cS), and the terms of its angle.
EBEM_DI void group_node(double T[7], const FrontGroup& W, int g, bool cP, bool cS, bool angle, double rP, double rS,
                        double t2, double k1, double ks) {
    if (cP) {
        const double ca = cS ? ks - k1 : -k1, cb = cS ? 0.0 : t2, c0 = cS ? ks + k1 : k1;
        const double* fu = W.full[g];
        T[0] += c0 * fu[0] + cb * fu[7];
#pragma unroll
        for (int e = 1; e < 7; e++) T[e] += ca * fu[e] - cb * fu[7 + e];
    }
    if (angle) {
        double rhoP, rhoS;
        const int type = classify(W.zeta[g], rP, rS, W.dmin[g], rhoP, rhoS);
        if (type != T_NONE)
            front_node_terms(T, W.ang[g], W.zeta[g], W.zs[g], type, rP, rS, rhoP, rhoS, !cP, !cS, t2, k1, ks);
    }
}

// Constants of a split child, whose foot the P front has passed and the S front
// has not.
EBEM_DI void group_foot(double T[7], const FrontGroup& W, int slot, double t2) {
    front_foot(T, FrontView{W.f + slot, kSlots}, t2);
}

// Child `slot` at one instant, front P or S, added to T; foot: not a split one.
EBEM_DI void group_item(double T[7], const FrontGroup& W, int slot, bool foot, bool isP, double r, double kk) {
    const FrontView C{W.f + slot, kSlots};
    const double w = kk * C(FC_W);
    double H[7];
    front_item(H, C, r, isP, foot);
    front_to_plane(T, H, C(FC_UX), C(FC_UY), C(FC_ZS), w, isP ? -w : w);
}

// F = (S I + C^T M C) / 2 in global axes, entries 11, 12, 13, 22, 23, 33, from
// (S, T11, T12, T22, T13, T23, T33) in the plane frame C.
EBEM_DI void front_rotate(double Fk[6], const double T[7], const double* C) {
    const double M[3][3] = {{T[1], T[2], T[4]}, {T[2], T[3], T[5]}, {T[4], T[5], T[6]}};
    double MC[3][3], R[3][3];
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++) MC[r][c] = M[r][0] * C[c] + M[r][1] * C[3 + c] + M[r][2] * C[6 + c];
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = r; c < 3; c++) R[r][c] = C[r] * MC[0][c] + C[3 + r] * MC[1][c] + C[6 + r] * MC[2][c];
    Fk[0] = 0.5 * (T[0] + R[0][0]);
    Fk[1] = 0.5 * R[0][1];
    Fk[2] = 0.5 * R[0][2];
    Fk[3] = 0.5 * (T[0] + R[1][1]);
    Fk[4] = 0.5 * R[1][2];
    Fk[5] = 0.5 * (T[0] + R[2][2]);
}

}  // namespace ebem
