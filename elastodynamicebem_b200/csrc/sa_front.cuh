// Closed form of the semi-analytic inner integral, one front at a time.
//
// The quantity is the reference's (SA/calcoloMatrice/
// BEMenerg_coreSA_calcIntgInt_childTriangle.m with the region integrals of
// f/BEMenerg_analiticIntg/*.m and the weights of
// BEMenerg_coreSA_calcMatrixSubBlock.m:101-104); the evaluation is not: every
// piece has its antiderivative in a coordinate along the side, free of the
// skew basis of coeffB.m whose 1/sin^2 factors amplify rounding by 1e6 on
// thin children, and the P and the S front separate.
//
// Radial antiderivatives in r = sqrt(rho^2 + zeta^2):
//   A1 = r, A3 = -1/r                     (1/r, 1/r^3 times rho d rho)
//   B2 = r + zeta^2/r, C2 = ln(rho + r) - rho/r, D2 = -zeta^2/r
//                                         (in-plane, mixed, normal parts of r_i r_j / r^3)
//   B4 = -1/r + zeta^2/(3 r^3), C4 = -(r^2 + r rho + rho^2)/(3 (r + rho) r^3),
//   D4 = -zeta^2/(3 r^3)                  (the same of r_i r_j / r^5)
//
// Separation.  A field triangle seen from the projection O of an outer node
// is a signed sum of children (O, V1, V2).  Along the ray at polar angle
// theta the integrand's radial antiderivatives V are taken between the S and
// the P front (weights wP) and inside the S front (weights wS), clipped at
// the side R(theta).  Collecting the terms by the front they end on, with
// r = c t the front's radius, k = 1/c^2 and t^2 = k r^2,
//   F(t) = Phi_P(c_P t) + Phi_S(c_S t) - (terms at O, a multiple of the
//          angle the triangle fills around O),
//   Phi  = k ( sc , -/+ Q ):  scalar k (A1 -/+ r^2 A3), tensor -/+ k (B2 - 3
//          r^2 B4, C2 - 3 r^2 C4, D2 - 3 r^2 D4)   (upper sign P, lower S),
// each integrated over the angle of the child with V at min(R(theta), rho),
// rho = sqrt(r^2 - zeta^2).  Phi is written as [V(rho) x (angle of the
// triangle)] + sum over children of H, H the part of the side inside the
// front: its antiderivative minus V(rho) x (its angle).  H = 0 until the
// front meets the side; the angle of the triangle is zero for every outer
// node that projects outside the field triangle.
//
// Edge coordinate.  On a side at distance F from O let x be the signed
// position along the side from the foot of the perpendicular (from V2
// towards V1), R = sqrt(x^2 + F^2), r = sqrt(R^2 + zeta^2), r0^2 = F^2 +
// zeta^2, and take the tensor in the frame (side direction, foot direction,
// normal).  d(theta) = F dx / R^2 and everything is elementary in
//   L = asinh(x / r0), J = int F dx / (r R^2) = atan(zeta x / (F r)) / zeta,
//   phi = atan(F / x), ln(R + r)
// and rational functions.  H at an end that moves with the front (R = rho)
// collapses to L, J, phi and r / (r + x) alone (the terms in ln(rho + r) and
// the mixed in-plane term cancel against V(rho) x (angle)); at an end that
// is a vertex of the child the same functions are level-independent.
//
// Rounding.  J and the rational terms tend to constants of size 1/F and 1/r0
// as x grows, which cancel between two ends on one side of the foot; they
// are therefore kept as tails (integrals from |x| to infinity, Psi for J,
// chi, K), and the constants enter only when the piece contains the foot.
// They come with the weight t^2 in both fronts and opposite signs, t^2 / F on
// children as thin as the outer rule's nodes lie to the sides; there they are
// left out where the S front has passed the foot too (front_foot).  With them the
// blocks were off by up to 12 times the rounding of what is left.
//
// The reference's thresholds are kept: a front crosses a side when rho^2 -
// F^2 > 1e-6 (childTriangle.m:62, 75), |2 area| < 1e-6 skips a child, zeta <
// 1e-6 is 0, and an instant with c_S t == zeta exactly finds no front
// (BEMenerg_coreSA_calcMatrixSubBlock.m:58-69).
#pragma once

#include "sa_math.cuh"
#include "sa_pair.cuh"

namespace ebem {

// Level-independent data of one child, kept as numbered fields so that a
// kernel can hold them field by field in shared memory.
enum : int {
    FC_F, FC_Z, FC_IZ, FC_R02, FC_IR0, FC_X1, FC_X2, FC_J2, FC_W, FC_UX, FC_UY, FC_ZS,
    FC_E1,                                    // first field of the end V1
    FC_NE = 10,                               // fields of an end
    FC_E2 = FC_E1 + FC_NE,
    FC_N = FC_E2 + FC_NE
};
// (FC_IZ: 1 / zeta, 0 for zeta = 0); fields of an end: L, Psi, phi, chi = F /
// (r (r + |x|)), d = F / (R^2 r), r, ln(R + r), K (the tail of -3 int C4 sin),
// q = 1 / (r (r + R)), 1 / R
enum : int { FE_L, FE_PSI, FE_PHI, FE_CHI, FE_D, FE_R, FE_LN, FE_K, FE_Q, FE_IR };

// Position of a child in edge coordinates; false when it is degenerate.
struct FrontSide {
    double F, x1, x2, ux, uy, sgnC, R1s, R2s;   // R1s, R2s: squared distances of V1, V2 from O
};

EBEM_DI bool front_side(FrontSide& s, const NodeGeo& G, int k) {
    const int k1 = (k == 2) ? 0 : k + 1;
    const double C = G.c[k];
    if (fabs(C) < 1.0e-06) return false;
    double v1x = G.tri[k][0], v1y = G.tri[k][1], v2x = G.tri[k1][0], v2y = G.tri[k1][1];
    if (C < 0) {
        double tx = v1x, ty = v1y;
        v1x = v2x; v1y = v2y;
        v2x = tx; v2y = ty;
    }
    const double dx = v1x - v2x, dy = v1y - v2y;
    const double il = q_rcp(q_sqrt(dx * dx + dy * dy));
    s.ux = dx * il;
    s.uy = dy * il;
    s.F = (v1x * v2y - v1y * v2x) * il;
    s.x1 = v1x * s.ux + v1y * s.uy;
    s.x2 = v2x * s.ux + v2y * s.uy;
    s.sgnC = sgn(C);
    s.R1s = v1x * v1x + v1y * v1y;
    s.R2s = v2x * v2x + v2y * v2y;
    return true;
}

// Psi(x) = int_x^inf F dx / (r R^2), x >= 0: atan(zeta w) / zeta with w = F
// r0^2 / ((r + x) (F^2 r + zeta^2 x)), F / (r (r + x)) = chi at zeta = 0.
EBEM_DI double front_psi(double F, double z, double iz, double r02, double x, double r, double chi) {
    const double a = q_atan2(z * F * r02, (r + x) * (F * F * r + z * z * x));
    return z > 0 ? a * iz : chi;
}

// The fields of the end at position x of the side; one division serves all
// the reciprocals.
EBEM_DI void front_end(double e[FC_NE], double F, double z, double iz, double r02, double ir0, double x) {
    const double ax = fabs(x), R = q_sqrt(ax * ax + F * F), r = q_sqrt(ax * ax + r02);
    const double a = r + ax, b = R + ax, c = R + r;
    const double rR = r * R, ab = a * b, i = q_rcp(rR * c * ab);
    const double iR = i * (r * c * ab), q = i * (R * ab), iab = i * (rR * c);      // 1/R, 1/(r c), 1/(a b)
    e[FE_L] = q_log(a * ir0);
    e[FE_CHI] = F * (i * (R * c * b));
    e[FE_PSI] = front_psi(F, z, iz, r02, ax, r, e[FE_CHI]);
    e[FE_PHI] = q_atan2(F, ax);
    e[FE_D] = F * iR * iR * (c * q);
    e[FE_R] = r;
    e[FE_LN] = q_log(c);
    e[FE_K] = F * F * iR * q * (a + R) * iab;
    e[FE_Q] = q;
    e[FE_IR] = iR;
}

// H of one child for the front of radius r (r > zeta; the caller has checked
// that it meets the side): scalar, then the tensor Q in the side's frame
// (cc, sc, ss, c, s, zz), c and s the mixed parts.  C(f) returns field f.
// No branches: the piece runs from the lower end (the front's crossing or V2)
// to the upper one (the crossing or V1), and the functions of the crossing
// and of both vertices are always formed, the unused ones with weight 0.
// foot: with the constants t^2 front_foot of a piece that contains the foot.
template <class View>
EBEM_DI void front_item(double H[7], const View& C, double r, bool isP, bool foot = true) {
    const double F = C(FC_F), z = C(FC_Z), r02 = C(FC_R02), x1 = C(FC_X1), x2 = C(FC_X2), ir0 = C(FC_IR0);
    const double z2 = z * z, r2 = r * r, rp = r2 + z2, rm = r2 - z2;
    const double xr = q_sqrt(r2 - r02), rho = q_sqrt(rm);
    const bool mhi = xr < x1, mlo = -xr > x2;
    // at the crossing
    const double a = r + xr, b = r + rho, ar = a * r, i = q_rcp(ar * b);
    const double g = r2 * (i * b), L = q_log(a * ir0);               // r / (r + x)
    const double m = q_log(b) + r * (i * ar);                        // ln(rho + r) + r / (r + rho)
    const double Psi = front_psi(F, z, C(FC_IZ), r02, xr, r, F * (i * b));
    const double phi = q_atan2(F, xr);
    const double n = (mhi ? 1.0 : 0.0) + (mlo ? 1.0 : 0.0);
    double hL = n * L, hPsi = n * Psi, hPhi = n * phi, hChi = n * (F * g), hs = -n * (L + g);
    double xD = 0.0, hsc = 0.0, hc = 0.0;
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const int p = e == 0 ? FC_E1 : FC_E2;
        const double x = e == 0 ? x1 : x2, ax = fabs(x), iR = C(p + FE_IR);
        // +1 for the upper end, -1 for the lower one, 0 for one at the crossing;
        // times the sign of x for the odd parts
        const double ev = (e == 0 ? mhi : mlo) ? 0.0 : (e == 0 ? 1.0 : -1.0), od = x >= 0 ? ev : -ev;
        const double Le = C(p + FE_L), dm = m - C(p + FE_LN), dr = r - C(p + FE_R), D = C(p + FE_D) * (dr * dr);
        hL += od * Le;
        hPsi += od * C(p + FE_PSI);
        hPhi += od * C(p + FE_PHI);
        hChi += od * (r2 * C(p + FE_CHI));
        hs -= od * (Le + ax * iR * dm + r2 * C(p + FE_K));
        xD += od * (ax * D);
        hsc -= ev * (F * D);
        hc += ev * (F * iR * (dm - r2 * C(p + FE_Q)));
    }
    const double FL = F * hL;
    double B = FL - rp * hPsi + 2 * r * hPhi;
    double ss = B - FL - hChi + xD, zz = hChi - rm * hPsi, S = FL + rm * hPsi;
    // twice the constants of the odd parts when the piece contains the foot
    const double in = ((mhi || x1 >= 0) && (mlo || x2 < 0)) ? 1.0 : 0.0;
    const double tt = foot ? r2 : 0.0;
    const double J2 = in * C(FC_J2), Jm = (tt - z2) * J2, y2 = in * 2 * tt * (ir0 * ir0), Fy = F * y2;
    const double b0 = (tt + z2) * J2 - in * 2 * kPi * r;
    B += b0;
    ss += b0 + Fy;
    zz += Jm - Fy;
    H[0] = isP ? B : S - Jm;
    H[1] = B - xD;
    H[2] = hsc;
    H[3] = ss;
    H[4] = hc;
    H[5] = hs + y2;
    H[6] = zz;
}

// Whole side of one child: G = a + r^2 b of the same seven functions without
// the V(rho) x (angle) terms (the scalar's b enters as +b for P, -b for S).
// foot as in front_item.
template <class View>
EBEM_DI void front_full(double a[7], double b[7], const View& C, bool foot = true) {
    const double F = C(FC_F), z = C(FC_Z), x1 = C(FC_X1), x2 = C(FC_X2), z2 = z * z;
    double L = 0, J = 0, X1 = 0, XI = 0, CH = 0, sca = 0, scb = 0, ca = 0, cb = 0, sa = 0, sb = 0;
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const int p = e == 0 ? FC_E1 : FC_E2;
        const double x = e == 0 ? x1 : x2, ev = e == 0 ? 1.0 : -1.0, od = x >= 0 ? ev : -ev;
        const double r = C(p + FE_R), d = C(p + FE_D), ax = fabs(x), ln = C(p + FE_LN), fR = F * C(p + FE_IR);
        L += od * C(p + FE_L);
        J -= od * C(p + FE_PSI);
        X1 += od * (ax * d * r * r);
        XI += od * (ax * d);
        CH -= od * C(p + FE_CHI);
        sca += ev * (F * d * r * r);
        scb += ev * (F * d);
        ca += ev * (fR * ln);
        cb += ev * (fR * C(p + FE_Q));
        sa += od * (ax * C(p + FE_IR) * ln);
        sb += od * C(p + FE_K);
    }
    double JA = J;
    if (x1 >= 0 && x2 < 0) {
        JA += C(FC_J2);
        if (foot) {
            const double i2 = 2 * C(FC_IR0) * C(FC_IR0);
            J = JA;
            CH += F * i2;
            sb -= i2;
        }
    }
    const double A1 = F * L + z2 * JA;
    a[0] = A1;            b[0] = J;
    a[1] = A1 - X1;       b[1] = J - XI;
    a[2] = -sca;          b[2] = -scb;
    a[3] = X1 + z2 * JA;  b[3] = J + CH + XI;
    a[4] = -ca;           b[4] = -cb;
    a[5] = sa - L;        b[5] = -sb;
    a[6] = -z2 * JA;      b[6] = J - CH;
}

// The constants of a child whose side contains the foot, which a front adds t^2
// times from where it passes the foot on: +K for P, -K for S, in the plane frame
// (S, T11, T12, T22, T13, T23, T33) with the node's weight.
template <class View>
EBEM_DI void front_foot(double T[7], const View& C, double t2) {
    const double w = t2 * C(FC_W), ux = C(FC_UX), uy = C(FC_UY), ir0 = C(FC_IR0);
    const double wJ = w * C(FC_J2), wy = w * (2 * ir0 * ir0), wF = wy * C(FC_F), wz = wy * C(FC_ZS);
    T[0] += wJ;
    T[1] -= wJ + uy * uy * wF;
    T[2] += ux * uy * wF;
    T[3] -= wJ + ux * ux * wF;
    T[4] -= uy * wz;
    T[5] += ux * wz;
    T[6] -= wJ - wF;
}

// Angle of the whole child and its moments (1, cc, sc, ss, c, s).
template <class View>
EBEM_DI void front_angles(double g[6], const View& C) {
    const double x1 = C(FC_X1), x2 = C(FC_X2);
    double a0 = 0, h = 0, sc = 0, c = 0, s = 0;
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const int p = e == 0 ? FC_E1 : FC_E2;
        const double x = e == 0 ? x1 : x2, ev = e == 0 ? 1.0 : -1.0, od = x >= 0 ? ev : -ev;
        const double fR = C(FC_F) * C(p + FE_IR), xR = fabs(x) * C(p + FE_IR);
        a0 -= od * C(p + FE_PHI);
        h += od * (0.5 * fR * xR);
        sc -= ev * (0.5 * fR * fR);
        c -= ev * fR;
        s += od * xR;
    }
    if (x1 >= 0 && x2 < 0) a0 += kPi;
    g[0] = a0;
    g[1] = 0.5 * a0 - h;
    g[2] = sc;
    g[3] = 0.5 * a0 + h;
    g[4] = c;
    g[5] = s;
}

// Side frame -> plane frame: (scalar, cc, sc, ss, c, s, zz) times the weights
// w0 (scalar) and w (tensor) added to (S, T11, T12, T22, T13, T23, T33).
EBEM_DI void front_to_plane(double T[7], const double H[7], double ux, double uy, double zs, double w0, double w) {
    const double cc = ux * ux, ss = uy * uy, cs = ux * uy;
    T[0] += w0 * H[0];
    T[1] += w * (cc * H[1] - 2 * cs * H[2] + ss * H[3]);
    T[2] += w * (cs * H[1] + (cc - ss) * H[2] - cs * H[3]);
    T[3] += w * (ss * H[1] + 2 * cs * H[2] + cc * H[3]);
    T[4] += -zs * w * (ux * H[4] - uy * H[5]);
    T[5] += -zs * w * (uy * H[4] + ux * H[5]);
    T[6] += w * H[6];
}

// First level k >= 1 (t_k = k dt) at which a front of speed c lies beyond the
// radius tau: c k dt > tau; at most `most` (1 when tau is not a number).
EBEM_DI int front_level(double tau, double icdt, int most) {
    const double k = tau * icdt;
    return k >= (double)most ? most : (int)k + 1;
}

// Level-independent data of one child of an outer node: fields into p[f *
// stride].  w is the node weight (with the child's sign).
EBEM_DI void front_fields(double* p, int stride, const FrontSide& s, double zeta, double sigma, double w) {
    const double r02 = s.F * s.F + zeta * zeta, r0 = q_sqrt(r02), ir0 = q_rcp(r0);
    const double iz = zeta > 0 ? q_rcp(zeta) : 0.0;
    p[FC_F * stride] = s.F;
    p[FC_Z * stride] = zeta;
    p[FC_IZ * stride] = iz;
    p[FC_R02 * stride] = r02;
    p[FC_IR0 * stride] = ir0;
    p[FC_X1 * stride] = s.x1;
    p[FC_X2 * stride] = s.x2;
    p[FC_J2 * stride] = zeta > 0 ? 2.0 * q_atan2(zeta, s.F) * iz : 2.0 * ir0;
    p[FC_W * stride] = w;
    p[FC_UX * stride] = s.ux;
    p[FC_UY * stride] = s.uy;
    p[FC_ZS * stride] = zeta * sigma;
#pragma unroll 1
    for (int e = 0; e < 2; e++) {
        double v[FC_NE];
        front_end(v, s.F, zeta, iz, r02, ir0, e == 0 ? s.x1 : s.x2);
#pragma unroll
        for (int f = 0; f < FC_NE; f++) p[((e == 0 ? FC_E1 : FC_E2) + f) * stride] = v[f];
    }
}

struct FrontView {
    const double* p;
    int stride;
    EBEM_DI double operator()(int f) const { return p[f * stride]; }
};

// Radial antiderivatives at in-plane radius rho (r = sqrt(rho^2+zeta^2)
// supplied by the caller).  The mixed (C) and normal (D) parts are only used
// for zeta > 0.
struct Rad { double A1, A3, B2, C2, D2, B4, C4, D4; };

EBEM_DI Rad radial_at(double rho, double r, double zeta) {
    Rad v;
    // one reciprocal gives both 1/r and 1/(r + rho)
    const double q = 1.0 / (r * (r + rho));
    const double ir = (r + rho) * q, ir3 = ir * ir * ir, z2 = zeta * zeta;
    v.A1 = r;
    v.A3 = -ir;
    v.B2 = r + z2 * ir;
    v.D2 = -z2 * ir;
    v.B4 = -ir + z2 * ir3 * (1.0 / 3.0);
    v.D4 = -z2 * ir3 * (1.0 / 3.0);
    if (zeta > 0) {
        v.C2 = q_log(rho + r) - rho * ir;
        v.C4 = -(r * r + r * rho + rho * rho) * ir3 * (r * q) * (1.0 / 3.0);
    } else {
        v.C2 = 0.0;
        v.C4 = 0.0;
    }
    return v;
}

// Terms of a node whose field triangle fills the angle moments g (1, cc, sc,
// ss, c, s; plane frame, signed and weighted) around it: V at the fronts that
// have not passed the whole triangle (inP, inS) and at O.  zs = zeta sigma.
EBEM_DI void front_node_terms(double T[7], const double g[6], double zeta, double zs, int type, double rP, double rS,
                              double rhoP, double rhoS, bool inP, bool inS, double t2, double k1, double ks) {
    double sc = 0.0, in = 0.0, mx = 0.0, zz = 0.0;
    if (inP) {
        sc += 2 * k1 * rP;
        in -= 4 * k1 * rP;
        if (zeta > 0) mx -= k1 * (q_log(rhoP + rP) + rP / (rP + rhoP));
    }
    if (type == T_P) {
        const double v = k1 * zeta + t2 / zeta;
        const double lz = q_log(zeta);
        sc -= v;
        in += 2 * v;
        mx += k1 * lz + t2 / (zeta * zeta);
        zz -= k1 * zeta - t2 / zeta;
    } else if (type == T_SP_P) {
        const Rad v = radial_at(rhoS, rS, zeta);
        sc -= k1 * v.A1 - t2 * v.A3;
        in -= -k1 * v.B2 + 3 * t2 * v.B4;
        mx -= -k1 * v.C2 + 3 * t2 * v.C4;
        zz -= -k1 * v.D2 + 3 * t2 * v.D4;
    } else {
        if (inS) {
            in += 4 * ks * rS;
            if (zeta > 0) mx += ks * (q_log(rhoS + rS) + rS / (rS + rhoS));
        }
        if (zeta > 0) {
            const double k5 = ks + k1, k6 = ks - k1;
            sc -= k5 * zeta;
            in -= 2 * k6 * zeta;
            mx -= k6 * q_log(zeta);
            zz += k6 * zeta;
        }
    }
    T[0] += sc * g[0];
    T[1] += in * g[1];
    T[2] += in * g[2];
    T[3] += in * g[3];
    T[4] += -zs * mx * g[4];
    T[5] += -zs * mx * g[5];
    T[6] += zz * g[0];
}

}  // namespace ebem
