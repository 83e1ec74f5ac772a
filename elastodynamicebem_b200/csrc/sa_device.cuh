// Basics shared by the kernels' semi-analytic algebra: qualifiers (the same
// headers compile as host code for the tests), the case split's names and the
// per-triangle data.
#pragma once

#include <math.h>

#ifdef __CUDACC__
#include <cuda_runtime.h>
#define EBEM_DI __device__ __forceinline__
#define EBEM_HDI __host__ __device__ inline
#else
#define EBEM_DI inline
#define EBEM_HDI inline
#endif

namespace ebem {

constexpr double kPi = 3.141592653589793238462643383279502884;

// Fronts at a projected node: none, both within the triangle's reach, the S
// front still short of it, only the P front in its plane.
enum : int { T_NONE = 0, T_SP_SP = 1, T_SP_P = 2, T_P = 3 };

EBEM_HDI double sgn(double x) { return x > 0 ? 1.0 : (x < 0 ? -1.0 : 0.0); }
EBEM_DI double acos_c(double x) { return acos(fmin(1.0, fmax(-1.0, x))); }
EBEM_DI double sqrt_c(double x) { return x > 0.0 ? sqrt(x) : 0.0; }

// Per field triangle data produced by the preparation kernel.
struct TriGeom {
    double P1[3];          // first vertex
    double e1[3], e2[3];   // in-plane frame (calcoloSistemaRiferimento.m)
    double n[3];           // unit normal (readSpaceMesh.m:114-122)
    double L1, L3, cd, sd; // |P2-P1|, |P3-P1|, cos/sin of the angle at P1
    double C[9];           // Euler matrix, row-major (rotazioneInversaEulero.m:160-176)
    double ctr[3];         // centroid
    double maxL;           // longest edge
    double area;
    double pad;
};

}  // namespace ebem
