// field.h -- launch interface of the field-evaluation kernels (field.cu):
// velocity potential at observation points from a boundary solution,
// phi(p) = sum_sources + sum_j (Mk_j phi_j - Lk_j dphi_j), Mk and Lk by the
// 7-point triangle rule of order 5 (BoundaryElementSolver::BemOperatorField,
// boundaryelementsolver.cpp:2318-2353).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "bem_types.h"

namespace bemgpu {

// FP32 record of two consecutive elements for the mixed-precision field kernel
// (240 bytes), every value as the pair (even element, odd element): the centroid
// as two floats c_hi + c_lo and the 7 rule points as offsets from it, all
// negated (p - q is an addition), and the unit normal. An odd last element is
// paired with a copy of itself that has zero coefficients.
struct __align__(16) FieldPairF {
  float2 nc_hi[3], nc_lo[3];
  float2 nq[21];
  float2 nrm[3];
};
static_assert(sizeof(FieldPairF) == 240, "FieldPairF is fifteen 16-byte pieces");
inline int64_t field_pairs(int64_t N) { return (N + 1) / 2; }

// Coefficients of the elements and right-hand sides: a = A phi, b = A dphi (A
// the element area), complex; two elements at a time in FP32.
struct __align__(16) FieldCoefPairF {
  float2 ax, ay, bx, by;
};
struct FieldCoef {
  double2 a, b;
};

// FP64 element record (224 bytes): centroid, unit normal, the 7 rule points
// and the largest distance of a rule point from the centroid.
struct __align__(16) FieldElem {
  double c[3], nrm[3], q[21], rho;
};
static_assert(sizeof(FieldElem) == 224, "FieldElem is fourteen 16-byte pieces");

// Observation points (threads) per CTA, and elements per shared-memory tile:
// below 4,096 points CTAs of 64, so that a ragged last CTA idles at most 63
// threads and there are enough CTAs to even out the SMs (5,120 elements, FP64: 250
// points 0.95 ms, CTAs of 256 1.21; 500 points 1.73, 2.00); above, 256 points
// share one staging of the elements (FP32, 4,096 points 148 us, CTAs of 64 152;
// 8,192 points 267, 274; but where 256 does not divide them the idle threads cost
// up to 8 %: FP64, 5,000 points 18.5 ms, 17.0).
constexpr int FIELD_PTS_SMALL = 64, FIELD_PTS_LARGE = 256;
constexpr int64_t FIELD_SMALL_POINTS = 4096;
inline int field_points(int64_t M) {
  return M < FIELD_SMALL_POINTS ? FIELD_PTS_SMALL : FIELD_PTS_LARGE;
}
constexpr int FIELD_RB = 4;     // right-hand sides per pass

// Element records and the coefficients of R columns: phi, dphi are N x R
// complex FP64 in the caller's order, perm[j] the caller index of cluster-order
// element j. Precision 1: fe field_pairs(N) FieldPairF, coef R x field_pairs(N)
// FieldCoefPairF; precision 0: fe N FieldElem, coef R x N FieldCoef. R = 0: the records only (perm, phi, dphi,
// coef unused).
int launch_field_prep(const Elem* E, const int64_t* perm, int64_t N, const double2* phi,
                      const double2* dphi, int R, int precision, void* fe, void* coef,
                      cudaStream_t s);

// Partial sums over S element chunks: partial[(s R + r) M + i] for the M
// points pts (M x 3, FP64) and all R columns. k is the wavenumber.
int launch_field_sum(const void* fe, const void* coef, int64_t N, int R, const double* pts,
                     int64_t M, double k, int precision, int S, double2* partial,
                     cudaStream_t s);

// phi_f = sum over the S partials + point sources (src: nsrc x 5 doubles x, y,
// z, Re w, Im w; sourcePhiTerm, boundaryelementsolver.cpp:3443-3450), added to
// every column; p_f = pfac phi_f. phi_f, p_f (M x R complex) may be null.
int launch_field_finish(const double2* partial, int S, int64_t M, int R, const double* pts,
                        const double* src, int nsrc, double k, double2 pfac, double2* phi_f,
                        double2* p_f, cudaStream_t s);

}  // namespace bemgpu
