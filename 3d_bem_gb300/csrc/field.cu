// field.cu -- field evaluation: velocity potential at observation points from
// a boundary solution (BoundaryElementSolver::calculateFieldSolutionRegular,
// boundaryelementsolver.cpp:2263-2316, with BemOperatorField :2318-2353).
//
// Dense sum over (observation point, element) pairs with the 7-point rule:
// one thread per observation point, elements staged through shared memory in
// tiles, element range split over a second grid dimension so that few points
// still fill the GPU; partial sums land in a buffer and a second kernel adds
// them in a fixed order (deterministic, no atomics), adds the point sources
// and scales to sound pressure.
//
// Mixed precision (precision 1): the integrand in FP32 with two-float
// centroids (p - c_j keeps ~7 digits, the rule points are offsets from c_j),
// exp(ikr) from the hardware sin / cos after an exact reduction of
// k r / (2 pi) to [-1/2, 1/2] (absolute error ~4e-7 on [-pi, pi]), per-tile
// sums in FP32
// folded into FP64 accumulators every FIELD_TILE elements. Precision 0: the
// same sum in FP64.
#include "field.h"

namespace bemgpu {
namespace {

constexpr double kInv4Pi = 0.0795774715459476678844418816862571885;

// 7-point rule of order 5 (trianglequadraturerules.cpp:50-59 of the
// reference; orderLow = 5, boundaryelementsolver.h:653-654): barycentric xi1,
// xi2 and weight (weights sum to 1; the element area multiplies afterwards).
constexpr double kR7x1[7] = {0.33333333333333, 0.47014206410511, 0.47014206410511,
                             0.05971587178977, 0.10128650732346, 0.10128650732346,
                             0.79742698535309};
constexpr double kR7x2[7] = {0.33333333333333, 0.47014206410511, 0.05971587178977,
                             0.47014206410511, 0.10128650732346, 0.79742698535309,
                             0.10128650732346};
constexpr double kR7w[7] = {0.22500000000000, 0.13239415278851, 0.13239415278851,
                            0.13239415278851, 0.12593918054483, 0.12593918054483,
                            0.12593918054483};

__constant__ double cR7x1[7] = {kR7x1[0], kR7x1[1], kR7x1[2], kR7x1[3],
                                kR7x1[4], kR7x1[5], kR7x1[6]};
__constant__ double cR7x2[7] = {kR7x2[0], kR7x2[1], kR7x2[2], kR7x2[3],
                                kR7x2[4], kR7x2[5], kR7x2[6]};
// w / (4 pi)
__constant__ double cR7g[7] = {kR7w[0] * kInv4Pi, kR7w[1] * kInv4Pi, kR7w[2] * kInv4Pi,
                               kR7w[3] * kInv4Pi, kR7w[4] * kInv4Pi, kR7w[5] * kInv4Pi,
                               kR7w[6] * kInv4Pi};
__constant__ float cR7gf[7] = {
    (float)(kR7w[0] * kInv4Pi), (float)(kR7w[1] * kInv4Pi), (float)(kR7w[2] * kInv4Pi),
    (float)(kR7w[3] * kInv4Pi), (float)(kR7w[4] * kInv4Pi), (float)(kR7w[5] * kInv4Pi),
    (float)(kR7w[6] * kInv4Pi)};

__global__ void field_prep_kernel(const Elem* __restrict__ E, const int64_t* __restrict__ perm,
                                  int64_t N, const double2* __restrict__ phi,
                                  const double2* __restrict__ dphi, int R, int precision,
                                  void* __restrict__ fe, void* __restrict__ coef) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= N) return;
  const Elem& e = E[j];
  if (precision == 1) {
    FieldElemF f;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const float hi = (float)e.c[d];
      f.c_hi[d] = hi;
      f.c_lo[d] = (float)(e.c[d] - (double)hi);
      f.nrm[d] = (float)e.nrm[d];
    }
#pragma unroll
    for (int i = 0; i < 7; i++) {
      const double a1 = cR7x1[i], a2 = cR7x2[i], a3 = 1.0 - a2 - a1;
      double on = 0.0;
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const double o = (a1 * e.n1[d] + a2 * e.n2[d] + a3 * e.n3[d]) - e.c[d];
        f.q[3 * i + d] = (float)o;
        on += o * e.nrm[d];
      }
      f.qn[i] = (float)on;
    }
    f.pad[0] = f.pad[1] = f.pad[2] = 0.0f;
    static_cast<FieldElemF*>(fe)[j] = f;
  } else {
    FieldElem f;
    double rho = 0.0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      f.c[d] = e.c[d];
      f.nrm[d] = e.nrm[d];
    }
#pragma unroll
    for (int i = 0; i < 7; i++) {
      const double a1 = cR7x1[i], a2 = cR7x2[i], a3 = 1.0 - a2 - a1;
      double o2 = 0.0;
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const double q = (a1 * e.n1[d] + a2 * e.n2[d]) + a3 * e.n3[d];
        f.q[3 * i + d] = q;
        o2 += (q - e.c[d]) * (q - e.c[d]);
      }
      rho = fmax(rho, o2);
    }
    f.rho = sqrt(rho);
    static_cast<FieldElem*>(fe)[j] = f;
  }
  if (R == 0) return;  // element records only (the reflected elements)
  const int64_t cj = perm[j];
  const double A = e.area;
  for (int r = 0; r < R; r++) {
    const double2 p = phi[(int64_t)r * N + cj], dp = dphi[(int64_t)r * N + cj];
    if (precision == 1) {
      FieldCoefF c;
      c.a = make_float2((float)(A * p.x), (float)(A * p.y));
      c.b = make_float2((float)(A * dp.x), (float)(A * dp.y));
      static_cast<FieldCoefF*>(coef)[(int64_t)r * N + j] = c;
    } else {
      FieldCoef c;
      c.a = make_double2(A * p.x, A * p.y);
      c.b = make_double2(A * dp.x, A * dp.y);
      static_cast<FieldCoef*>(coef)[(int64_t)r * N + j] = c;
    }
  }
}

// Columns r0 .. r0 + RB - 1, element chunk blockIdx.y.
template <int RB, int FIELD_PTS>
__global__ void __launch_bounds__(FIELD_PTS)
    field_sum32_kernel(const FieldElemF* __restrict__ fe, const FieldCoefF* __restrict__ coef,
                       int64_t N, int64_t chunk, const double* __restrict__ pts, int64_t M,
                       float k, float kc, int r0, int R, double2* __restrict__ partial) {
  constexpr int FIELD_TILE = FIELD_PTS / 2;
  __shared__ FieldElemF se[FIELD_TILE];
  __shared__ FieldCoefF sc[RB][FIELD_TILE];
  const int64_t ip = (int64_t)blockIdx.x * FIELD_PTS + threadIdx.x;
  const int64_t e0 = (int64_t)blockIdx.y * chunk;
  const int64_t e1 = min(N, e0 + chunk);
  float ph[3] = {0.0f, 0.0f, 0.0f}, pl[3] = {0.0f, 0.0f, 0.0f};
  if (ip < M) {
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const double v = pts[3 * ip + d];
      ph[d] = (float)v;
      pl[d] = (float)(v - (double)ph[d]);
    }
  }
  double ax[RB], ay[RB];
#pragma unroll
  for (int r = 0; r < RB; r++) ax[r] = ay[r] = 0.0;
  for (int64_t t0 = e0; t0 < e1; t0 += FIELD_TILE) {
    const int nt = (int)min((int64_t)FIELD_TILE, e1 - t0);
    __syncthreads();
    const float4* src = reinterpret_cast<const float4*>(fe + t0);
    float4* dst = reinterpret_cast<float4*>(se);
    constexpr int PIECES = (int)(sizeof(FieldElemF) / sizeof(float4));
    for (int i = threadIdx.x; i < nt * PIECES; i += FIELD_PTS) dst[i] = src[i];
    for (int i = threadIdx.x; i < RB * nt; i += FIELD_PTS) {
      const int r = i / nt, j = i - r * nt;
      sc[r][j] = coef[(int64_t)(r0 + r) * N + t0 + j];
    }
    __syncthreads();
    float tx[RB], ty[RB];
#pragma unroll
    for (int r = 0; r < RB; r++) tx[r] = ty[r] = 0.0f;
    for (int j = 0; j < nt; j++) {
      const FieldElemF& E = se[j];
      const float dx = (ph[0] - E.c_hi[0]) + (pl[0] - E.c_lo[0]);
      const float dy = (ph[1] - E.c_hi[1]) + (pl[1] - E.c_lo[1]);
      const float dz = (ph[2] - E.c_hi[2]) + (pl[2] - E.c_lo[2]);
      const float dn = dx * E.nrm[0] + dy * E.nrm[1] + dz * E.nrm[2];
      float Lx = 0.0f, Ly = 0.0f, Mx = 0.0f, My = 0.0f;
#pragma unroll
      for (int i = 0; i < 7; i++) {
        const float rx = dx - E.q[3 * i], ry = dy - E.q[3 * i + 1], rz = dz - E.q[3 * i + 2];
        const float rr = rx * rx + ry * ry + rz * rz;
        const float ir = rsqrtf(rr);
        const float r = rr * ir;
        // exp(ikr): x = k r / (2 pi) reduced exactly to [-1/2, 1/2] (x - rint(x)
        // has no rounding), then the hardware sin / cos on 2 pi (x - rint(x))
        const float x = kc * r;
        const float xr = x - rintf(x);
        float sn, cs;
        __sincosf(6.28318530717959f * xr, &sn, &cs);
        const float kr = k * r;
        const float g0 = ir * cR7gf[i];  // w / (4 pi r)
        Lx = fmaf(g0, cs, Lx);
        Ly = fmaf(g0, sn, Ly);
        // w dG/dr rnq = g0 (p - q_i) . n / r^2 (cos + kr sin, sin - kr cos)
        const float tg = (dn - E.qn[i]) * (ir * ir * g0);
        Mx = fmaf(tg, fmaf(kr, sn, cs), Mx);
        My = fmaf(tg, fmaf(-kr, cs, sn), My);
      }
#pragma unroll
      for (int r = 0; r < RB; r++) {
        const FieldCoefF c = sc[r][j];
        tx[r] += (Mx * c.a.x - My * c.a.y) - (Lx * c.b.x - Ly * c.b.y);
        ty[r] += (Mx * c.a.y + My * c.a.x) - (Lx * c.b.y + Ly * c.b.x);
      }
    }
#pragma unroll
    for (int r = 0; r < RB; r++) {
      ax[r] += (double)tx[r];
      ay[r] += (double)ty[r];
    }
  }
  if (ip < M) {
#pragma unroll
    for (int r = 0; r < RB; r++)
      partial[((int64_t)blockIdx.y * R + r0 + r) * M + ip] = make_double2(ax[r], ay[r]);
  }
}

// sin and cos of x, |x| <= X, by their Taylor series to x^(2 NS + 1) and
// x^(2 NC): for X = 0.35 (6, 6) the first terms left out are below 3e-19 and
// 5e-18 of the functions, for X = 1 (8, 9) below 9e-18 and 5e-19.
template <int NS, int NC>
__device__ __forceinline__ void sincos_taylor(double x, double& sn, double& cs) {
  constexpr double is[9] = {1.0,
                            -1.0 / 6,
                            1.0 / 120,
                            -1.0 / 5040,
                            1.0 / 362880,
                            -1.0 / 39916800,
                            1.0 / 6227020800.0,
                            -1.0 / 1307674368000.0,
                            1.0 / 355687428096000.0};
  constexpr double ic[10] = {1.0,
                             -1.0 / 2,
                             1.0 / 24,
                             -1.0 / 720,
                             1.0 / 40320,
                             -1.0 / 3628800,
                             1.0 / 479001600.0,
                             -1.0 / 87178291200.0,
                             1.0 / 20922789888000.0,
                             -1.0 / 6402373705728000.0};
  const double t = x * x;
  double ps = is[NS], pc = ic[NC];
#pragma unroll
  for (int q = NS - 1; q >= 1; q--) ps = fma(ps, t, is[q]);
#pragma unroll
  for (int q = NC - 1; q >= 0; q--) pc = fma(pc, t, ic[q]);
  sn = fma(x * t, ps, x);
  cs = pc;
}

// Sums over the 7 rule points of w G / (4 pi r) and of its radial part
// w (1 - ikr) G / (4 pi r^3), both times exp(-ik r_c) unless FULL (NS, NC:
// terms of the series of the phase differences k (r - r_c)).
template <bool FULL, int NS, int NC>
__device__ __forceinline__ void field_points64(const FieldElem& e, double px, double py, double pz,
                                               double k, double krc, double& Lx, double& Ly,
                                               double& Mx, double& My) {
  for (int i = 0; i < 7; i++) {
    const double rx = px - e.q[3 * i], ry = py - e.q[3 * i + 1], rz = pz - e.q[3 * i + 2];
    const double rr = fma(rx, rx, fma(ry, ry, rz * rz));
    const double ir = rsqrt(rr);
    double r = rr * ir;
    r = fma(0.5 * ir, fma(-r, r, rr), r);  // one correction: r to half an ulp
    double sn, cs;
    if constexpr (FULL) sincos(k * r, &sn, &cs);
    else sincos_taylor<NS, NC>(fma(k, r, -krc), sn, cs);
    const double g0 = ir * cR7g[i];
    Lx = fma(g0, cs, Lx);
    Ly = fma(g0, sn, Ly);
    const double h = g0 * (ir * ir), kr = k * r;
    Mx = fma(h, fma(kr, sn, cs), Mx);
    My = fma(h, fma(-kr, cs, sn), My);
  }
}

// FP64: bound by the FP64 pipe (2 FMA per clock and SM on this GPU), so the
// kernel is laid out for few FP64 instructions per rule point (about 55; a
// sincos, a square root and a division each took ~80 with the rule points
// recomputed): rule points come ready from the element records, 1 / r from one
// rsqrt, (p - q) . n is the same for all points of the plane, and exp(ikr) =
// exp(ik r_c) exp(ik (r - r_c)) takes one sincos per element at its centroid
// and a short Taylor series per point (|k (r - r_c)| <= k rho; elements with
// k rho > 1 take the full sincos). 5,123 elements x 997 points, 3 columns:
// 3.70 ms; 18.99 ms before, with 40 CTAs on 152 SMs (see field_split).
template <int RB, int FIELD_PTS>
__global__ void __launch_bounds__(FIELD_PTS)
    field_sum64_kernel(const FieldElem* __restrict__ fe, const FieldCoef* __restrict__ coef,
                       int64_t N, int64_t chunk, const double* __restrict__ pts, int64_t M,
                       double k, int r0, int R, double2* __restrict__ partial) {
  constexpr int FIELD_TILE = FIELD_PTS / 4;
  __shared__ FieldElem se[FIELD_TILE];
  __shared__ FieldCoef sc[RB][FIELD_TILE];
  const int64_t ip = (int64_t)blockIdx.x * FIELD_PTS + threadIdx.x;
  const int64_t e0 = (int64_t)blockIdx.y * chunk;
  const int64_t e1 = min(N, e0 + chunk);
  double p[3] = {0.0, 0.0, 0.0};
  if (ip < M) {
#pragma unroll
    for (int d = 0; d < 3; d++) p[d] = pts[3 * ip + d];
  }
  double ax[RB], ay[RB];
#pragma unroll
  for (int r = 0; r < RB; r++) ax[r] = ay[r] = 0.0;
  for (int64_t t0 = e0; t0 < e1; t0 += FIELD_TILE) {
    const int nt = (int)min((int64_t)FIELD_TILE, e1 - t0);
    __syncthreads();
    const double2* src = reinterpret_cast<const double2*>(fe + t0);
    double2* dst = reinterpret_cast<double2*>(se);
    constexpr int PIECES = (int)(sizeof(FieldElem) / sizeof(double2));
    for (int i = threadIdx.x; i < nt * PIECES; i += FIELD_PTS) dst[i] = src[i];
    for (int i = threadIdx.x; i < RB * nt; i += FIELD_PTS) {
      const int r = i / nt, j = i - r * nt;
      sc[r][j] = coef[(int64_t)(r0 + r) * N + t0 + j];
    }
    __syncthreads();
    for (int j = 0; j < nt; j++) {
      const FieldElem& e = se[j];
      const double dx = p[0] - e.c[0], dy = p[1] - e.c[1], dz = p[2] - e.c[2];
      const double dn = fma(dx, e.nrm[0], fma(dy, e.nrm[1], dz * e.nrm[2]));
      const double krho = k * e.rho;
      double Lx = 0.0, Ly = 0.0, Mx = 0.0, My = 0.0;
      if (krho <= 1.0) {  // the same for every thread: an element's property
        const double krc = k * sqrt(fma(dx, dx, fma(dy, dy, dz * dz)));
        double s0, c0, ax0 = 0.0, ay0 = 0.0, bx0 = 0.0, by0 = 0.0;
        if (krho <= 0.35)
          field_points64<false, 6, 6>(e, p[0], p[1], p[2], k, krc, ax0, ay0, bx0, by0);
        else
          field_points64<false, 8, 9>(e, p[0], p[1], p[2], k, krc, ax0, ay0, bx0, by0);
        sincos(krc, &s0, &c0);
        Lx = ax0 * c0 - ay0 * s0;
        Ly = ax0 * s0 + ay0 * c0;
        Mx = bx0 * c0 - by0 * s0;
        My = bx0 * s0 + by0 * c0;
      } else {
        field_points64<true, 1, 1>(e, p[0], p[1], p[2], k, 0.0, Lx, Ly, Mx, My);
      }
      Mx *= dn;
      My *= dn;
#pragma unroll
      for (int r = 0; r < RB; r++) {
        const FieldCoef c = sc[r][j];
        ax[r] += (Mx * c.a.x - My * c.a.y) - (Lx * c.b.x - Ly * c.b.y);
        ay[r] += (Mx * c.a.y + My * c.a.x) - (Lx * c.b.y + Ly * c.b.x);
      }
    }
  }
  if (ip < M) {
#pragma unroll
    for (int r = 0; r < RB; r++)
      partial[((int64_t)blockIdx.y * R + r0 + r) * M + ip] = make_double2(ax[r], ay[r]);
  }
}

// Eight threads per value add its S partial sums, each an interleaved share in
// order, then their sums in order (with one thread per value and S up to 300
// chunks this kernel was a chain of 300 additions on a dozen CTAs).
__global__ void __launch_bounds__(256)
    field_finish_kernel(const double2* __restrict__ partial, int S, int64_t M, int R,
                        const double* __restrict__ pts, const double* __restrict__ src, int nsrc,
                        double k, double2 pfac, double2* __restrict__ phi_f,
                        double2* __restrict__ p_f) {
  __shared__ double2 red[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t i = (int64_t)blockIdx.x * 32 + lane;
  const bool on = i < M * R;
  double ax = 0.0, ay = 0.0;
  if (on) {
#pragma unroll 4
    for (int s = w; s < S; s += 8) {
      const double2 v = partial[(int64_t)s * R * M + i];
      ax += v.x;
      ay += v.y;
    }
  }
  red[w][lane] = make_double2(ax, ay);
  __syncthreads();
  if (w != 0 || !on) return;
#pragma unroll
  for (int q = 1; q < 8; q++) {
    ax += red[q][lane].x;
    ay += red[q][lane].y;
  }
  const int64_t ip = i % M;
  if (nsrc > 0) {  // sourcePhiTerm: w exp(ikr) / (4 pi r)
    const double px = pts[3 * ip], py = pts[3 * ip + 1], pz = pts[3 * ip + 2];
    for (int q = 0; q < nsrc; q++) {
      const double* sq = src + 5 * q;
      const double dx = sq[0] - px, dy = sq[1] - py, dz = sq[2] - pz;
      const double rr = sqrt(dx * dx + dy * dy + dz * dz);
      double sn, cs;
      sincos(k * rr, &sn, &cs);
      const double g = kInv4Pi / rr;
      const double Gx = cs * g, Gy = sn * g;
      ax += sq[3] * Gx - sq[4] * Gy;
      ay += sq[3] * Gy + sq[4] * Gx;
    }
  }
  if (phi_f) phi_f[i] = make_double2(ax, ay);
  if (p_f) p_f[i] = make_double2(pfac.x * ax - pfac.y * ay, pfac.x * ay + pfac.y * ax);
}

template <int RB, int PTS>
void sum_pass(const void* fe, const void* coef, int64_t N, int R, const double* pts, int64_t M,
              double k, int precision, int S, int64_t chunk, int r0, double2* partial,
              cudaStream_t s) {
  const dim3 grid((unsigned)((M + PTS - 1) / PTS), (unsigned)S);
  if (precision == 1) {
    const double kc = k / (2.0 * 3.14159265358979323846);
    field_sum32_kernel<RB, PTS><<<grid, PTS, 0, s>>>(
        static_cast<const FieldElemF*>(fe), static_cast<const FieldCoefF*>(coef), N, chunk, pts, M,
        (float)k, (float)kc, r0, R, partial);
  } else {
    field_sum64_kernel<RB, PTS><<<grid, PTS, 0, s>>>(static_cast<const FieldElem*>(fe),
                                                     static_cast<const FieldCoef*>(coef), N, chunk,
                                                     pts, M, k, r0, R, partial);
  }
}

template <int PTS>
int sum_passes(const void* fe, const void* coef, int64_t N, int R, const double* pts, int64_t M,
               double k, int prec, int S, int64_t chunk, double2* partial, cudaStream_t s) {
  int n = 0;
  for (int r0 = 0; r0 < R; r0 += FIELD_RB, n++) {
    switch (R - r0 >= FIELD_RB ? FIELD_RB : R - r0) {
      case 1: sum_pass<1, PTS>(fe, coef, N, R, pts, M, k, prec, S, chunk, r0, partial, s); break;
      case 2: sum_pass<2, PTS>(fe, coef, N, R, pts, M, k, prec, S, chunk, r0, partial, s); break;
      case 3: sum_pass<3, PTS>(fe, coef, N, R, pts, M, k, prec, S, chunk, r0, partial, s); break;
      default: sum_pass<4, PTS>(fe, coef, N, R, pts, M, k, prec, S, chunk, r0, partial, s); break;
    }
  }
  return n;
}

}  // namespace

int launch_field_prep(const Elem* E, const int64_t* perm, int64_t N, const double2* phi,
                      const double2* dphi, int R, int precision, void* fe, void* coef,
                      cudaStream_t s) {
  if (N <= 0) return 0;
  field_prep_kernel<<<(unsigned)((N + 255) / 256), 256, 0, s>>>(E, perm, N, phi, dphi, R,
                                                                precision, fe, coef);
  return 1;
}

int launch_field_sum(const void* fe, const void* coef, int64_t N, int R, const double* pts,
                     int64_t M, double k, int precision, int S, double2* partial,
                     cudaStream_t s) {
  if (M <= 0 || R <= 0 || S <= 0) return 0;
  const int64_t chunk = (N + S - 1) / S;
  return field_points(M) == FIELD_PTS_SMALL
             ? sum_passes<FIELD_PTS_SMALL>(fe, coef, N, R, pts, M, k, precision, S, chunk, partial, s)
             : sum_passes<FIELD_PTS_LARGE>(fe, coef, N, R, pts, M, k, precision, S, chunk, partial, s);
}

int launch_field_finish(const double2* partial, int S, int64_t M, int R, const double* pts,
                        const double* src, int nsrc, double k, double2 pfac, double2* phi_f,
                        double2* p_f, cudaStream_t s) {
  const int64_t cnt = M * R;
  if (cnt <= 0) return 0;
  field_finish_kernel<<<(unsigned)((cnt + 31) / 32), 256, 0, s>>>(partial, S, M, R, pts, src, nsrc,
                                                                  k, pfac, phi_f, p_f);
  return 1;
}

}  // namespace bemgpu
