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
// sums in FP32 folded into FP64 accumulators every 128 (32) elements. Precision 0: the
// same sum in FP64.
#include "field.h"
#include "phase.cuh"

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
    // the element's half of its pair; the last one of an odd count writes both
    float* f = reinterpret_cast<float*>(static_cast<FieldPairF*>(fe) + (j >> 1));
    float v[30];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const float hi = (float)e.c[d];
      v[d] = -hi;
      v[3 + d] = -(float)(e.c[d] - (double)hi);
      v[27 + d] = (float)e.nrm[d];
    }
#pragma unroll
    for (int i = 0; i < 7; i++) {
      const double a1 = cR7x1[i], a2 = cR7x2[i], a3 = 1.0 - a2 - a1;
#pragma unroll
      for (int d = 0; d < 3; d++)
        v[6 + 3 * i + d] = -(float)((a1 * e.n1[d] + a2 * e.n2[d] + a3 * e.n3[d]) - e.c[d]);
    }
    const bool alone = j == N - 1 && !(j & 1);
#pragma unroll
    for (int i = 0; i < 30; i++) {
      f[2 * i + (j & 1)] = v[i];
      if (alone) f[2 * i + 1] = v[i];
    }
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
      float* c = reinterpret_cast<float*>(static_cast<FieldCoefPairF*>(coef) +
                                          (int64_t)r * ((N + 1) / 2) + (j >> 1));
      const float v[4] = {(float)(A * p.x), (float)(A * p.y), (float)(A * dp.x), (float)(A * dp.y)};
#pragma unroll
      for (int i = 0; i < 4; i++) {
        c[2 * i + (j & 1)] = v[i];
        if (j == N - 1 && !(j & 1)) c[2 * i + 1] = 0.0f;
      }
    } else {
      FieldCoef c;
      c.a = make_double2(A * p.x, A * p.y);
      c.b = make_double2(A * dp.x, A * dp.y);
      static_cast<FieldCoef*>(coef)[(int64_t)r * N + j] = c;
    }
  }
}

// Two FP32 values as one operand: an add, multiply or FMA of both takes one
// issue slot (and twice the pipe cycles of a scalar one).
struct P2 {
  uint64_t v;
};
__device__ __forceinline__ P2 p2(float a, float b) {
  P2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 f2(P2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
  return r;
}
__device__ __forceinline__ P2 add2(P2 a, P2 b) {
  P2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ P2 mul2(P2 a, P2 b) {
  P2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ P2 fma2(P2 a, P2 b, P2 c) {
  P2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Columns r0 .. r0 + RB - 1, element chunk blockIdx.y. Bound by the special
// functions (rsqrt, sin and cos of every rule point, 8 cycles a warp each: 168 of
// them per element) beside the FMA pipe (about as much); issue slots were the
// limit with scalar arithmetic (258 per element, 86 % of the cycles), so two
// elements go through every operation together. (p - q) . n is the same for all
// points of an element's plane, and the radial part is summed as
// sum w (cos, sin) / r^3 and k sum w (cos, sin) / r^2. 20,480 elements x 20,480
// points, one column: 2.31 ms (3.07 ms with scalar arithmetic).
template <int RB, int FIELD_PTS>
__global__ void __launch_bounds__(FIELD_PTS)
    field_sum32_kernel(const FieldPairF* __restrict__ fe, const FieldCoefPairF* __restrict__ coef,
                       int64_t NP, int64_t chunk, const double* __restrict__ pts, int64_t M,
                       float k, float kc, int r0, int R, double2* __restrict__ partial) {
  constexpr int TILE = FIELD_PTS / 4;  // pairs
  __shared__ FieldPairF se[TILE];
  __shared__ FieldCoefPairF sc[RB][TILE];
  const int64_t ip = (int64_t)blockIdx.x * FIELD_PTS + threadIdx.x;
  const int64_t e0 = (int64_t)blockIdx.y * chunk;
  const int64_t e1 = min(NP, e0 + chunk);
  P2 ph[3], pl[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const double v = ip < M ? pts[3 * ip + d] : 0.0;
    const float hi = (float)v, lo = (float)(v - (double)hi);
    ph[d] = p2(hi, hi);
    pl[d] = p2(lo, lo);
  }
  const P2 kc2 = p2(kc, kc), k2 = p2(k, k), nk2 = p2(-k, -k), minus = p2(-1.0f, -1.0f);
  const float magic = 12582912.0f;  // 1.5 2^23: adding it rounds to an integer
  const P2 mg = p2(magic, magic), nmg = p2(-magic, -magic);
  const P2 twopi = p2(6.28318530717959f, 6.28318530717959f);
  double ax[RB], ay[RB];
#pragma unroll
  for (int r = 0; r < RB; r++) ax[r] = ay[r] = 0.0;
  for (int64_t t0 = e0; t0 < e1; t0 += TILE) {
    const int nt = (int)min((int64_t)TILE, e1 - t0);
    __syncthreads();
    const float4* src = reinterpret_cast<const float4*>(fe + t0);
    float4* dst = reinterpret_cast<float4*>(se);
    constexpr int PIECES = (int)(sizeof(FieldPairF) / sizeof(float4));
    for (int i = threadIdx.x; i < nt * PIECES; i += FIELD_PTS) dst[i] = src[i];
    for (int i = threadIdx.x; i < RB * nt; i += FIELD_PTS) {
      const int r = i / nt, j = i - r * nt;
      sc[r][j] = coef[(int64_t)(r0 + r) * NP + t0 + j];
    }
    __syncthreads();
    P2 tx[RB], ty[RB];
#pragma unroll
    for (int r = 0; r < RB; r++) tx[r] = ty[r] = p2(0.0f, 0.0f);
    for (int j = 0; j < nt; j++) {
      const ulonglong2* E = reinterpret_cast<const ulonglong2*>(&se[j]);
      P2 f[30];
#pragma unroll
      for (int i = 0; i < 15; i++) {
        const ulonglong2 v = E[i];
        f[2 * i].v = v.x;
        f[2 * i + 1].v = v.y;
      }
      const P2 dx = add2(add2(ph[0], f[0]), add2(pl[0], f[3]));
      const P2 dy = add2(add2(ph[1], f[1]), add2(pl[1], f[4]));
      const P2 dz = add2(add2(ph[2], f[2]), add2(pl[2], f[5]));
      const P2 dn = fma2(dx, f[27], fma2(dy, f[28], mul2(dz, f[29])));
      const P2 zero = p2(0.0f, 0.0f);
      P2 Lx = zero, Ly = zero, Ax = zero, Ay = zero, Bx = zero, By = zero;
#pragma unroll
      for (int i = 0; i < 7; i++) {
        const P2 rx = add2(dx, f[6 + 3 * i]), ry = add2(dy, f[7 + 3 * i]), rz = add2(dz, f[8 + 3 * i]);
        const P2 rr = fma2(rx, rx, fma2(ry, ry, mul2(rz, rz)));
        const float2 q = f2(rr);
        const P2 ir = p2(rsqrt_approx(q.x), rsqrt_approx(q.y));
        // exp(ikr): x = k r / (2 pi) reduced exactly to [-1/2, 1/2] (x - rint(x)
        // has no rounding), then the hardware sin / cos on 2 pi (x - rint(x))
        const P2 x = mul2(kc2, mul2(rr, ir));
        const P2 xr = mul2(fma2(add2(add2(x, mg), nmg), minus, x), twopi);
        const float2 t = f2(xr);
        const P2 cs = p2(__cosf(t.x), __cosf(t.y)), sn = p2(__sinf(t.x), __sinf(t.y));
        const P2 g0 = mul2(ir, p2(cR7gf[i], cR7gf[i]));  // w / (4 pi r)
        const P2 g1 = mul2(g0, ir), g2 = mul2(g1, ir);
        Lx = fma2(g0, cs, Lx);
        Ly = fma2(g0, sn, Ly);
        Ax = fma2(g2, cs, Ax);
        Ay = fma2(g2, sn, Ay);
        Bx = fma2(g1, cs, Bx);
        By = fma2(g1, sn, By);
      }
      // w dG/dr rnq = (p - q) . n w / r^3 (cos + kr sin, sin - kr cos)
      const P2 Mx = mul2(dn, fma2(k2, By, Ax)), My = mul2(dn, fma2(nk2, Bx, Ay));
      const P2 nMy = mul2(My, minus), nLx = mul2(Lx, minus), nLy = mul2(Ly, minus);
#pragma unroll
      for (int r = 0; r < RB; r++) {
        const ulonglong2* C = reinterpret_cast<const ulonglong2*>(&sc[r][j]);
        const ulonglong2 c0 = C[0], c1 = C[1];
        const P2 cax{c0.x}, cay{c0.y}, cbx{c1.x}, cby{c1.y};
        tx[r] = fma2(Mx, cax, fma2(nMy, cay, fma2(nLx, cbx, fma2(Ly, cby, tx[r]))));
        ty[r] = fma2(Mx, cay, fma2(My, cax, fma2(nLx, cby, fma2(nLy, cbx, ty[r]))));
      }
    }
#pragma unroll
    for (int r = 0; r < RB; r++) {
      const float2 sx = f2(tx[r]), sy = f2(ty[r]);
      ax[r] += (double)(sx.x + sx.y);
      ay[r] += (double)(sy.x + sy.y);
    }
  }
  if (ip < M) {
#pragma unroll
    for (int r = 0; r < RB; r++)
      partial[((int64_t)blockIdx.y * R + r0 + r) * M + ip] = make_double2(ax[r], ay[r]);
  }
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
    const double r = newton_sqrt(rr, ir);
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
        static_cast<const FieldPairF*>(fe), static_cast<const FieldCoefPairF*>(coef),
        field_pairs(N), (chunk + 1) / 2, pts, M, (float)k, (float)kc, r0, R, partial);
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
