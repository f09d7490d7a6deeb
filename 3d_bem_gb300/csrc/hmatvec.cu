// hmatvec.cu -- K5: H-matrix times a block of R vectors, y = beta*y + H x.
//
// Reference: HArithm::MVM (HMatrix/harithm.cpp:3-28) loops over the partition
// and scatters each block's U(s o (V^T x)) or F x into y under an omp critical.
// Here the product runs in two passes with no atomics and a fixed summation
// order:
//   pass V: t_b = s_b o (V_b x_C) for every admissible block, one warp per 16
//           rows of V;
//   pass U: one CTA (or cluster of CTAs) per leaf row cluster sums, for its
//           rows, every block whose row range contains them (U_b rows . t_b
//           and dense F_b rows . x_C).
// Every stored matrix entry is read once per call for all R vectors.
//
// Arithmetic variants (GB300's FP64 rate is far below what HBM can feed):
//   double2 storage, FP64 math  -- the plain complex-FP64 method;
//   float2 storage,  FP64 math  -- exact products of the stored operator;
//   float2 storage,  FP32 math  -- FP32 products inside a block, compensated
//                                  FP32 sums across blocks; the inner GMRES
//                                  operator;
//   float2 storage,  two-float  -- FP64-accurate products on the FP32 units;
//                                  the iterative-refinement residual.
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>

#include "bem_kernels.h"
#include "quadrature.cuh"

namespace bemgpu {
namespace {

namespace cg = cooperative_groups;

constexpr int VT = 128;          // threads of a pass-V CTA
constexpr int VCTAS_PER_SM = 64;  // pass-V CTAs beyond the long rows (16 or 64: the same)
constexpr int UT = 128;          // threads of a pass-U CTA

// Launch shapes, measured per product (V + U pass, us). Pass V: 4 columns ahead
// for one vector (20,480 sphere: 72 us; 2: 75, 1: 120), no unrolling for more
// (20,480 pencil, 8 vectors: 104 us; 2: 150, 4: 130 -- fewer warps fit).
// Pass U: 16 columns in flight and 6 CTAs of 128 per SM for one vector (20,480
// sphere 68 us; 8 columns and 8 CTAs 81, 32 and 4: 83, CTAs of 64: 120, of 256:
// 86), 8 columns for more (pencil, 8 vectors 107 us; 4 columns 121). Two-float
// sums spill beyond 4 columns.
__host__ __device__ constexpr int vunroll(int R) { return R == 1 ? 4 : 1; }
template <class A>
__host__ __device__ constexpr int ucolumns(int R) {
  return A::kLo ? 4 : (R == 1 ? 16 : 8);
}
__host__ __device__ constexpr int uctas(int R) { return R == 1 ? 6 : (R <= 3 ? 5 : 4); }

// ----- arithmetic policies: storage S, vector value X, accumulator Acc -----

// FP64 products of either storage; vectors in the caller's columns
template <typename T>
struct ArF64 {
  using S = T;
  using X = double2;
  using Acc = double2;
  static constexpr bool kInterleaved = false;
  static constexpr int kWords = 4;  // 32-bit registers of an accumulator
  static constexpr bool kLo = false;  // dense blocks may have a low part (near_fp64)
  static __device__ __forceinline__ Acc zero() { return make_double2(0.0, 0.0); }
  static __device__ __forceinline__ void fma(Acc& a, S v, X x) {
    double2 w;
    if constexpr (sizeof(T) == sizeof(float2)) w = make_double2((double)v.x, (double)v.y);
    else w = v;
    a.x += w.x * x.x - w.y * x.y;
    a.y += w.x * x.y + w.y * x.x;
  }
  static __device__ __forceinline__ void add(Acc& a, Acc b) {
    a.x += b.x;
    a.y += b.y;
  }
  static __device__ __forceinline__ Acc shfl(Acc a, int o) {
    return make_double2(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o));
  }
  static __device__ __forceinline__ X scaled(S s, Acc a) {  // s * a as a vector value
    double2 w;
    if constexpr (sizeof(T) == sizeof(float2)) w = make_double2((double)s.x, (double)s.y);
    else w = s;
    return cmul(w, a);
  }
};

// FP32 products and sums; vectors as FP32, the R values of an index together
struct ArF32 {
  using S = float2;
  using X = float2;
  using Acc = float2;
  static constexpr bool kInterleaved = true;
  static constexpr int kWords = 2;
  static constexpr bool kLo = false;
  static __device__ __forceinline__ Acc zero() { return make_float2(0.0f, 0.0f); }
  static __device__ __forceinline__ void fma(Acc& a, S v, X x) {
    a.x += v.x * x.x - v.y * x.y;
    a.y += v.x * x.y + v.y * x.x;
  }
  static __device__ __forceinline__ void add(Acc& a, Acc b) {
    a.x += b.x;
    a.y += b.y;
  }
  static __device__ __forceinline__ Acc shfl(Acc a, int o) {
    return make_float2(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o));
  }
  static __device__ __forceinline__ X scaled(S s, Acc a) { return fmul(s, a); }
};

// Two-float products and sums on complex-FP32 storage. x and t are unevaluated
// sums hi + lo of two floats; each stored entry a (exact in FP32) times hi is
// split exactly with an FMA (p + e = a * hi), and sums run in two-float
// precision (~2^-48). The refinement residual b - A x needs ~1e-14 relative
// accuracy but would be FP64-pipe-bound in native FP64 on GB300.
struct DF {
  float hi = 0, lo = 0;
  // this += a * (yh + yl), a exact
  __device__ __forceinline__ void fma(float a, float yh, float yl) {
    const float p = a * yh;
    const float ep = fmaf(a, yh, -p);
    const float s = hi + p;
    const float bb = s - hi;
    const float e = (hi - (s - bb)) + (p - bb);
    lo += e + ep + a * yl;
    hi = s;
  }
  __device__ __forceinline__ void add(float h2, float l2) {
    const float s = hi + h2;
    const float bb = s - hi;
    const float e = (hi - (s - bb)) + (h2 - bb);
    lo += e + l2;
    hi = s;
  }
};

// complex two-float accumulator
struct CDF {
  DF re, im;
  // += a * y, a = (ax, ay) exact floats, y = (yrh + yrl) + i (yih + yil)
  __device__ __forceinline__ void fma(float2 a, float4 y) {
    re.fma(a.x, y.x, y.y);
    re.fma(-a.y, y.z, y.w);
    im.fma(a.x, y.z, y.w);
    im.fma(a.y, y.x, y.y);
  }
};

struct ArDF {
  using S = float2;
  using X = float4;
  using Acc = CDF;
  static constexpr bool kInterleaved = true;
  static constexpr int kWords = 4;
  static constexpr bool kLo = true;
  static __device__ __forceinline__ Acc zero() { return CDF(); }
  static __device__ __forceinline__ void fma(Acc& a, S v, X x) { a.fma(v, x); }
  static __device__ __forceinline__ void add(Acc& a, const Acc& b) {
    a.re.add(b.re.hi, b.re.lo);
    a.im.add(b.im.hi, b.im.lo);
  }
  static __device__ __forceinline__ Acc shfl(const Acc& a, int o) {
    CDF b;
    b.re.hi = __shfl_xor_sync(0xffffffffu, a.re.hi, o);
    b.re.lo = __shfl_xor_sync(0xffffffffu, a.re.lo, o);
    b.im.hi = __shfl_xor_sync(0xffffffffu, a.im.hi, o);
    b.im.lo = __shfl_xor_sync(0xffffffffu, a.im.lo, o);
    return b;
  }
  static __device__ __forceinline__ X scaled(S s, const Acc& a) {
    CDF o;
    o.fma(s, make_float4(a.re.hi, a.re.lo, a.im.hi, a.im.lo));
    return make_float4(o.re.hi, o.re.lo, o.im.hi, o.im.lo);
  }
};

__device__ __forceinline__ float2 ldg_s(const float2* p) { return __ldg(p); }
__device__ __forceinline__ double2 ldg_s(const double2* p) { return __ldg(p); }

// The R vector values of index i: FP64 vectors in columns of ld (x, or t with
// its R values together), FP32 and two-float ones together, read as 16-byte
// pieces where R makes them aligned.
template <int R>
__device__ __forceinline__ void load_vec(const float2* __restrict__ p, int64_t i, float2 (&v)[R]) {
  if constexpr (R % 2 == 0) {
    const float4* q = reinterpret_cast<const float4*>(p + i * R);
#pragma unroll
    for (int r = 0; r < R; r += 2) {
      const float4 w = __ldg(q + r / 2);
      v[r] = make_float2(w.x, w.y);
      v[r + 1] = make_float2(w.z, w.w);
    }
  } else {
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = __ldg(p + i * R + r);
  }
}
template <int R>
__device__ __forceinline__ void load_vec(const float4* __restrict__ p, int64_t i, float4 (&v)[R]) {
#pragma unroll
  for (int r = 0; r < R; r++) v[r] = __ldg(p + i * R + r);
}
template <int R>
__device__ __forceinline__ void load_vec(const double2* __restrict__ p, int64_t i, double2 (&v)[R]) {
#pragma unroll
  for (int r = 0; r < R; r++) v[r] = __ldg(p + i * R + r);
}
template <class A, int R>
__device__ __forceinline__ void load_x(const typename A::X* __restrict__ x, int64_t ldx, int64_t i,
                                       typename A::X (&v)[R]) {
  if constexpr (A::kInterleaved) {
    load_vec<R>(x, i, v);
  } else {
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = __ldg(x + r * ldx + i);
  }
}
// ---------------------------------------------------------------------------
// Pass V: t[soff + l][r] = s_l * sum_j V[l, j] x[c0 + j, r].
// Work items come longest first, in two forms. Rows of more than HMV_VLONG
// entries: a CTA takes HMV_VLROWS rows, its warps a quarter of the columns each
// (a warp alone on 16 rows of 2,560 entries was the tail of the whole pass).
// Shorter ones: a warp takes 16 rows, its four groups of 8 lanes rows l0 + g +
// 4 i (i < G at a time). Most blocks are small (mean rank 17, mean row 126
// entries at 20,480 sphere elements), where the reduction over the lanes costs
// as much as the products: 8 lanes per row and a halving exchange (each step
// halves what a lane still sums) take 8 shuffles for 16 rows at R = 1; one row
// per warp step and a full butterfly took 160. A lane's plain FP32 sum has up to
// 32 terms; sums of 8 terms, or 32 lanes a row, change the error of a product in
// the third digit at most (sphere of 20,480, phi matrix: 8.84e-8 -> 8.81e-8) and
// take 7 to 30 us more there.
// ---------------------------------------------------------------------------

// acc[n] summed over the lanes that differ in the bits M, M / 2, .. 1 of their
// number: each step halves the values a lane keeps while their number is
// even; returns the index of the first value the lane ends with and clears
// `mine` where another lane holds the same sums
template <class A, int N, int M>
__device__ __forceinline__ int halve(typename A::Acc (&acc)[N], int lane, bool& mine) {
  if constexpr (M == 0) {
    return 0;
  } else if constexpr (N % 2 == 0) {
    using Acc = typename A::Acc;
    const bool up = lane & M;
    Acc half[N / 2];
#pragma unroll
    for (int i = 0; i < N / 2; i++) {
      const Acc send = up ? acc[i] : acc[i + N / 2];
      const Acc got = A::shfl(send, M);
      half[i] = up ? acc[i + N / 2] : acc[i];
      A::add(half[i], got);
    }
    const int o = halve<A, N / 2, M / 2>(half, lane, mine) + (up ? N / 2 : 0);
#pragma unroll
    for (int i = 0; i < N / 2; i++) acc[i] = half[i];
    return o;
  } else {
#pragma unroll
    for (int i = 0; i < N; i++) A::add(acc[i], A::shfl(acc[i], M));
    if (lane & M) mine = false;
    return halve<A, N, M / 2>(acc, lane, mine);
  }
}
// values a lane keeps after halve<A, n, m>
__host__ __device__ constexpr int kept(int n, int m) {
  return m == 0 ? n : kept(n % 2 == 0 ? n / 2 : n, m / 2);
}

// acc[i R + r] += sum over j = j0, j0 + step, .. < j1 of row[i][j] x[j, r]
template <class A, int R, int G>
__device__ __forceinline__ void vdots(const typename A::S* const (&row)[G],
                                      const typename A::X* __restrict__ x, int64_t ldx, int64_t c0,
                                      int j0, int j1, int step, typename A::Acc (&acc)[G * R]) {
  constexpr int UN = vunroll(R);
#pragma unroll UN
  for (int j = j0; j < j1; j += step) {
    typename A::S v[G];
#pragma unroll
    for (int i = 0; i < G; i++) v[i] = ldg_s(row[i] + j);
    typename A::X xv[R];
    load_x<A, R>(x, ldx, c0 + j, xv);
#pragma unroll
    for (int i = 0; i < G; i++)
#pragma unroll
      for (int r = 0; r < R; r++) A::fma(acc[i * R + r], v[i], xv[r]);
  }
}

// Expands the work list into records, so that a warp of pass V reaches its rows
// after one load instead of three dependent ones.
__global__ void vrec_kernel(const int2* __restrict__ vwork, int nlong, int64_t nvwork,
                            const FarBlock* __restrict__ far, const int32_t* __restrict__ rank,
                            HmvVRec* __restrict__ rec) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= nvwork) return;
  const int2 w = vwork[i];
  const FarBlock fb = far[w.x];
  HmvVRec r;
  r.voff = fb.voff + (int64_t)w.y * fb.n;
  r.soff = fb.soff + w.y;
  r.c0 = (int32_t)fb.c0;
  r.n = fb.n;
  r.rows = min(i < nlong ? HMV_VLROWS : HMV_VROWS, rank[w.x] - w.y);
  r.pad = 0;
  rec[i] = r;
}

__device__ __forceinline__ HmvVRec load_rec(const HmvVRec* p) {
  HmvVRec r;
  const int4 a = __ldg(reinterpret_cast<const int4*>(p));
  const int4 b = __ldg(reinterpret_cast<const int4*>(p) + 1);
  r.voff = (int64_t)(uint32_t)a.x | ((int64_t)a.y << 32);
  r.soff = (int64_t)(uint32_t)a.z | ((int64_t)a.w << 32);
  r.c0 = b.x;
  r.n = b.y;
  r.rows = b.z;
  return r;
}

template <class A, int R, int G>
__global__ void __launch_bounds__(VT) hmv_vpass(const HmvVRec* __restrict__ rec, int nlong,
                                                int64_t nrec,
                                                const typename A::S* __restrict__ Vp,
                                                const typename A::S* __restrict__ Sp,
                                                const typename A::X* __restrict__ x, int64_t ldx,
                                                typename A::X* __restrict__ t, HmvGate gate) {
  using S = typename A::S;
  using Acc = typename A::Acc;
  if (gate_closed(gate)) return;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if ((int)blockIdx.x < nlong) {
    constexpr int GL = G < HMV_VLROWS ? G : HMV_VLROWS;  // rows at a time
    constexpr int K = kept(GL * R, 16);
    __shared__ Acc part[VT / 32][GL][R];
    const HmvVRec rc = load_rec(rec + blockIdx.x);
    const int quarter = (rc.n + VT / 32 - 1) / (VT / 32);
    const int jb = w * quarter, je = min(rc.n, jb + quarter);
    for (int l0 = 0; l0 < rc.rows; l0 += GL) {
      const S* row[GL];
#pragma unroll
      for (int i = 0; i < GL; i++)  // rows past the end repeat the last one
        row[i] = Vp + rc.voff + (int64_t)min(l0 + i, rc.rows - 1) * rc.n;
      Acc acc[GL * R];
#pragma unroll
      for (int i = 0; i < GL * R; i++) acc[i] = A::zero();
      vdots<A, R, GL>(row, x, ldx, rc.c0, jb + lane, je, 32, acc);
      bool mine = true;
      const int o = halve<A, GL * R, 16>(acc, lane, mine);
      if (mine) {
#pragma unroll
        for (int i = 0; i < K; i++) part[w][(o + i) / R][(o + i) % R] = acc[i];
      }
      __syncthreads();
      if (threadIdx.x < GL * R) {
        const int l = threadIdx.x / R, r = threadIdx.x % R;
        Acc v = part[0][l][r];
#pragma unroll
        for (int q = 1; q < VT / 32; q++) A::add(v, part[q][l][r]);
        if (l0 + l < rc.rows)
          t[(rc.soff + l0 + l) * R + r] = A::scaled(ldg_s(Sp + rc.soff + l0 + l), v);
      }
      __syncthreads();
    }
    return;
  }
  // the shorter items, dealt to the warps of the grid in turn (longest first);
  // the next record is loaded while the current one's rows are
  const int64_t stride = (int64_t)(gridDim.x - nlong) * (VT / 32);
  int64_t item = nlong + (int64_t)(blockIdx.x - nlong) * (VT / 32) + w;
  if (item >= nrec) return;
  const int g = lane >> 3, c = lane & 7;
  constexpr int K = kept(G * R, 4);
  HmvVRec rc = load_rec(rec + item);
  while (true) {
    const int64_t next = item + stride;
    const HmvVRec rn = load_rec(rec + (next < nrec ? next : item));
    const S sl = ldg_s(Sp + rc.soff + min(lane, rc.rows - 1));  // lane l: scale of row l
    for (int q0 = 0; q0 < rc.rows; q0 += 4 * G) {
      const S* row[G];
#pragma unroll
      for (int i = 0; i < G; i++)  // rows past the end repeat the last one
        row[i] = Vp + rc.voff + (int64_t)min(q0 + g + 4 * i, rc.rows - 1) * rc.n;
      Acc acc[G * R];
#pragma unroll
      for (int i = 0; i < G * R; i++) acc[i] = A::zero();
      vdots<A, R, G>(row, x, ldx, rc.c0, c, rc.n, 8, acc);
      bool mine = true;
      const int o = halve<A, G * R, 4>(acc, lane, mine);
#pragma unroll
      for (int i = 0; i < K; i++) {
        const int l = q0 + g + 4 * ((o + i) / R);
        S sc;
        sc.x = __shfl_sync(0xffffffffu, sl.x, l);
        sc.y = __shfl_sync(0xffffffffu, sl.y, l);
        if (mine && l < rc.rows) t[(rc.soff + l) * R + (o + i) % R] = A::scaled(sc, acc[i]);
      }
    }
    if (next >= nrec) break;
    item = next;
    rc = rn;
  }
}

// ---------------------------------------------------------------------------
// Pass U: y rows of a leaf += U t of its admissible and F x of its dense
// blocks. The CTAs of a cluster (one, two or four) load the descriptors of the
// leaf's blocks into shared memory at once, lay all their columns end to end
// and give every warp the same number of consecutive columns; lanes own rows. A
// warp takes 32 columns at a time: lane i finds the block and address of the
// i-th, loads its values of t or x and leaves both in shared memory, where the
// loop over the columns reads them as broadcasts. So the loads in flight do not
// stop at the end of a block (mean rank 17), and blocks of rank 5 and 80 do not
// unbalance the warps. FP32 sums are plain over 16 columns and compensated beyond:
// over 32 a product of 20,480 elements was 1.04e-7 to 1.09e-7 from the exact one, so
// 0.79e-7 to 0.86e-7 (sums per block, as before the columns were laid end to end:
// 0.95e-7 to 1.02e-7). The partial sums of the warps and CTAs are added in a fixed
// order. Bound by the bytes of U and F for one vector (20,480 sphere, 351 MB: 68 us,
// 5.2 TB/s; one warp per block with 125 us before) and by the shared-memory
// broadcasts and FMAs for eight (pencil, 20,480: 117 us, 107 with sums of 32 columns,
// before 221 us).
// ---------------------------------------------------------------------------

// FP32 sums across blocks, compensated
struct TwoSum {
  float hi = 0, lo = 0;
  __device__ __forceinline__ void add(float v) {
    const float s = hi + v;
    const float bp = s - hi;
    lo += (hi - (s - bp)) + (v - bp);
    hi = s;
  }
};

// two FP32 FMAs as one instruction: same FMA rate, half the issue slots
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t ffma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// Row sums of a warp over its columns: column() per column, flush() after 16 of
// them; total[r][lane] (shared memory, zero at first) holds what is summed over
// the warps in the end.
template <class A, int R>
struct RowSum {  // FP64, two-float
  using Out = typename A::Acc;
  static __device__ __forceinline__ Out none() { return A::zero(); }
  typename A::Acc acc[R];
  __device__ __forceinline__ RowSum() {
#pragma unroll
    for (int r = 0; r < R; r++) acc[r] = A::zero();
  }
  __device__ __forceinline__ void column(typename A::S u, const typename A::X* v) {
#pragma unroll
    for (int r = 0; r < R; r++) A::fma(acc[r], u, v[r]);
  }
  __device__ __forceinline__ void flush(Out (*total)[32], int lane) {}
  __device__ __forceinline__ void finish(Out (*total)[32], int lane) {
#pragma unroll
    for (int r = 0; r < R; r++) total[r][lane] = acc[r];
  }
  static __device__ __forceinline__ void join(Out& a, const Out& b) { A::add(a, b); }
};
template <int R>
struct RowSum<ArF32, R> {
  using Out = float4;  // compensated sums (re.hi, re.lo, im.hi, im.lo)
  static __device__ __forceinline__ Out none() { return make_float4(0.0f, 0.0f, 0.0f, 0.0f); }
  // partial sums of up to 16 columns; with 4 or more vectors as packed pairs: pa
  // sums u.x (t.x, t.y) and pb sums u.y (t.x, t.y), re = pa.x - pb.y,
  // im = pa.y + pb.x
  static constexpr bool kPacked = R >= 4;
  uint64_t pa[kPacked ? R : 1], pb[kPacked ? R : 1];
  float2 acc[kPacked ? 1 : R];
  __device__ __forceinline__ RowSum() { clear(); }
  __device__ __forceinline__ void clear() {
    if constexpr (kPacked) {
#pragma unroll
      for (int r = 0; r < R; r++) pa[r] = pb[r] = 0;
    } else {
#pragma unroll
      for (int r = 0; r < R; r++) acc[r] = make_float2(0.0f, 0.0f);
    }
  }
  __device__ __forceinline__ void column(float2 u, const float2* v) {
    if constexpr (kPacked) {
      const uint64_t ux = pack2(u.x, u.x), uy = pack2(u.y, u.y);
#pragma unroll
      for (int r = 0; r < R; r++) {
        const uint64_t w = pack2(v[r].x, v[r].y);
        pa[r] = ffma2(ux, w, pa[r]);
        pb[r] = ffma2(uy, w, pb[r]);
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; r++) ArF32::fma(acc[r], u, v[r]);
    }
  }
  __device__ __forceinline__ void flush(Out (*total)[32], int lane) {
#pragma unroll
    for (int r = 0; r < R; r++) {
      float2 s;
      if constexpr (kPacked) {
        const float2 a = unpack2(pa[r]), b = unpack2(pb[r]);
        s = make_float2(a.x - b.y, a.y + b.x);
      } else {
        s = acc[r];
      }
      const Out o = total[r][lane];
      TwoSum sx{o.x, o.y}, sy{o.z, o.w};
      sx.add(s.x);
      sy.add(s.y);
      total[r][lane] = make_float4(sx.hi, sx.lo, sy.hi, sy.lo);
    }
    clear();
  }
  __device__ __forceinline__ void finish(Out (*total)[32], int lane) {}
  static __device__ __forceinline__ void join(Out& a, const Out& b) {
    TwoSum x{a.x, a.y}, y{a.z, a.w};
    x.add(b.x);
    x.add(b.y);
    y.add(b.z);
    y.add(b.w);
    a = make_float4(x.hi, x.lo, y.hi, y.lo);
  }
};
__device__ __forceinline__ double2 out_value(double2 v) { return v; }
__device__ __forceinline__ double2 out_value(const float4& v) {
  return make_double2((double)v.x + (double)v.y, (double)v.z + (double)v.w);
}
__device__ __forceinline__ double2 out_value(const CDF& v) {
  return make_double2((double)v.re.hi + (double)v.re.lo, (double)v.im.hi + (double)v.im.lo);
}

// inclusive prefix sums of v over the CTA; total returned in sum
template <int NW>
__device__ __forceinline__ int cta_scan(int v, int (&scan)[NW], int& sum) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  if (lane == 31) scan[w] = v;
  __syncthreads();
  sum = 0;
  int before = 0;
#pragma unroll
  for (int q = 0; q < NW; q++) {
    before += q < w ? scan[q] : 0;
    sum += scan[q];
  }
  __syncthreads();
  return before + v;
}

template <class A, int R, int MINB, int UN>
__global__ void __launch_bounds__(UT, MINB) hmv_upass(
    const LeafRows* __restrict__ leaves, const int32_t* __restrict__ list_off,
    const int32_t* __restrict__ list, const FarBlock* __restrict__ far,
    const int32_t* __restrict__ rank, const NearBlock* __restrict__ nearb,
    const typename A::S* __restrict__ Up, const typename A::S* __restrict__ F,
    const typename A::S* __restrict__ Flo, const typename A::X* __restrict__ x, int64_t ldx,
    const typename A::X* __restrict__ t, double2* __restrict__ y, int64_t ldy, int accumulate,
    int ncta, HmvGate gate) {
  using S = typename A::S;
  using X = typename A::X;
  using Sum = RowSum<A, R>;
  using Out = typename Sum::Out;
  static_assert(16 % UN == 0, "flush() after 16 columns");
  constexpr int NW = UT / 32;
  struct __align__(16) Stage {  // the warp's 32 columns
    X v[32][R];
    const S* ptr[32];
  };
  __shared__ const S* d_ptr[UT];  // first column at the leaf's row base
  __shared__ int d_ld[UT];        // column stride
  __shared__ int d_vec[UT];       // first index into t or x
  __shared__ int d_end[2][UT];    // columns up to the end of the block: admissible, dense
  __shared__ int scan[NW];
  __shared__ __align__(16) unsigned char stage_raw[sizeof(Stage) * NW];
  __shared__ __align__(16) unsigned char part_raw[sizeof(Out) * NW * R * 32];
  Out(*part)[R][32] = reinterpret_cast<Out(*)[R][32]>(part_raw);
  if (gate_closed(gate)) return;  // the same for every CTA of a cluster
  const int leaf = blockIdx.x / ncta, cta = blockIdx.x - leaf * ncta;
  const LeafRows lf = leaves[leaf];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Stage& st = reinterpret_cast<Stage*>(stage_raw)[w];
  const int beg = list_off[leaf], end = list_off[leaf + 1];
  const int nwarp = ncta * NW, me = cta * NW + w;
  for (int base = 0; base < lf.size; base += 32) {
    const bool active = base + lane < lf.size;
    const int64_t grow = lf.start + base;
    const int my = active ? lane : 0;  // idle lanes repeat the first row
    Sum sum;
#pragma unroll
    for (int r = 0; r < R; r++) part[w][r][lane] = Sum::none();
    for (int e0 = beg; e0 < end; e0 += UT) {
      const int e = e0 + threadIdx.x, cntb = min(UT, end - e0);
      int nf = 0, nn = 0;
      if (e < end) {
        const int32_t code = list[e];
        if (code >= 0) {
          const FarBlock fb = far[code];
          nf = rank[code];
          d_ptr[threadIdx.x] = Up + fb.uoff + (grow - fb.r0);
          d_ld[threadIdx.x] = fb.m;
          d_vec[threadIdx.x] = (int)fb.soff;
        } else {
          const NearBlock nb = nearb[-code - 1];
          nn = nb.n;
          d_ptr[threadIdx.x] = F + nb.off + (grow - nb.r0);
          d_ld[threadIdx.x] = nb.m;
          d_vec[threadIdx.x] = (int)nb.c0;
        }
      }
      int total[2];
      d_end[0][threadIdx.x] = cta_scan<NW>(nf, scan, total[0]);
      d_end[1][threadIdx.x] = cta_scan<NW>(nn, scan, total[1]);
      __syncthreads();
#pragma unroll
      for (int dense = 0; dense < 2; dense++) {
        const int* ends = d_end[dense];
        const int c1 = (int)((int64_t)total[dense] * (me + 1) / nwarp);
        int c = (int)((int64_t)total[dense] * me / nwarp);
        // the lane's column of the 32 from c (past the end: the last one)
        const S* ptr = nullptr;
        X v[R];
        const auto find = [&]() {
          const int col = min(c + lane, c1 - 1);
          int lo = 0, hi = cntb - 1;  // first block that ends after it
          while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (ends[mid] > col) hi = mid;
            else lo = mid + 1;
          }
          const int l = col - (lo > 0 ? ends[lo - 1] : 0);
          ptr = d_ptr[lo] + (int64_t)l * d_ld[lo];
          if (dense) load_x<A, R>(x, ldx, d_vec[lo] + l, v);
          else load_vec<R>(t, d_vec[lo] + l, v);
        };
        if (c < c1) find();
        while (c < c1) {
          const int nb = min(32, c1 - c);
          __syncwarp();
          st.ptr[lane] = ptr;
#pragma unroll
          for (int r = 0; r < R; r++) st.v[lane][r] = v[r];
          __syncwarp();
          c += 32;
          if (c < c1) find();  // the next 32 load meanwhile
          for (int i = 0; i < nb; i += UN) {
            S u[UN];
#pragma unroll
            for (int q = 0; q < UN; q++) {
              u[q] = ldg_s(st.ptr[i + q] + my);
              if (i + q >= nb) u[q].x = u[q].y = 0;
            }
#pragma unroll
            for (int q = 0; q < UN; q++) sum.column(u[q], st.v[i + q]);
            if constexpr (A::kLo) {
              if (dense && Flo) {  // FP64 entries as hi + lo
#pragma unroll
                for (int q = 0; q < UN; q++) {
                  u[q] = ldg_s(Flo + (st.ptr[i + q] - F) + my);
                  if (i + q >= nb) u[q].x = u[q].y = 0;
                }
#pragma unroll
                for (int q = 0; q < UN; q++) sum.column(u[q], st.v[i + q]);
              }
            }
            if (i + UN == 16 && nb > 16) sum.flush(part[w], lane);
          }
          sum.flush(part[w], lane);
        }
      }
      __syncthreads();
    }
    sum.finish(part[w], lane);
    __syncthreads();
    for (int i = threadIdx.x; i < R * 32; i += UT) {
      const int r = i >> 5;
      Out s = part[0][r][lane];
#pragma unroll
      for (int q = 1; q < NW; q++) Sum::join(s, part[q][r][lane]);
      part[0][r][lane] = s;
    }
    if (ncta > 1) {
      cg::cluster_group cl = cg::this_cluster();
      cl.sync();
      if (cta == 0)
        for (int i = threadIdx.x; i < R * 32; i += UT) {
          const int r = i >> 5;
          Out s = part[0][r][lane];
          for (int q = 1; q < ncta; q++) Sum::join(s, *cl.map_shared_rank(&part[0][r][lane], q));
          part[0][r][lane] = s;
        }
      cl.sync();
    }
    if (cta == 0)
      for (int i = threadIdx.x; i < R * 32; i += UT)
        if (active) {
          const double2 v = out_value(part[0][i >> 5][lane]);
          double2* yp = y + (i >> 5) * ldy + grow + lane;
          *yp = accumulate ? cadd(*yp, v) : v;
        }
    __syncthreads();
  }
}

// FP32 and two-float copies of the vectors, the R values of an index together
__global__ void to_float_kernel(const double2* __restrict__ x, int64_t ldx, int R,
                                float2* __restrict__ xf, HmvGate gate) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= ldx || gate_closed(gate)) return;
  for (int r = 0; r < R; r++) {
    const double2 v = x[r * ldx + i];
    xf[i * R + r] = make_float2((float)v.x, (float)v.y);
  }
}

__global__ void to_df_kernel(const double2* __restrict__ x, int64_t ldx, int R,
                             float4* __restrict__ xd) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= ldx) return;
  for (int r = 0; r < R; r++) {
    const double2 v = x[r * ldx + i];
    const float rh = (float)v.x, ih = (float)v.y;
    xd[i * R + r] =
        make_float4(rh, (float)(v.x - (double)rh), ih, (float)(v.y - (double)ih));
  }
}

// streaming multiprocessors of the current device (cached per device)
int sm_count() {
  static int cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 152;
  if (!cached[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 152;
    cached[dev] = n;
  }
  return cached[dev];
}

template <class A, int R>
void launch_passes(const HmvArgs& a, const typename A::X* x, typename A::X* t, cudaStream_t s) {
  using S = typename A::S;
  // rows per lane group: as many as about 64 accumulator registers hold
  constexpr int G = A::kWords * R * 4 <= 64 ? 4 : (A::kWords * R * 2 <= 64 ? 2 : 1);
  if (a.nvwork > 0) {
    const int64_t rest = (a.nvwork - a.nlong + VT / 32 - 1) / (VT / 32);
    const int64_t grid = a.nlong + std::min<int64_t>(rest, (int64_t)VCTAS_PER_SM * sm_count());
    hmv_vpass<A, R, G><<<(unsigned)grid, VT, 0, s>>>(a.vrec, (int)a.nlong, a.nvwork, (const S*)a.V,
                                                     (const S*)a.S, x, a.ldx, t, a.gate);
  }
  if (a.nleaves <= 0) return;
  // CTAs per leaf: with fewer than 16 warps per SM a leaf's columns go to a
  // cluster of two, below 5 to one of four. Products of one vector on boxes, with
  // one / two / four CTAs (us): 33 leaves FP64 49 / 35 / 29, 160 leaves 187 / 163 /
  // 160, 263 leaves (7 warps per SM) FP32 45 / 41 / 46, 360 leaves 63 / 54 / 60, 499
  // leaves (13) 70 / 74 / 77, 660 leaves (17) 82 / 89 / 91; FP64 above 263 leaves
  // within 5 %, 8 vectors alike.
  const int64_t per_sm = a.nleaves * (UT / 32) / sm_count();
  const int ncta = per_sm >= 16 ? 1 : (per_sm >= 5 ? 2 : 4);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(a.nleaves * ncta));
  cfg.blockDim = dim3(UT);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)ncta;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = ncta > 1 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, hmv_upass<A, R, uctas(R), ucolumns<A>(R)>, a.leaves, a.list_off, a.list,
                     a.far, a.rank, a.nearb, (const S*)a.U, (const S*)a.F, (const S*)a.Flo, x,
                     a.ldx, (const typename A::X*)t, a.y, a.ldy, a.accumulate, ncta, a.gate);
}

template <int R>
void launch32_r(const HmvArgs& a, cudaStream_t s) {
  to_float_kernel<<<(unsigned)((a.ldx + 255) / 256), 256, 0, s>>>(a.x, a.ldx, R, a.xf, a.gate);
  launch_passes<ArF32, R>(a, a.xf, a.tf, s);
}

template <int R>
void launchdf_r(const HmvArgs& a, cudaStream_t s) {
  float4* xd = (float4*)a.xf;
  to_df_kernel<<<(unsigned)((a.ldx + 255) / 256), 256, 0, s>>>(a.x, a.ldx, R, xd);
  launch_passes<ArDF, R>(a, xd, (float4*)a.tf, s);
}

void launch32(const HmvArgs& a, cudaStream_t s) {
  switch (a.nrhs) {
    case 1: launch32_r<1>(a, s); break;
    case 2: launch32_r<2>(a, s); break;
    case 3: launch32_r<3>(a, s); break;
    case 4: launch32_r<4>(a, s); break;
    case 5: launch32_r<5>(a, s); break;
    case 6: launch32_r<6>(a, s); break;
    case 7: launch32_r<7>(a, s); break;
    default: launch32_r<8>(a, s); break;
  }
}

void launchdf(const HmvArgs& a, cudaStream_t s) {
  switch (a.nrhs) {
    case 1: launchdf_r<1>(a, s); break;
    case 2: launchdf_r<2>(a, s); break;
    case 3: launchdf_r<3>(a, s); break;
    default: launchdf_r<4>(a, s); break;  // the runtime passes at most 4 per pass
  }
}

template <typename T>
void launch64(const HmvArgs& a, cudaStream_t s) {
  switch (a.nrhs) {
    case 1: launch_passes<ArF64<T>, 1>(a, a.x, a.t, s); break;
    case 2: launch_passes<ArF64<T>, 2>(a, a.x, a.t, s); break;
    case 3: launch_passes<ArF64<T>, 3>(a, a.x, a.t, s); break;
    case 4: launch_passes<ArF64<T>, 4>(a, a.x, a.t, s); break;
    case 5: launch_passes<ArF64<T>, 5>(a, a.x, a.t, s); break;
    case 6: launch_passes<ArF64<T>, 6>(a, a.x, a.t, s); break;
    case 7: launch_passes<ArF64<T>, 7>(a, a.x, a.t, s); break;
    default: launch_passes<ArF64<T>, 8>(a, a.x, a.t, s); break;  // the runtime splits R > 8
  }
}
}  // namespace

// ---------------------------------------------------------------------------
// Fixed scratch for bem_hmatvec_noalloc: the per-block projections t = s o (V x)
// of one pass (ldt x nrhs complex FP64 values) live in this file-scope device
// array instead of a cudaMalloc'd buffer. Every GPU that loads the library
// holds it (32 MiB) until the process exits; all calls share it, so calls that
// overlap on the GPU race. Nothing in it needs clearing: pass V writes every
// entry pass U reads.
// ---------------------------------------------------------------------------
static __device__ __align__(256) double2 g_noalloc_t[HMV_NOALLOC_SCRATCH];

int64_t hmatvec_noalloc_capacity() { return HMV_NOALLOC_SCRATCH; }

// Device address of the scratch array on the current device. The first call
// on each device looks it up (cudaGetSymbolAddress, with that device current);
// later calls reuse the cached address. The cache is keyed by device ordinal,
// i.e. it assumes the device's primary context (the one the CUDA runtime
// uses): after cudaDeviceReset, or under a driver-API context of its own, the
// cached address no longer belongs to the current context.
cudaError_t hmatvec_noalloc_scratch(double2** out) {
  static std::mutex mu;
  static void* addr[256] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 256) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_t);
    if (e != cudaSuccess) return e;
    addr[dev] = p;
  }
  *out = static_cast<double2*>(addr[dev]);
  return cudaSuccess;
}

void launch_vrec(const HmvArgs& a, HmvVRec* rec, cudaStream_t s) {
  if (a.nvwork > 0)
    vrec_kernel<<<(unsigned)((a.nvwork + 255) / 256), 256, 0, s>>>(a.vwork, (int)a.nlong, a.nvwork,
                                                                   a.far, a.rank, rec);
}

int launch_hmatvec(const HmvArgs& a, cudaStream_t s) {
  if (a.precision == 0) launch64<double2>(a, s);
  else if (a.fp32_math == 1) {
    launch32(a, s);
    return 1 + (a.nfar > 0) + (a.nleaves > 0);
  } else if (a.fp32_math == 2) {
    launchdf(a, s);
    return 1 + (a.nfar > 0) + (a.nleaves > 0);
  } else launch64<float2>(a, s);
  return (a.nfar > 0) + (a.nleaves > 0);
}

}  // namespace bemgpu
