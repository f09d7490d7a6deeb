// hlu_solve.cu -- K7: the H-LU preconditioner's forward and backward
// block-triangular solves, x = U^{-1} L^{-1} b, for R right-hand sides.
//
// Reference: HArithm::forwardSubstitution / backwardSubstitution
// (HMatrix/harithm.cpp:1314-1340, :1386-1412), called twice per GMRES
// iteration by LUPrecondidionedHMatrixWrapper (HMatrix/gmres.h:134-147). The
// recursion is flattened on the host into a schedule of leaf operations in
// exactly the reference's order: a diagonal leaf (QR leaf: y = Q^H w forward,
// R x = w backward) or an off-diagonal leaf (w_rows -= B x_cols, B full or
// low rank). Each diagonal leaf depends on every earlier one, so one CTA per
// right-hand side walks the schedule; its 16 warps share each operation with
// coalesced reads of the leaf (warp per Q column / V row, lanes over
// contiguous entries; threads over rows of column-major full and U blocks).
//
// Precision follows the factors' storage: complex FP64 factors (plain
// method) in FP64, complex FP32 factors (mixed method: the preconditioner
// only steers GMRES, the FP64 refinement residual keeps the accuracy) in
// FP32 arithmetic, which is what GB300 runs fast -- its FP64 rate would make
// each 32 x 32 leaf cost ~1 us on one SM. The vectors stay complex FP64.
#include "bem_kernels.h"
#include "hlu_solve.h"
#include "quadrature.cuh"

#include <algorithm>
#include <atomic>
#include <stdexcept>
#include <string>

namespace bemgpu {
namespace {

constexpr int HT = 512;
constexpr int HW = HT / 32;

template <typename T2> struct HC;
template <> struct HC<double2> {
  using R = double;
  static __device__ __forceinline__ double2 ld(const double2* p) { return *p; }
};
template <> struct HC<float2> {
  using R = float;
  static __device__ __forceinline__ float2 ld(const float2* p) { return __ldg(p); }
};

template <typename R>
__device__ __forceinline__ R wsum(R v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// w: right-hand sides (consumed), x: solution, both R x N, complex FP64
template <typename T2>
__global__ void __launch_bounds__(HT) hlu_sweep_kernel(const int32_t* __restrict__ sched,
                                                       int nops, const int64_t* __restrict__ lv,
                                                       const T2* __restrict__ data,
                                                       double2* __restrict__ w,
                                                       double2* __restrict__ x, int64_t N,
                                                       int upper) {
  using R = typename HC<T2>::R;
  __shared__ R tkx[HLU_MAX_RANK], tky[HLU_MAX_RANK];
  __shared__ R xsx[HLU_MAX_LEAF], xsy[HLU_MAX_LEAF];
  __shared__ R px[HW][32], py[HW][32];
  double2* wr = w + (int64_t)blockIdx.x * N;
  double2* xr = x + (int64_t)blockIdx.x * N;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int o = 0; o < nops; o++) {
    const int op = sched[o];
    if (op >= 0) {  // diagonal leaf
      const int64_t* L = lv + 7 * (int64_t)op;
      const int64_t r0 = L[0];
      const int m = (int)L[1];
      const T2* D = data + L[6];
      if (!upper) {  // x_i = (Q^H w)_i = sum_t conj(Q[t, i]) w_t: warp per i, lanes over t
        for (int i = warp; i < m; i += HW) {
          const T2* q = D + (int64_t)i * m;
          R sx = 0, sy = 0;
          for (int t = lane; t < m; t += 32) {
            const T2 a = HC<T2>::ld(q + t);
            const double2 b = wr[r0 + t];
            sx += a.x * (R)b.x + a.y * (R)b.y;
            sy += a.x * (R)b.y - a.y * (R)b.x;
          }
          sx = wsum(sx);
          sy = wsum(sy);
          if (lane == 0) xr[r0 + i] = make_double2((double)sx, (double)sy);
        }
      } else if (warp == 0) {  // R x = w by columns: x_i = w_i / R_ii, then w_t -= R_ti x_i
        for (int i = lane; i < m; i += 32) {
          xsx[i] = (R)wr[r0 + i].x;
          xsy[i] = (R)wr[r0 + i].y;
        }
        __syncwarp();
        for (int i = m - 1; i >= 0; i--) {
          const T2 d = HC<T2>::ld(D + (int64_t)i * m + i);
          // x_i = xs_i / d (all lanes compute the same value)
          const R den = d.x * d.x + d.y * d.y;
          const R ax = xsx[i], ay = xsy[i];
          const R xi = (ax * d.x + ay * d.y) / den, yi = (ay * d.x - ax * d.y) / den;
          __syncwarp();
          const T2* col = D + (int64_t)i * m;
          for (int t = lane; t < i; t += 32) {
            const T2 c = HC<T2>::ld(col + t);
            xsx[t] -= c.x * xi - c.y * yi;
            xsy[t] -= c.x * yi + c.y * xi;
          }
          if (lane == 0) {
            xsx[i] = xi;
            xsy[i] = yi;
          }
          __syncwarp();
        }
        for (int i = lane; i < m; i += 32) xr[r0 + i] = make_double2((double)xsx[i], (double)xsy[i]);
      }
    } else {  // off-diagonal leaf: w_rows -= B x_cols
      const int64_t* L = lv + 7 * (int64_t)(-op - 1);
      const int64_t r0 = L[0], c0 = L[2];
      const int m = (int)L[1], n = (int)L[3], kind = (int)L[4], k = (int)L[5];
      const T2* D = data + L[6];
      if (kind == 0) {
        // full, column-major m x n: 32-row panels; warp w takes columns
        // w, w + 16, ..., lane = row; the 16 partials meet in shared memory
        for (int i0 = 0; i0 < m; i0 += 32) {
          const int i = i0 + lane;
          R sx = 0, sy = 0;
          if (i < m)
            for (int j = warp; j < n; j += HW) {
              const T2 f = HC<T2>::ld(D + (int64_t)j * m + i);
              const double2 xv = xr[c0 + j];
              sx += f.x * (R)xv.x - f.y * (R)xv.y;
              sy += f.x * (R)xv.y + f.y * (R)xv.x;
            }
          px[warp][lane] = sx;
          py[warp][lane] = sy;
          __syncthreads();
          if (warp == 0 && i < m) {
            R ax = 0, ay = 0;
#pragma unroll
            for (int q = 0; q < HW; q++) {
              ax += px[q][lane];
              ay += py[q][lane];
            }
            double2 v = wr[r0 + i];
            v.x -= (double)ax;
            v.y -= (double)ay;
            wr[r0 + i] = v;
          }
          __syncthreads();
        }
      } else {  // low rank: U (m x k col-major), V (k x n row-major)
        const T2* U = D;
        const T2* V = D + (int64_t)m * k;
        for (int l = warp; l < k; l += HW) {
          R sx = 0, sy = 0;
          for (int j = lane; j < n; j += 32) {
            const T2 v = HC<T2>::ld(V + (int64_t)l * n + j);
            const double2 xv = xr[c0 + j];
            sx += v.x * (R)xv.x - v.y * (R)xv.y;
            sy += v.x * (R)xv.y + v.y * (R)xv.x;
          }
          sx = wsum(sx);
          sy = wsum(sy);
          if (lane == 0) {
            tkx[l] = sx;
            tky[l] = sy;
          }
        }
        __syncthreads();
        for (int i = tid; i < m; i += HT) {
          R sx = 0, sy = 0;
          for (int l = 0; l < k; l++) {
            const T2 u = HC<T2>::ld(U + (int64_t)l * m + i);
            sx += u.x * tkx[l] - u.y * tky[l];
            sy += u.x * tky[l] + u.y * tkx[l];
          }
          double2 v = wr[r0 + i];
          v.x -= (double)sx;
          v.y -= (double)sy;
          wr[r0 + i] = v;
        }
      }
    }
    __syncthreads();
  }
}

}  // namespace

int launch_hlu_sweep(const int32_t* sched, int nops, const int64_t* leaves, const void* data,
                     int precision, double2* w, double2* x, int64_t N, int R, int upper,
                     cudaStream_t s) {
  if (nops <= 0 || R <= 0) return 0;
  if (precision == 0)
    hlu_sweep_kernel<double2><<<(unsigned)R, HT, 0, s>>>(sched, nops, leaves, (const double2*)data,
                                                         w, x, N, upper);
  else
    hlu_sweep_kernel<float2><<<(unsigned)R, HT, 0, s>>>(sched, nops, leaves, (const float2*)data,
                                                        w, x, N, upper);
  return 1;
}


// ---------------------------------------------------------------------------
// Dataflow sweep (plan: hlu_solve.h). CTAs claim the items in plan order, level
// by level; every item waits only on items earlier in the order, so each wait
// is on a CTA that is already running: the launch needs no co-residency and any
// number of CTAs works. What an item needs that does not depend on the solve
// (entries of M, U, V) is loaded or prefetched before its wait. Each sum has one
// fixed order: results do not depend on which CTA ran an item or on how many
// there are. Every wait is bounded: after DfArgs::wait_ns the CTA sets the
// sticky error word and returns.
//
// Bound by the latency of a level -- three hand-overs through flags in L2 (x ->
// t -> s -> x, 0.7 us each) and 1.5 to 6 us of work after each (row 4.3, diag 4.5,
// dot 6.8 us with 8 vectors, 2.2, 3.4 and 3.3 us with one) -- times the number of
// levels. At 81,920 pencil elements the chain has 248 levels of ~330 rows instead of
// 3,627 of ~22 (the diagonal leaves), for one more pass over the inverses (N x ~330
// entries): a sweep of 8 vectors takes 3.8 ms, of one 2.1 ms; the 38
// launches of a solve of 8 (14 of them gated off after convergence) 2.4 ms on average,
// over the leaves 14.2 ms. 32, 64 and 120 CTAs beyond the first measured the same.
//
// All arithmetic and every vector inside the sweep is in the factor's type T2:
// complex FP32 for the mixed method, whose FP64 rate on GB300 would otherwise
// bound the sweep; only w is read and x written in complex FP64.
// ---------------------------------------------------------------------------
namespace {

constexpr int NW = HLU_DF_WARPS;
constexpr int DT = 32 * NW;  // threads per CTA
constexpr int MSTEPS = 10;   // entries of M a thread holds across the wait (320 columns)

#define CUDA_OK(x)                                                                     \
  do {                                                                                 \
    const cudaError_t e_ = (x);                                                        \
    if (e_ != cudaSuccess)                                                             \
      throw std::runtime_error(std::string(#x) + ": " + cudaGetErrorString(e_));      \
  } while (0)

template <typename T2> __device__ __forceinline__ T2 mk(typename HC<T2>::R x, typename HC<T2>::R y) {
  T2 t;
  t.x = x;
  t.y = y;
  return t;
}
// s += a b (complex)
template <typename T2> __device__ __forceinline__ void cmac(T2& s, T2 a, T2 b) {
  s.x += a.x * b.x - a.y * b.y;
  s.y += a.x * b.y + a.y * b.x;
}
template <typename T2> __device__ __forceinline__ void cacc(T2& s, T2 a) {
  s.x += a.x;
  s.y += a.y;
}
template <typename T2> __device__ __forceinline__ T2 cshfl(T2 a, int o) {
  return mk<T2>(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o));
}

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void add_release(int* p, int v) {
  asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}
// loads of vectors written during the launch: L2 only (no stale L1 lines)
__device__ __forceinline__ float2 ldv(const float2* p) { return __ldcg(p); }
__device__ __forceinline__ double2 ldv(const double2* p) { return __ldcg(p); }
// the RT values of an index (16-byte pieces for complex FP32)
template <int RT>
__device__ __forceinline__ void ldv_all(const float2* p, float2 (&v)[RT]) {
  if constexpr (RT % 2 == 0) {
#pragma unroll
    for (int r = 0; r < RT; r += 2) {
      const float4 q = __ldcg(reinterpret_cast<const float4*>(p) + r / 2);
      v[r] = make_float2(q.x, q.y);
      v[r + 1] = make_float2(q.z, q.w);
    }
  } else {
#pragma unroll
    for (int r = 0; r < RT; r++) v[r] = __ldcg(p + r);
  }
}
template <int RT>
__device__ __forceinline__ void ldv_all(const double2* p, double2 (&v)[RT]) {
#pragma unroll
  for (int r = 0; r < RT; r++) v[r] = __ldcg(p + r);
}

// thread 0 only: wait until *p >= v; false (and the error word set) after the
// time limit or when another CTA already gave up
__device__ bool df_wait(const int* p, int v, int* err, unsigned long long lim) {
  if (ld_acquire(p) >= v) return true;
  const unsigned long long t0 = gtimer();
  for (unsigned it = 1;; it++) {
    if (ld_acquire(p) >= v) return true;
    if ((it & 63) == 1) {  // after the first failed poll, then every 64
      if (ld_acquire(err)) return false;
      if (gtimer() - t0 > lim) {
        atomicCAS(err, 0, 1);
        return false;
      }
    }
  }
}

struct DfArgs {
  HluDfDev p;
  const void* data;
  const double2* w;  // right-hand sides (complex FP64)
  double2* x;        // result (complex FP64)
  void* xi;          // result in the factor type, RT values per row
  void* s;           // right-hand sides less the earlier supers' contributions
  void* t;
  int* ctrl;  // [0] item counter, then per level the ROW, DIAG and DOT items done
  int* err;
  unsigned long long wait_ns;
  unsigned long long* trace;  // HluDfWork::trace
  int64_t N;
  int R;
  HmvGate gate;
  __device__ int* done(int level, int kind) const { return ctrl + 1 + 3 * level + kind; }
  // thread 0 only: wait for all items of a kind of a level
  __device__ bool wait(int level, int kind) const {
    return df_wait(done(level, kind), p.need[3 * level + kind], err, wait_ns);
  }
};

// an item's results are written: every thread's writes, then the count (the
// barrier orders them before thread 0's release)
__device__ __forceinline__ void df_publish(const DfArgs& a, const HluDfItem& it) {
  __syncthreads();
  if (threadIdx.x == 0) {
    if (a.trace) atomicMax(a.trace + 1 + 3 * it.level + it.type, gtimer());
    add_release(a.done(it.level, it.type), 1);
  }
}

// shared memory: the warps' staged vectors (ROW) or the super's x / s, and the
// warps' partial sums
template <typename T2, int RT>
constexpr size_t df_smem() {
  constexpr size_t stage = (size_t)NW * 32 * RT, vec = (size_t)(HLU_DF_SUPER + 1) * RT;
  return ((stage > vec ? stage : vec) + (size_t)NW * 32 * RT) * sizeof(T2);
}

// n indices of a vector (RT values each) into shared memory, all threads
template <typename T2, int RT>
__device__ __forceinline__ void load_vectors(T2* dst, const T2* src, int n) {
  if constexpr (sizeof(T2) == 8 && RT % 2 == 0) {
    for (int e = threadIdx.x; e < n * RT / 2; e += DT)
      reinterpret_cast<float4*>(dst)[e] = __ldcg(reinterpret_cast<const float4*>(src) + e);
  } else {
    for (int e = threadIdx.x; e < n * RT; e += DT) dst[e] = ldv(src + e);
  }
}

// ROW: s(chunk) = w - sum over its columns of entry * t or x. Warps share the
// columns evenly, lanes are rows. The first UP entries of a lane are loaded
// before the wait, the vectors of 32 columns at once after it.
template <typename T2, int RT>
__device__ bool df_row_item(const DfArgs& a, const HluDfItem& it, T2* sm) {
  constexpr int UP = sizeof(T2) == 8 ? 16 : 8;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  T2* stage = sm + warp * 32 * RT;
  T2* part = sm + NW * 32 * RT;  // [warp][r][row]
  const T2* data = (const T2*)a.data;
  const int row = lane < it.m ? lane : 0;
  const int64_t ncol = it.end - it.beg;
  const int c0 = it.beg + (int)(ncol * warp / NW), c1 = it.beg + (int)(ncol * (warp + 1) / NW);
  HluDfColumn col{0, 0, 0};
  T2 u[UP];
  const auto load_u = [&](int i0, int nb) {
#pragma unroll
    for (int q = 0; q < UP; q++) {
      const int64_t off = __shfl_sync(0xffffffffu, col.off, (i0 + q) & 31);
      u[q] = i0 + q < nb ? HC<T2>::ld(data + off + row) : mk<T2>(0, 0);
    }
  };
  const auto load_cols = [&](int c) {
    const int4 v = __ldg(reinterpret_cast<const int4*>(a.p.columns + min(c + lane, c1 - 1)));
    col.off = (int64_t)(uint32_t)v.x | ((int64_t)v.y << 32);
    col.vec = v.z;
  };
  if (c0 < c1) {
    load_cols(c0);
    load_u(0, min(32, c1 - c0));
  }
  // w of the thread's output (row, r), in flight during the wait
  const int orow = tid & 31, orr = tid >> 5;
  double2 wv = make_double2(0.0, 0.0);
  if (orr < a.R && orow < it.m) wv = __ldcg(a.w + (int64_t)orr * a.N + it.r0 + orow);
  if (it.level > 0) {
    bool ok = true;
    if (tid == 0) ok = a.wait(it.level - 1, HLU_DF_DOT);
    if (!__syncthreads_and(ok)) return false;
  }
  T2 acc[RT];
#pragma unroll
  for (int r = 0; r < RT; r++) acc[r] = mk<T2>(0, 0);
  for (int c = c0; c < c1; c += 32) {
    const int nb = min(32, c1 - c);
    if (c > c0) load_cols(c);
    {
      T2 v[RT];
      const T2* src = col.vec >= 0 ? (const T2*)a.t + (int64_t)col.vec * RT
                                   : (const T2*)a.xi + (int64_t)(-1 - col.vec) * RT;
      ldv_all<RT>(src, v);
      __syncwarp();
#pragma unroll
      for (int r = 0; r < RT; r++) stage[lane * RT + r] = v[r];
      __syncwarp();
    }
    for (int i0 = 0; i0 < nb; i0 += UP) {
      if (c > c0 || i0 > 0) load_u(i0, nb);
#pragma unroll
      for (int q = 0; q < UP; q += 2) {  // mostly 5 to 20 columns: stop at the last
        if (i0 + q >= nb) break;
#pragma unroll
        for (int r = 0; r < RT; r++) cmac(acc[r], u[q], stage[(i0 + q) * RT + r]);
#pragma unroll
        for (int r = 0; r < RT; r++) cmac(acc[r], u[q + 1], stage[((i0 + q + 1) & 31) * RT + r]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < RT; r++) part[(warp * RT + r) * 32 + lane] = acc[r];
  __syncthreads();
  if (orr < RT && orow < it.m) {
    T2 v = mk<T2>((typename HC<T2>::R)wv.x, (typename HC<T2>::R)wv.y);
    T2 sum[NW];  // pairwise
#pragma unroll
    for (int q = 0; q < NW; q++) sum[q] = part[(q * RT + orr) * 32 + orow];
#pragma unroll
    for (int n = NW / 2; n >= 1; n /= 2)
#pragma unroll
      for (int q = 0; q < n; q++) cacc(sum[q], sum[q + n]);
    v.x -= sum[0].x;
    v.y -= sum[0].y;
    ((T2*)a.s)[(int64_t)(it.r0 + orow) * RT + orr] = v;
  }
  df_publish(a, it);
  return true;
}

// hi + lo += v, the rounding error of hi + v kept in lo (Knuth's TwoSum)
template <typename R>
__device__ __forceinline__ void two_sum(R& hi, R& lo, R v) {
  const R s = hi + v, b = s - hi;
  lo += (hi - (s - b)) + (v - b);
  hi = s;
}

// The sum of the 32 partial sums of a row of M s: compensated in FP32, pairwise in
// FP64, whose pipe has no room for the compensation. A row of an inverse has
// hundreds of columns where a leaf has some 22, and with these sums in order the
// sweeps were further from the exact solve than leaf by leaf: 8 FP32 vectors,
// sphere of 1,280 elements 1.47e-7 (leaf by leaf 1.33e-7, now 1.14e-7), pencil of
// 20,480 1.35e-7 (1.28e-7, 1.09e-7). FP64, sphere of 1,280: 2.54e-16 (2.39e-16,
// 2.33e-16). Cost at 20,480 elements and 8 vectors: 2.01 -> 2.05 ms.
template <typename T2>
struct Joined {  // FP64
  T2 hi;
  __device__ __forceinline__ void join(const T2 (&p)[8]) {
    T2 a = p[0], b = p[2], c = p[4], d = p[6];
    cacc(a, p[1]);
    cacc(b, p[3]);
    cacc(c, p[5]);
    cacc(d, p[7]);
    cacc(a, b);
    cacc(c, d);
    cacc(a, c);
    hi = a;
  }
  __device__ __forceinline__ void store(T2* s, int i, int) const { s[i] = hi; }
  // this thread's sum and those of i + n, i + 2 n, i + 3 n
  __device__ __forceinline__ T2 join_stored(const T2* s, int i, int n) const {
    T2 a = hi, b = s[2 * n + i];
    cacc(a, s[n + i]);
    cacc(b, s[3 * n + i]);
    cacc(a, b);
    return a;
  }
};
template <>
struct Joined<float2> {
  float2 hi, lo;
  __device__ __forceinline__ void add(float2 v) {
    two_sum(hi.x, lo.x, v.x);
    two_sum(hi.y, lo.y, v.y);
  }
  __device__ __forceinline__ void join(const float2 (&p)[8]) {
    hi = p[0];
    lo = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int q = 1; q < 8; q++) add(p[q]);
  }
  __device__ __forceinline__ void store(float2* s, int i, int n) const {
    s[i] = hi;
    s[n + i] = lo;
  }
  __device__ __forceinline__ float2 join_stored(const float2* s, int i, int n) {
#pragma unroll
    for (int q = 1; q < 4; q++) add(s[q * n + i]);
#pragma unroll
    for (int q = 1; q < 4; q++) cacc(lo, s[(4 + q) * n + i]);
    return make_float2(hi.x + lo.x, hi.y + lo.y);
  }
};

// DIAG: 16 rows of x = M s. Lanes are 16 rows x 2 columns, warp w takes the
// columns c0 + 2 w + (0, 1), then every 32nd; the entries of M are held in
// registers across the wait.
template <typename T2, int RT>
__device__ bool df_diag_item(const DfArgs& a, const HluDfItem& it, T2* sm) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  T2* sv = sm;  // [column][r]
  T2* part = sm + (NW * 32 > HLU_DF_SUPER + 1 ? NW * 32 : HLU_DF_SUPER + 1) * RT;  // [2 NW][16][r]
  const int row = it.t0 + (lane & 15), nrow = min(HLU_DF_TILE, it.m - it.t0);
  const int cb = it.c0 + 2 * warp + (lane >> 4);
  const T2* M = (const T2*)a.p.minv + it.moff + min(row, it.m - 1);
  T2 u[MSTEPS];
#pragma unroll
  for (int q = 0; q < MSTEPS; q++) {
    const int c = cb + 32 * q;
    u[q] = c < it.c1 ? HC<T2>::ld(M + (int64_t)c * it.m) : mk<T2>(0, 0);
  }
  bool ok = true;
  if (tid == 0) ok = a.wait(it.level, HLU_DF_ROW);
  if (!__syncthreads_and(ok)) return false;
  load_vectors<T2, RT>(sv + it.c0 * RT, (const T2*)a.s + ((int64_t)it.r0 + it.c0) * RT,
                       it.c1 - it.c0);
  __syncthreads();
  T2 acc[RT];
#pragma unroll
  for (int r = 0; r < RT; r++) acc[r] = mk<T2>(0, 0);
#pragma unroll
  for (int q = 0; q < MSTEPS; q++) {
    const int c = cb + 32 * q;
    if (it.c0 + 2 * warp + 32 * q >= it.c1) break;
    const T2* v = sv + (c < it.c1 ? c : it.c1 - 1) * RT;  // u = 0 past the end
#pragma unroll
    for (int r = 0; r < RT; r++) cmac(acc[r], u[q], v[r]);
  }
  for (int c = cb + 32 * MSTEPS; c < it.c1; c += 32) {
    const T2 v = HC<T2>::ld(M + (int64_t)c * it.m);
#pragma unroll
    for (int r = 0; r < RT; r++) cmac(acc[r], v, sv[c * RT + r]);
  }
  // partial sums [2 warp + half][r][row]; four threads per output add 8 of the
  // 32 each, then one the four
  T2* pw = part + (2 * warp + (lane >> 4)) * 16 * RT + (lane & 15);
#pragma unroll
  for (int r = 0; r < RT; r++) pw[r * 16] = acc[r];
  __syncthreads();
  constexpr int NO = 16 * RT;
  Joined<T2> j;
  if (tid < 4 * NO) {
    const T2* pp = part + (tid / NO) * (2 * NW / 4) * NO + tid % NO;
    T2 p[2 * NW / 4];
#pragma unroll
    for (int q = 0; q < 2 * NW / 4; q++) p[q] = pp[q * NO];
    j.join(p);
    j.store(sv, tid, 4 * NO);  // s is no longer read
  }
  __syncthreads();
  if (tid < NO) {
    const T2 v = j.join_stored(sv, tid, NO);
    const int orow = tid & 15, r = tid >> 4;
    if (orow < nrow) {
      const int64_t g = (int64_t)it.r0 + it.t0 + orow;
      ((T2*)a.xi)[g * RT + r] = v;
      if (r < a.R) a.x[r * a.N + g] = make_double2((double)v.x, (double)v.y);
    }
  }
  df_publish(a, it);
  return true;
}

// DOT: one warp per dot, two rows of V at a time over the super's columns; the
// 2 RT sums over the lanes by halving exchange
template <typename T2, int N, int M>
__device__ __forceinline__ int df_halve(T2 (&acc)[N], int lane, bool& mine) {
  if constexpr (M == 0) {
    return 0;
  } else if constexpr (N % 2 == 0) {
    const bool up = lane & M;
    T2 half[N / 2];
#pragma unroll
    for (int i = 0; i < N / 2; i++) {
      const T2 send = up ? acc[i] : acc[i + N / 2];
      const T2 got = cshfl(send, M);
      half[i] = up ? acc[i + N / 2] : acc[i];
      cacc(half[i], got);
    }
    const int o = df_halve<T2, N / 2, M / 2>(half, lane, mine) + (up ? N / 2 : 0);
#pragma unroll
    for (int i = 0; i < N / 2; i++) acc[i] = half[i];
    return o;
  } else {
#pragma unroll
    for (int i = 0; i < N; i++) cacc(acc[i], cshfl(acc[i], M));
    if (lane & M) mine = false;
    return df_halve<T2, N, M / 2>(acc, lane, mine);
  }
}

// index of the value a lane ends with (one value: N a power of two <= 2 M)
template <int N, int M>
__device__ __forceinline__ int df_kept(int lane) {
  if constexpr (M == 0 || N == 1) return 0;
  else return df_kept<N / 2, M / 2>(lane) + (lane & M ? N / 2 : 0);
}

template <typename T2, int RT>
__device__ bool df_dot_item(const DfArgs& a, const HluDfItem& it, T2* sm) {
  constexpr int VP = 4;  // column steps loaded before the wait
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int e = it.beg + warp;
  const bool has = e < it.end;
  HluDfDot d{};
  const T2 *v0 = nullptr, *v1 = nullptr;
  T2 p0[VP], p1[VP];
  if (has) {
    const int4 q0 = __ldg(reinterpret_cast<const int4*>(a.p.dots + e));
    const int4 q1 = __ldg(reinterpret_cast<const int4*>(a.p.dots + e) + 1);
    d.off = (int64_t)(uint32_t)q0.x | ((int64_t)q0.y << 32);
    d.ld = q0.z;
    d.rows = q0.w;
    d.w = q1.x;
    d.xo = q1.y;
    d.t = q1.z;
    d.first = q1.w;
    v0 = (const T2*)a.data + d.off;
    v1 = v0 + (d.rows > 1 ? d.ld : 0);
#pragma unroll
    for (int q = 0; q < VP; q++) {
      const int c = lane + 32 * q;
      p0[q] = c < d.w ? HC<T2>::ld(v0 + c) : mk<T2>(0, 0);
      p1[q] = c < d.w ? HC<T2>::ld(v1 + c) : mk<T2>(0, 0);
    }
    for (int c = lane + 32 * VP; c < d.w; c += 32) {
      prefetch_l2(v0 + c);
      prefetch_l2(v1 + c);
    }
  }
  bool ok = true;
  if (tid == 0) {
    ok = a.wait(it.level, HLU_DF_DIAG);
    if (ok && it.level > 0) ok = a.wait(it.level - 1, HLU_DF_DOT);
  }
  if (!__syncthreads_and(ok)) return false;
  // the old value of the sum this lane may end with (index below: the halving
  // exchange leaves value o of the 2 RT to one or more lanes)
  T2* const tp = (T2*)a.t + (int64_t)d.t * RT;
  const int ob = df_kept<2 * RT, 16>(lane);
  T2 old = mk<T2>(0, 0);
  if (has && !d.first && ob < d.rows * RT) old = ldv(tp + ob);
  const int ldx = HLU_DF_SUPER + 1;  // x of the super, [r][column]
  const T2* xg = (const T2*)a.xi + (int64_t)it.r0 * RT;
  for (int q = tid; q < it.m * RT; q += DT) sm[(q % RT) * ldx + q / RT] = ldv(xg + q);
  __syncthreads();
  if (has) {
    T2 acc[2 * RT];
#pragma unroll
    for (int r = 0; r < 2 * RT; r++) acc[r] = mk<T2>(0, 0);
    const T2* xs = sm + d.xo;
#pragma unroll
    for (int q = 0; q < VP; q++) {
      if (32 * q >= d.w) break;
      const int c = min(lane + 32 * q, d.w - 1);  // V = 0 past the end
#pragma unroll
      for (int r = 0; r < RT; r++) {
        const T2 xv = xs[r * ldx + c];
        cmac(acc[r], p0[q], xv);
        cmac(acc[RT + r], p1[q], xv);
      }
    }
    for (int c = lane + 32 * VP; c < d.w; c += 32) {
      const T2 a0 = HC<T2>::ld(v0 + c), a1 = HC<T2>::ld(v1 + c);
#pragma unroll
      for (int r = 0; r < RT; r++) {
        const T2 xv = xs[r * ldx + c];
        cmac(acc[r], a0, xv);
        cmac(acc[RT + r], a1, xv);
      }
    }
    bool mine = true;
    const int o = df_halve<T2, 2 * RT, 16>(acc, lane, mine);  // one value each (2 RT <= 32)
    if (mine && o < d.rows * RT) {
      T2 v = acc[0];
      cacc(v, old);
      tp[o] = v;
    }
  }
  df_publish(a, it);
  return true;
}

template <typename T2, int RT>
__global__ void __launch_bounds__(DT, 1) hlu_df_kernel(DfArgs a) {
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ int sq;
  T2* sm = (T2*)raw;
  if (gate_closed(a.gate)) return;  // every CTA reads the same flags
  while (true) {
    __syncthreads();
    if (threadIdx.x == 0) {
      sq = atomicAdd(a.ctrl, 1);
      if (a.trace && sq == 0) a.trace[0] = gtimer();
    }
    __syncthreads();
    const int q = sq;
    if (q >= a.p.nitems) return;
    const HluDfItem it = a.p.items[q];
    bool ok;
    if (it.type == HLU_DF_ROW) ok = df_row_item<T2, RT>(a, it, sm);
    else if (it.type == HLU_DF_DIAG) ok = df_diag_item<T2, RT>(a, it, sm);
    else ok = df_dot_item<T2, RT>(a, it, sm);
    if (!ok) return;
  }
}

// ---- inverses of the supers' diagonal blocks ----

// one CTA per leaf inside a diagonal block: its entries into the dense copy, which
// starts at value d0 of all the dense blocks
template <typename T2>
__global__ void __launch_bounds__(128) df_expand_kernel(const HluDfInner* __restrict__ inner,
                                                        const T2* __restrict__ data,
                                                        T2* __restrict__ dense, int64_t d0) {
  const HluDfInner in = inner[blockIdx.x];
  const T2* D = data + in.off;
  for (int e = threadIdx.x; e < in.m * in.n; e += 128) {
    const int r = e / in.n, c = e % in.n;
    T2 v = mk<T2>(0, 0);
    if (in.lowrank) {
      const T2* V = D + (int64_t)in.m * in.k;
      for (int l = 0; l < in.k; l++)
        cmac(v, D[(int64_t)l * in.m + r], V[(int64_t)l * in.n + c]);
    } else {
      v = D[(int64_t)c * in.m + r];
    }
    dense[in.dst - d0 + (int64_t)r * in.ld + c] = v;
  }
}

// One CTA per PW columns of a super's inverse: block substitution of the unit
// vectors, the panel in shared memory, lanes over its columns, warps over the
// rows of a chunk; the dense block's entries are read as broadcasts.
constexpr int IT = 256;
// Columns of a plain sum; sums of sums are compensated. A thread's one sum over all
// columns before (up to 480) made the inverse a little worse than its storage.
constexpr int KB = 8;
template <typename T2, int PW>
__global__ void __launch_bounds__(IT) df_invert_kernel(HluDfDev p, int panel_beg,
                                                       const T2* __restrict__ dense, int64_t d0) {
  extern __shared__ __align__(16) unsigned char raw[];
  constexpr int LD = PW + 1, SUB = 32 / PW, RSTEP = (IT / 32) * SUB;
  constexpr int RT = (HLU_DF_MAX_M + RSTEP - 1) / RSTEP;
  const HluDfPanel pn = p.panels[panel_beg + blockIdx.x];
  const HluDfSuper su = p.supers[pn.super];
  const int m = su.m, w = min(PW, m - pn.p0);
  T2* X = (T2*)raw;  // [row][column]
  T2* tmp = X + (int64_t)m * LD;
  const T2* D = dense + (su.moff - d0);
  const int tid = threadIdx.x, lane = tid & 31, c = lane % PW;
  const int rs = (tid >> 5) * SUB + lane / PW;  // the thread's first row of a chunk
  for (int e = tid; e < m * LD; e += IT) X[e] = mk<T2>(0, 0);
  __syncthreads();
  int first = -1, f0 = 0, f1 = 0;  // rows of the panel's first chunk in solve order
  for (int q = su.chunk_beg; q < su.chunk_end; q++) {
    const HluDfChunk ch = p.chunks[q];
    const int a = ch.r0, b = ch.r0 + ch.m;
    if (first < 0) {
      if (p.lower ? b <= pn.p0 : a >= pn.p0 + w) continue;
      first = q;
      f0 = a;
      f1 = b;
    }
    // rows already solved: [f0, a) going down, [b, f1) going up
    const int k0 = p.lower ? f0 : b, k1 = p.lower ? a : f1;
    T2 acc[RT], low[RT];
#pragma unroll
    for (int t = 0; t < RT; t++) acc[t] = low[t] = mk<T2>(0, 0);
    const T2* row[RT];
#pragma unroll
    for (int t = 0; t < RT; t++) row[t] = D + (int64_t)min(a + rs + t * RSTEP, b - 1) * m;
    for (int k = k0; k < k1; k += KB) {
      T2 part[RT];
#pragma unroll
      for (int t = 0; t < RT; t++) part[t] = mk<T2>(0, 0);
      const int ke = min(k + KB, k1);
#pragma unroll 4
      for (int q = k; q < ke; q++) {
        const T2 xv = X[q * LD + c];
#pragma unroll
        for (int t = 0; t < RT; t++) cmac(part[t], HC<T2>::ld(row[t] + q), xv);
      }
#pragma unroll
      for (int t = 0; t < RT; t++) {
        two_sum(acc[t].x, low[t].x, part[t].x);
        two_sum(acc[t].y, low[t].y, part[t].y);
      }
    }
#pragma unroll
    for (int t = 0; t < RT; t++) {
      const int r = rs + t * RSTEP;
      if (r < ch.m)
        tmp[r * LD + c] = mk<T2>(((a + r == pn.p0 + c ? 1 : 0) - acc[t].x) - low[t].x,
                                 -(acc[t].y + low[t].y));
    }
    __syncthreads();
    const T2* A = (const T2*)p.diag + ch.aoff;
#pragma unroll
    for (int t = 0; t < RT; t++) {
      const int r = rs + t * RSTEP;
      if (r < ch.m) {
        T2 v[4];  // by quarters of the terms
#pragma unroll
        for (int e = 0; e < 4; e++) v[e] = mk<T2>(0, 0);
        for (int k = 0; k < ch.m; k += 4)
#pragma unroll
          for (int e = 0; e < 4; e++)
            if (k + e < ch.m) cmac(v[e], HC<T2>::ld(A + r * ch.m + k + e), tmp[(k + e) * LD + c]);
        cacc(v[0], v[1]);
        cacc(v[2], v[3]);
        cacc(v[0], v[2]);
        X[(a + r) * LD + c] = v[0];
      }
    }
    __syncthreads();
  }
  T2* M = (T2*)p.minv + su.moff;
  for (int e = tid; e < m * w; e += IT) {
    const int cc = e / m, r = e % m;
    M[(int64_t)(pn.p0 + cc) * m + r] = X[r * LD + cc];
  }
}

// Above 48 KiB a kernel's shared memory has to be asked for, once per device. The
// limit is the kernel's, not a handle's or a stream's, so `most` is what any launch
// of it can need: a smaller value would fail another thread's launch.
template <typename K>
void allow_smem(K* kernel, size_t most, std::atomic<uint64_t>& ready) {
  int dev = 0;
  CUDA_OK(cudaGetDevice(&dev));
  const uint64_t bit = 1ull << (dev & 63);
  if (dev >= 64 || !(ready.load() & bit)) {
    CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    ready |= bit;
  }
}

template <typename T2, int RT>
void df_launch(const DfArgs& a, int grid, cudaStream_t s) {
  static std::atomic<uint64_t> ready{0};
  allow_smem(hlu_df_kernel<T2, RT>, df_smem<T2, RT>(), ready);
  hlu_df_kernel<T2, RT><<<grid, DT, df_smem<T2, RT>(), s>>>(a);
}

template <typename T2>
void df_launch_r(const DfArgs& a, int grid, cudaStream_t s) {
  if (a.R == 1) df_launch<T2, 1>(a, grid, s);
  else if (a.R == 2) df_launch<T2, 2>(a, grid, s);
  else if (a.R <= 4) df_launch<T2, 4>(a, grid, s);
  else df_launch<T2, 8>(a, grid, s);
}

// shared memory of the inversion of blocks of up to m rows
template <typename T2, int PW>
constexpr size_t df_invert_smem(int m) {
  return (size_t)(m + HLU_DF_MAX_M) * (PW + 1) * sizeof(T2);
}

template <typename T2, int PW>
int df_invert(const HluDfDev& p, const HluDfBatch& b, const void* data, void* dense,
              cudaStream_t s) {
  static std::atomic<uint64_t> ready{0};
  allow_smem(df_invert_kernel<T2, PW>, df_invert_smem<T2, PW>(HLU_DF_SUPER), ready);
  // blocks without a leaf (rank 0) are zero, whatever the buffer held before
  CUDA_OK(cudaMemsetAsync(dense, 0, (size_t)b.size * sizeof(T2), s));
  if (b.ninner > 0)
    df_expand_kernel<T2><<<(unsigned)b.ninner, 128, 0, s>>>(p.inner + b.inner_beg, (const T2*)data,
                                                            (T2*)dense, b.moff);
  df_invert_kernel<T2, PW><<<(unsigned)b.npanels, IT, df_invert_smem<T2, PW>(p.maxm), s>>>(
      p, b.panel_beg, (const T2*)dense, b.moff);
  return 1 + (b.ninner > 0);
}

}  // namespace

int launch_hlu_df_invert(const HluDfDev& p, const HluDfBatch& b, const void* data, int precision,
                         void* dense, cudaStream_t s) {
  if (b.npanels <= 0) return 0;
  return precision == 0 ? df_invert<double2, HLU_DF_PANEL>(p, b, data, dense, s)
                        : df_invert<float2, HLU_DF_PANEL>(p, b, data, dense, s);
}

int launch_hlu_df(const HluDfDev& p, const void* data, int precision, const double2* w, double2* x,
                  int64_t N, int R, const HluDfWork& ws, int helpers, cudaStream_t s,
                  HmvGate gate) {
  if (p.D <= 0 || R <= 0) return 0;
  if (R > HLU_DF_MAX_R) throw std::runtime_error("launch_hlu_df: more than 8 right-hand sides");
  CUDA_OK(cudaMemsetAsync(ws.ctrl, 0, (size_t)(1 + 3 * p.D) * sizeof(int), s));
  DfArgs a;
  a.p = p;
  a.data = data;
  a.w = w;
  a.x = x;
  a.xi = ws.xi;
  a.s = ws.s;
  a.t = ws.t;
  a.ctrl = ws.ctrl;
  a.err = ws.err;
  a.N = N;
  a.R = R;
  a.gate = gate;
  a.wait_ns = ws.wait_ns;
  a.trace = ws.trace;
  const int grid = std::min(1 + std::max(1, helpers), p.nitems);
  if (precision == 0) df_launch_r<double2>(a, grid, s);
  else df_launch_r<float2>(a, grid, s);
  return 2;
}

}  // namespace bemgpu
