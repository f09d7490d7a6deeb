// hlu_solve.h -- launch interface of the H-LU block-triangular solve kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "bem_kernels.h"

namespace bemgpu {

constexpr int HLU_MAX_RANK = 512;  // largest low-rank leaf of a factor
constexpr int HLU_MAX_LEAF = 512;  // largest diagonal leaf (leaf_size - 1)

// One sweep over a flattened factor: upper = 0 applies L^{-1} (y = Q^H w on
// diagonal leaves), upper = 1 applies U^{-1}. data holds the factor in complex
// FP64 (precision 0) or complex FP32 (precision 1, FP32 arithmetic). w (R x N,
// complex FP64) is consumed, x gets the result. Returns the kernels launched.
int launch_hlu_sweep(const int32_t* sched, int nops, const int64_t* leaves, const void* data,
                     int precision, double2* w, double2* x, int64_t N, int R, int upper,
                     cudaStream_t s);

// ---- dataflow form of the same sweep ----
//
// The rows are cut at cluster-tree nodes of at most HLU_DF_SUPER rows
// ("supers", numbered in solve order: increasing rows for L, decreasing for U).
// The diagonal block of a super is inverted once per factorization (dense), so
// a sweep is a chain of N / ~320 steps instead of one per diagonal leaf:
//   ROW(I): s = w - (leaves over rows of super I, columns in earlier supers),
//           one item per diagonal leaf ("chunk"); a full leaf reads x, a
//           low-rank one its t = V x;
//   DIAG(I): x = M s, M the inverse of super I's diagonal block, one item per
//           16 rows;
//   DOT(I): t of the low-rank leaves whose columns meet super I gains V x.
// Items of a level wait for those of the previous kind, and DOT(I) for
// DOT(I - 1), so t is summed in column order.
constexpr int HLU_DF_SUPER = 512;    // most rows of a super
// Most rows of a super in each precision: longer ones make the chain shorter, but the
// inversion is cubic in their rows. FP32, 81,920 pencil elements: a sweep of 8 (1)
// vectors 3.8 (2.1) ms with 512 rows, 5.9 (3.5) with 256, 8.0 (4.9) with 128, the
// inversions 4.3 / 1.8 / 0.7 ms, against 38 sweeps of a solve; beyond 512 a panel
// and the x of a super no longer fit. In complex FP64 the FP64 pipe bounds the
// inversion: 1,280 sphere elements, 1.2 ms and 0.19 ms a sweep with 256 rows, 3.1 and
// 0.11 with 512, 0.4 and 0.34 with 128, against 6 sweeps of a solve.
constexpr int hlu_df_super(int precision) { return precision == 0 ? 256 : HLU_DF_SUPER; }
constexpr int HLU_DF_MAX_M = 32;     // rows of a diagonal leaf
constexpr int HLU_DF_MAX_RANK = 32;  // rank of a low-rank leaf
constexpr int HLU_DF_MAX_R = 8;      // right-hand sides per launch
constexpr int HLU_DF_TILE = 16;      // rows of a DIAG item
constexpr int HLU_DF_WARPS = 16;     // warps of a sweep CTA; dots of a DOT item

enum { HLU_DF_ROW = 0, HLU_DF_DIAG = 1, HLU_DF_DOT = 2 };

// one item of the sweep
struct HluDfItem {
  int32_t type, level;  // level: the super
  int32_t beg, end;     // ROW: columns, DOT: dots
  int32_t r0, m;        // ROW: first row and rows of the chunk; else those of the super
  int32_t c0, c1;       // DIAG: columns of M that its rows use
  int64_t moff;         // DIAG: offset of M (column-major m x m)
  int32_t t0, pad;      // DIAG: first row of the tile inside the super
};
// a column over a chunk's rows: entries at off (of the chunk's first row), times
// t[vec] (vec >= 0) or x[-1 - vec]
struct HluDfColumn {
  int64_t off;
  int32_t vec, pad;
};
// t[t + q] (+)= V[q, 0 .. w) x[first row of the super + xo ..), q < rows <= 2; V at
// off, row stride ld; first: t is set instead of added to
struct HluDfDot {
  int64_t off;
  int32_t ld, rows, w, xo, t, first;
};
// a leaf inside a super's diagonal block, into the dense copy of that block
struct HluDfInner {
  int64_t off, dst;  // leaf data; first entry in the dense blocks (row-major, row stride ld)
  int32_t lowrank, m, n, k, ld, pad;
};
struct HluDfChunk {  // diagonal leaf, in solve order
  int32_t r0, m;     // rows, from the super's first row
  int64_t aoff;      // its m x m apply matrix (row-major): Q^H or R^{-1}
};
struct HluDfSuper {
  int32_t r0, m, chunk_beg, chunk_end;
  int64_t moff;  // offset of M and of the dense block
};
struct HluDfPanel {  // columns p0 .. of super's inverse (one CTA of the inversion)
  int32_t super, p0;
};
// Columns per inversion CTA (their panel stays in shared memory). Both factors of
// 81,920 pencil elements in FP32: 4.3 ms, 16 columns 5.0, 32 columns 10.3 (one CTA
// per SM); of 5,120 in FP64 2.8 ms, 4 columns 3.9, 16 columns 5.1.
constexpr int HLU_DF_PANEL = 8;

// device copy of one factor's plan
struct HluDfDev {
  const HluDfItem* items = nullptr;
  const HluDfColumn* columns = nullptr;
  const HluDfDot* dots = nullptr;
  const HluDfInner* inner = nullptr;
  const HluDfChunk* chunks = nullptr;
  const HluDfSuper* supers = nullptr;
  const HluDfPanel* panels = nullptr;
  const int32_t* need = nullptr;  // items per level: ROW, DIAG, DOT (3 D)
  const void* diag = nullptr;     // apply matrices of the chunks, factor precision
  void* minv = nullptr;           // inverses of the supers' diagonal blocks
  int64_t nt = 0;                 // values of t
  int64_t msize = 0;              // values of minv
  int nitems = 0, D = 0, lower = 0;
  int maxm = 0;                   // rows of the largest super
};

// Workspace shared by the sweeps of one handle, vectors in the factor type with
// the right-hand sides of an index together: xi and s (N x HLU_DF_MAX_R), t (nt
// x HLU_DF_MAX_R); ctrl (1 + 3 D ints, cleared by every launch), err (sticky
// error word: nonzero after a wait ran out of time).
struct HluDfWork {
  void* xi = nullptr;
  void* s = nullptr;
  void* t = nullptr;
  int* ctrl = nullptr;
  int* err = nullptr;
  // bound of one wait (ns): an item may wait for others whose CTAs share their
  // SMs with other streams' kernels
  unsigned long long wait_ns = 10000000000ull;
  // optional (profiling), 1 + 3 D values cleared by the caller: start of the sweep and
  // end of the last ROW, DIAG and DOT item of every level (ns)
  unsigned long long* trace = nullptr;
};

// A run of consecutive supers that are inverted together: their leaves and panels,
// and the range of their dense blocks (and inverses) among all of them.
struct HluDfBatch {
  int32_t inner_beg = 0, ninner = 0, panel_beg = 0, npanels = 0;
  int64_t moff = 0, size = 0;
};
// Values of the dense copies that are inverted at a time: the copies are scratch of
// every handle, so they are not all made at once (64 MiB in complex FP32; at 81,920
// pencil elements all of them would take 210 MB).
constexpr int64_t HLU_DF_BATCH = 8 << 20;

// Inverses of the diagonal blocks of a batch of supers from the factor's leaves
// (data) and apply matrices; dense: b.size values of scratch, cleared here. Returns
// the kernels launched.
int launch_hlu_df_invert(const HluDfDev& p, const HluDfBatch& b, const void* data, int precision,
                         void* dense, cudaStream_t s);

// w (R x N) -> x (R x N) with one launch of 1 + `helpers` CTAs (R <=
// HLU_DF_MAX_R; w is only read). Returns the kernels launched.
// gate: optional early exit (bem_kernels.h HmvGate; all its flags set -> no work)
int launch_hlu_df(const HluDfDev& p, const void* data, int precision, const double2* w, double2* x,
                  int64_t N, int R, const HluDfWork& ws, int helpers, cudaStream_t s,
                  HmvGate gate = HmvGate{nullptr, 0, 0});

}  // namespace bemgpu
