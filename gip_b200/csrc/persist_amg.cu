// Whole preconditioned solves as one launch: the mixed form's FP32 CG (with the AMG V-cycle
// or GIP's Jacobi) and the FP64 tolerance mode with AMG.
//
// Kernel by kernel an iteration with AMG is a chain of a dozen or more dependent launches,
// most of them on a few thousand unknowns: on the 63^3 cavity 13 kernels of 4 to 12 us, 75 us
// an iteration, for work that fits the L2 many times over.  Here the CTAs stay resident and
// every kernel boundary is a barrier, over a cluster of up to 16 CTAs or over a cooperative
// grid.  Every row of every product is summed in the order of the kernel it replaces (pcg.cu,
// amg.cu), so vectors are the same bit for bit given the same scalars; only the dots' partial
// sums are added in another order.  Vectors written inside the launch are read with plain
// loads (never through the read-only path), after a barrier that every thread of the CTA has
// passed.
//
// A phase is bound by latency: what it reads that does not change (operator words, columns,
// values) is loaded between its barrier's arrival and its wait, and a row's own operands
// with its gathers, so that a phase costs one dependent round trip to the L2 and its sums.
//
// Every CTA owns a contiguous range of each operator's rows, the same one in every phase on
// that operator: what a thread writes for its own level-0 rows needs no barrier, and an
// operator of a few hundred slices still occupies every SM.
// The search direction is never stored on its own: pair[i] = (z_i, p_i) holds the
// preconditioned residual and the previous direction, and p = z + beta p is formed where it
// is gathered (one 8- or 16-byte gather per nonzero).
#include <algorithm>
#include <cstdlib>
#include <type_traits>
#include <vector>

#include "persist.cuh"

namespace gipb200 {
namespace {

constexpr int kThreads = 512;  // 128 registers a thread
constexpr int kMaxOps = 40;  // products of a cycle below level 0's own two

// The CTAs of one solve: barriers and sums over them, and this CTA's share of their work.
struct GridTeam {
  GridScope G;
  __device__ __forceinline__ int rank() const { return G.rank; }
  __device__ __forceinline__ int ncta() const { return G.ncta; }
  __device__ __forceinline__ void arrive() { grid_arrive(G); }
  __device__ __forceinline__ bool wait() { return grid_wait(G); }
  template <int W, bool FENCE>
  __device__ __forceinline__ bool sum(double (&v)[W]) {
    return grid_sum<W, FENCE>(v, G);
  }
};

struct ClusterTeam {
  static constexpr int kMaxCtas = 16;
  double (*red)[kGridSums][kThreads / 32 * kMaxCtas];  // [parity][sum][warp of the cluster]
  int my_rank, size, par;
  __device__ __forceinline__ int rank() const { return my_rank; }
  __device__ __forceinline__ int ncta() const { return size; }
  __device__ __forceinline__ void arrive() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  }
  __device__ __forceinline__ bool wait() {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    return true;
  }
  // every warp sends its partial sums to every CTA, then adds all of them in the same order
  template <int W, bool FENCE>
  __device__ __forceinline__ bool sum(double (&v)[W]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < W; ++k) {
      const double t = warp_reduce<SumOp>(v[k]);
      if (lane < size)
        st_cluster(map_shared(smem_u32(&red[par][k][my_rank * nw + warp]), (unsigned)lane), t);
    }
    arrive();
    wait();
    const int total = nw * size;
#pragma unroll
    for (int k = 0; k < W; ++k) {
      double a = 0.0;
      for (int i = lane; i < total; i += 32) a = dadd(a, red[par][k][i]);
      v[k] = warp_reduce<SumOp>(a);
    }
    par ^= 1;
    return true;
  }
};
template <class Team>
__device__ __forceinline__ bool barrier(Team& t) {
  t.arrive();
  return t.wait();
}
// This CTA's range of `n` units (slices, rows).
template <class Team>
__device__ __forceinline__ int from(const Team& t, int n) {
  return (int)((long long)n * t.rank() / t.ncta());
}
template <class Team>
__device__ __forceinline__ int to(const Team& t, int n) {
  return (int)((long long)n * (t.rank() + 1) / t.ncta());
}

template <typename T>
struct Pair2;
template <>
struct Pair2<float> {
  using type = float2;
};
template <>
struct Pair2<double> {
  using type = double2;
};

__device__ __forceinline__ float fmat(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fmat(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float mulr(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mulr(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float addr(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double addr(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float arith(__half v) { return __half2float(v); }
__device__ __forceinline__ float arith(float v) { return v; }
__device__ __forceinline__ double arith(double v) { return v; }
// p = z + beta p as the separate kernels round it: one FMA in FP32, GIP's rounding in FP64
__device__ __forceinline__ float dir(float2 q, float beta) { return fmaf(beta, q.y, q.x); }
__device__ __forceinline__ double dir(double2 q, double beta) { return dadd(q.x, dmul(beta, q.y)); }
// term of the CG's own product: FMA in FP32, GIP's rounding in FP64
__device__ __forceinline__ float term(float x, float v, float s) { return fmaf(x, v, s); }
__device__ __forceinline__ double term(double x, double v, double s) { return dadd(s, dmul(x, v)); }

// The level-0 operator: packed rows (NIB = 4 or 8) with plain slices beside them, or the
// sliced layout alone (NIB = 0).  FP64: L itself, ghost columns (stored zeros) dropped.
template <typename T>
struct Op0 {
  SellView<T> A;
  const uint4* delta;
  const void* idx;
  const int* base;
  const unsigned char* plain;
  const T* table;
  int slots;   // 7: no packed row uses the eighth slot
  int cols;    // columns the iterations gather (ghost columns lie past them)
};

// One product of the V-cycle below the level-0 operator.
enum { kSell = 0, kCsr, kDense };
enum { kOpPlain = 0, kOpResid, kOpScaleAdd, kOpSmooth, kOpDiagAdd };
template <typename T>
struct CycleOp {
  int form, mode, nrows;
  int lanes;               // threads per row (a power of two)
  int units;               // passes of a warp: 32 / lanes rows each
  int half, scaled;        // values in FP16; the gathered vector scaled by xs
  const long long* sptr;
  const int* rp;
  const int* col;
  const void* val;
  const T* x;
  const T* b;
  const T* dinv;
  const T* xs;
  T* y;
  T w;
};

template <typename T>
struct SolveArgs {
  Op0<T> op;
  // FP64 side: the true residual (mixed) or the solve itself
  SellView<double> L;
  const unsigned* lidx;     // packed FP64 residual: value indices of the packed columns
  const double* ltable;
  const double* bp;         // right-hand side less the ghost part (b without ghost rows)
  const double* b;
  const double* x0;
  double* x;
  const double* scale;
  typename Pair2<T>::type* pair;
  T* r;
  T* q;                     // A p
  float* y;                 // mixed: correction
  double* rd;               // mixed, pinned: FP64 residual, then its sum's block partials
  double* rpart;
  int vblocks;              // blocks of the kernel whose order the sum keeps
  PcgScalars* S;
  int* gave_up;             // host flag: a wait gave up
  ulonglong2* slots;
  const CycleOp<T>* ops;    // null: no preconditioner beyond the Jacobi scaling
  int nops;                 // level 0's residual first, its smoothing after the last
  T* t0;                    // level 0: residual
  T* xc0;                   // level 0: iterate after the prolongation
  const T* dinv0;           // level 0 smoother (null: the constant w0)
  T w0;
  double tol, delta, pin_val;
  int n, n_all, maxit, max_outer, pin_row;
  int nib;                  // value-table index bits of the packed operator, 0: not packed
  int count;                // launches the solve's scalars report
};

struct State {
  double rz, beta, alpha, pAp, bb, rr, maxr2, trig, kappa_c, kappa;
  int total, outer, status, done, upd;
};

// ------------------------------------------------------------------ rows
template <typename T>
__device__ __forceinline__ void op0_words(const Op0<T>& O, int nib, int s, int lane, PackedWords& w) {
  const int i = s * 32 + lane;
  w.plain = __ldg(O.plain + s);
  w.d = __ldg(O.delta + i);
  if (nib == 4) {
    w.w0 = __ldg(static_cast<const unsigned*>(O.idx) + i);
    w.w1 = 0u;
  } else {
    const uint2 t = __ldg(static_cast<const uint2*>(O.idx) + i);
    w.w0 = t.x;
    w.w1 = t.y;
  }
}

// The first packed words of this warp's level-0 slices (loaded ahead of a phase's wait).
constexpr int kSlices = 2;  // slices a warp works on at once
struct Words {
  PackedWords w[kSlices];
};
template <typename T, class Team>
__device__ __forceinline__ void words_ahead(const Op0<T>& O, int nib, const Team& g, Words& W) {
  const int lane = threadIdx.x & 31, nw = kThreads >> 5;
  const int s = from(g, O.A.nslices) + (int)(threadIdx.x >> 5), s1 = to(g, O.A.nslices);
#pragma unroll
  for (int h = 0; h < kSlices; ++h) {
    W.w[h].plain = 1;
    if (nib && s + h * nw < s1) op0_words(O, nib, s + h * nw, lane, W.w[h]);
  }
}

// This CTA's level-0 rows: load(column) reads what is gathered and val(it) makes the gathered
// value of it, own(row) loads what the row's result needs (issued with the gathers),
// finish(row, sum, own) takes the result (rows past n are skipped).  CG: the rounding of the
// CG's own product, else the V-cycle's (FMA).  A warp works on kSlices packed slices at once,
// all their loads in one branch-free run, and loads its next slices' words behind them.
template <typename T, bool CG>
__device__ __forceinline__ T op0_sum(const T* tab, int nib, unsigned w0, unsigned w1, const T (&xv)[8]) {
  T sum = T(0);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const unsigned k = nib == 4 ? (w0 >> (4 * j)) & 15u : ((j < 4 ? w0 : w1) >> (8 * (j & 3))) & 255u;
    sum = CG ? term(xv[j], tab[k], sum) : fmat(xv[j], tab[k], sum);
  }
  return sum;
}

template <typename T, bool CG, class Team, class F, class Q, class R, class E>
__device__ __forceinline__ void op0_rows(const Op0<T>& O, int nib, int n, const T* tab, const Team& g,
                                         Words& W, F load, Q val, R own, E finish) {
  const int lane = threadIdx.x & 31, nw = kThreads >> 5;
  const int s1 = to(g, O.A.nslices);
  const bool eight = O.slots == 8;
  for (int sb = from(g, O.A.nslices) + (int)(threadIdx.x >> 5); sb < s1; sb += kSlices * nw) {
    bool fast = sb + (kSlices - 1) * nw < s1;
#pragma unroll
    for (int h = 0; h < kSlices; ++h) fast = fast && !W.w[h].plain;
    unsigned w0[kSlices], w1[kSlices];
    bool plain[kSlices];
    uint4 wd[kSlices];
#pragma unroll
    for (int h = 0; h < kSlices; ++h) {
      w0[h] = W.w[h].w0;
      w1[h] = W.w[h].w1;
      wd[h] = W.w[h].d;
      plain[h] = W.w[h].plain != 0;
    }
    if (fast) {
      decltype(load(0)) raw[kSlices][8];
      decltype(own(0)) mine[kSlices];
#pragma unroll
      for (int h = 0; h < kSlices; ++h) {
        const int s = sb + h * nw;
        int c[8];
        packed_cols(O.base, s, wd[h], c);
#pragma unroll
        for (int j = 0; j < 7; ++j) raw[h][j] = load(c[j]);
        raw[h][7] = load(eight ? c[7] : c[0]);
        mine[h] = own(min(s * 32 + lane, n - 1));
      }
#pragma unroll
      for (int h = 0; h < kSlices; ++h)
        if (sb + (kSlices + h) * nw < s1) op0_words(O, nib, sb + (kSlices + h) * nw, lane, W.w[h]);
#pragma unroll
      for (int h = 0; h < kSlices; ++h) {
        T xv[8];
#pragma unroll
        for (int j = 0; j < 7; ++j) xv[j] = val(raw[h][j]);
        xv[7] = eight ? val(raw[h][7]) : T(0);
        const T sum = op0_sum<T, CG>(tab, nib, w0[h], w1[h], xv);
        const int i = (sb + h * nw) * 32 + lane;
        if (i < n) finish(i, sum, mine[h]);
      }
      continue;
    }
#pragma unroll
    for (int h = 0; h < kSlices; ++h) {
      const int s = sb + h * nw, i = s * 32 + lane;
      if (s >= s1) continue;
      T sum = T(0);
      if (!plain[h]) {
        int c[8];
        packed_cols(O.base, s, wd[h], c);
        T xv[8];
#pragma unroll
        for (int j = 0; j < 7; ++j) xv[j] = val(load(c[j]));
        xv[7] = eight ? val(load(c[7])) : T(0);
        sum = op0_sum<T, CG>(tab, nib, w0[h], w1[h], xv);
      } else {
        long long base;
        int len;
        slice_range(O.A, s, base, len);
        for (int j = 0; j < len; ++j) {
          const int c = __ldg(O.A.col + base + 32LL * j + lane);
          if (c >= 0 && c < O.cols) {
            const T v = __ldg(O.A.val + base + 32LL * j + lane), xc = val(load(c));
            sum = CG ? term(xc, v, sum) : fmat(xc, v, sum);
          }
        }
      }
      if (i < n) finish(i, sum, own(i));
      if (nib && s + kSlices * nw < s1) op0_words(O, nib, s + kSlices * nw, lane, W.w[h]);
    }
  }
}

// ------------------------------------------------------------------ the cycle's products
// A warp's first unit of a product (32 / LANES rows) and each thread's first eight entries of
// it: loaded ahead of the phase's wait.
template <typename T>
struct Ahead {
  int u, uend;
  int k, len;  // sliced: first slot of the thread's row and the slice's length; CSR: first
               // entry and the row's length
  int c[8];
  T v[8];
};

// Entries first, first + step, ... (eight of them, those below `len`) of a row at k0.
template <typename T, typename V, int STEP, int STRIDE>
__device__ __forceinline__ void load8(const CycleOp<T>& o, int k0, int first, int len, Ahead<T>& a) {
  const int* __restrict__ cp = o.col + k0 + first * STRIDE;
  const V* __restrict__ vp = static_cast<const V*>(o.val) + k0 + first * STRIDE;
  const int left = len - first;
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const bool in = t * STEP < left;
    a.c[t] = in ? __ldg(cp + t * STEP * STRIDE) : -1;
    a.v[t] = in ? (T)arith(__ldg(vp + t * STEP * STRIDE)) : T(0);
  }
}
template <typename T, bool XS>
__device__ __forceinline__ void gather8(const CycleOp<T>& o, const Ahead<T>& a, T (&xv)[8]) {
  const T* x = o.x;
#pragma unroll
  for (int t = 0; t < 8; ++t)
    xv[t] = a.c[t] >= 0 ? (XS ? mulr(__ldg(o.xs + a.c[t]), x[a.c[t]]) : x[a.c[t]]) : T(0);
}
// A row's own operands, loaded with its gathers, and its result.
template <typename T>
struct RowOps {
  T b, d, x;
};
template <typename T>
__device__ __forceinline__ RowOps<T> row_ops(const CycleOp<T>& o, int i, bool writes) {
  RowOps<T> r{T(0), T(0), T(0)};
  if (writes && o.mode != kOpPlain) {
    r.b = o.b[i];
    if (o.mode >= kOpSmooth) r.d = __ldg(o.dinv + i);
    if (o.mode == kOpSmooth) r.x = o.x[i];
  }
  return r;
}
template <typename T>
__device__ __forceinline__ void row_store(const CycleOp<T>& o, int i, const RowOps<T>& r, T sum) {
  T y = sum;
  if (o.mode == kOpResid) y = r.b - sum;
  else if (o.mode == kOpScaleAdd) y = fmat(o.w, r.b, sum);
  else if (o.mode == kOpDiagAdd) y = addr(mulr(r.d, r.b), sum);
  else if (o.mode == kOpSmooth) y = fmat(r.d, r.b - sum, r.x);
  o.y[i] = y;
}

// Sliced rows, LANES threads per row: each takes runs of eight consecutive slots, and the
// running sum passes from thread to thread, so a row is still one chain of FMAs in slot
// order, but a row of 29 slots costs one round trip instead of four.
template <typename T, int LANES>
__device__ __forceinline__ void sell_unit(const CycleOp<T>& o, int u, int& k, int& len) {
  constexpr int RPW = 32 / LANES;
  const int lane = threadIdx.x & 31, s = u / LANES;
  const int b0 = (int)__ldg(o.sptr + s);
  len = ((int)__ldg(o.sptr + s + 1) - b0) >> 5;
  k = b0 + (u % LANES) * RPW + lane / LANES;
}
template <typename T, typename V, bool XS, int LANES>
__device__ __forceinline__ void sell_run(const CycleOp<T>& o, Ahead<T>& a) {
  constexpr int RPW = 32 / LANES;
  const int lane = threadIdx.x & 31, sub = lane % LANES, nw = kThreads >> 5;
  while (a.u < a.uend) {
    const int i = (a.u / LANES) * 32 + (a.u % LANES) * RPW + lane / LANES;
    const bool writes = i < o.nrows && sub == 0;
    const RowOps<T> r = row_ops(o, i, writes);
    int k1 = 0, len1 = 0;  // the warp's next unit
    if (a.u + nw < a.uend) sell_unit<T, LANES>(o, a.u + nw, k1, len1);
    T sum = T(0);
    for (int j0 = 0;;) {
      T xv[8], v[8];
      gather8<T, XS>(o, a, xv);
#pragma unroll
      for (int t = 0; t < 8; ++t) v[t] = a.v[t];
      j0 += 8 * LANES;
      const bool last = j0 >= a.len;
      if (last) {
        a.u += nw;
        a.k = k1;
        a.len = len1;
      }
      load8<T, V, 1, 32>(o, a.k, (last ? 0 : j0) + 8 * sub, a.len, a);
#pragma unroll
      for (int q = 0; q < LANES; ++q) {
        T part = sum;
#pragma unroll
        for (int t = 0; t < 8; ++t) part = fmat(xv[t], v[t], part);
        sum = LANES == 1 ? part : __shfl_sync(0xffffffffu, part, (lane & ~(LANES - 1)) | q);
      }
      if (last) break;
    }
    if (writes) row_store(o, i, r, sum);
  }
}

// CSR rows, LANES threads per row, each adding a strided part, combined by a fixed tree,
// the next unit's loads as above
template <typename T, int LANES>
__device__ __forceinline__ void csr_unit(const CycleOp<T>& o, int u, int& k, int& len) {
  const int i = u * (32 / LANES) + (int)(threadIdx.x & 31) / LANES;
  k = len = 0;
  if (i < o.nrows) {
    k = __ldg(o.rp + i);
    len = __ldg(o.rp + i + 1) - k;
  }
}
template <typename T, typename V, bool XS, int LANES>
__device__ __forceinline__ void csr_run(const CycleOp<T>& o, Ahead<T>& a) {
  const int lane = threadIdx.x & 31, sub = lane % LANES, nw = kThreads >> 5;
  while (a.u < a.uend) {
    const int i = a.u * (32 / LANES) + lane / LANES;
    const bool writes = i < o.nrows && sub == 0;
    const RowOps<T> r = row_ops(o, i, writes);
    int k1 = 0, len1 = 0;
    if (a.u + nw < a.uend) csr_unit<T, LANES>(o, a.u + nw, k1, len1);
    T sum = T(0);
    for (int q0 = sub;;) {
      T xv[8], v[8];
      gather8<T, XS>(o, a, xv);
      unsigned in = 0;
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        v[t] = a.v[t];
        in |= (a.c[t] >= 0 ? 1u : 0u) << t;
      }
      q0 += 8 * LANES;
      const bool more = __any_sync(0xffffffffu, q0 < a.len);
      if (!more) {
        a.k = k1;
        a.len = len1;
        q0 = sub;
      }
      load8<T, V, LANES, 1>(o, a.k, q0, a.len, a);
#pragma unroll
      for (int t = 0; t < 8; ++t)
        if (in >> t & 1u) sum = fmat(v[t], xv[t], sum);
      if (!more) break;
    }
#pragma unroll
    for (int d = LANES / 2; d > 0; d >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, d, LANES);
    if (writes) row_store(o, i, r, sum);
    a.u += nw;
  }
}

// Dense rows, a warp per row.
template <typename T>
__device__ __forceinline__ void dense_load(const CycleOp<T>& o, int i, int j0, Ahead<T>& a) {
  const T* __restrict__ C = static_cast<const T*>(o.val) + (size_t)i * o.nrows + j0;
#pragma unroll
  for (int t = 0; t < 8; ++t) a.v[t] = j0 + 32 * t < o.nrows ? __ldg(C + 32 * t) : T(0);
}
template <typename T>
__device__ __forceinline__ void dense_run(const CycleOp<T>& o, Ahead<T>& a) {
  const int lane = threadIdx.x & 31, nw = kThreads >> 5, m = o.nrows;
  const T* x = o.x;
  for (; a.u < a.uend; a.u += nw) {
    T sum = T(0);
    for (int j0 = lane;;) {
      T xv[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) xv[t] = j0 + 32 * t < m ? x[j0 + 32 * t] : T(0);
#pragma unroll
      for (int t = 0; t < 8; ++t)
        if (j0 + 32 * t < m) sum = fmat(a.v[t], xv[t], sum);
      j0 += 256;
      if (j0 >= m) break;
      dense_load(o, a.u, j0, a);
    }
    __syncwarp();
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, d);
    if (lane == 0) o.y[a.u] = sum;
    if (a.u + nw < a.uend) dense_load(o, a.u + nw, lane, a);
  }
}

// What a product reads first, none of it written inside the launch.
template <typename T, typename V, class Team>
__device__ __forceinline__ void first_load(const CycleOp<T>& o, Ahead<T>& a) {
  const int lane = threadIdx.x & 31;
  if (o.form == kSell) {
    if (o.lanes == 4) {
      sell_unit<T, 4>(o, a.u, a.k, a.len);
      load8<T, V, 1, 32>(o, a.k, 8 * (lane % 4), a.len, a);
    } else if (o.lanes == 2) {
      sell_unit<T, 2>(o, a.u, a.k, a.len);
      load8<T, V, 1, 32>(o, a.k, 8 * (lane % 2), a.len, a);
    } else {
      sell_unit<T, 1>(o, a.u, a.k, a.len);
      load8<T, V, 1, 32>(o, a.k, 0, a.len, a);
    }
  } else if (o.lanes == 32) {
    csr_unit<T, 32>(o, a.u, a.k, a.len);
    load8<T, V, 32, 1>(o, a.k, lane, a.len, a);
  } else if (o.lanes == 16) {
    csr_unit<T, 16>(o, a.u, a.k, a.len);
    load8<T, V, 16, 1>(o, a.k, lane % 16, a.len, a);
  } else if (o.lanes == 8) {
    csr_unit<T, 8>(o, a.u, a.k, a.len);
    load8<T, V, 8, 1>(o, a.k, lane % 8, a.len, a);
  } else {
    csr_unit<T, 4>(o, a.u, a.k, a.len);
    load8<T, V, 4, 1>(o, a.k, lane % 4, a.len, a);
  }
}
template <typename T, class Team>
__device__ __forceinline__ void product_ahead(const CycleOp<T>& o, const Team& g, Ahead<T>& a) {
  a.u = from(g, o.units) + (int)(threadIdx.x >> 5);
  a.uend = to(g, o.units);
  if (a.u >= a.uend) return;
  if (o.form == kDense) {
    dense_load(o, a.u, (int)(threadIdx.x & 31), a);
    return;
  }
  if constexpr (std::is_same<T, float>::value) {
    if (o.half) {
      first_load<T, __half, Team>(o, a);
      return;
    }
  }
  first_load<T, T, Team>(o, a);
}
template <typename T, typename V, bool XS>
__device__ __forceinline__ void sparse_run(const CycleOp<T>& o, Ahead<T>& a) {
  if (o.form == kSell) {
    if (o.lanes == 4) sell_run<T, V, XS, 4>(o, a);
    else if (o.lanes == 2) sell_run<T, V, XS, 2>(o, a);
    else sell_run<T, V, XS, 1>(o, a);
  } else if (o.lanes == 32) {
    csr_run<T, V, XS, 32>(o, a);
  } else if (o.lanes == 16) {
    csr_run<T, V, XS, 16>(o, a);
  } else if (o.lanes == 8) {
    csr_run<T, V, XS, 8>(o, a);
  } else {
    csr_run<T, V, XS, 4>(o, a);
  }
}
template <typename T>
__device__ __forceinline__ void product_run(const CycleOp<T>& shared_op, Ahead<T>& a) {
  const CycleOp<T> o = shared_op;
  if (o.form == kDense) {
    dense_run<T>(o, a);
    return;
  }
  if constexpr (std::is_same<T, float>::value) {
    if (o.half) {
      sparse_run<T, __half, false>(o, a);
      return;
    }
  }
  if (o.scaled) sparse_run<T, T, true>(o, a);
  else sparse_run<T, T, false>(o, a);
}

// r = b - L x of one row of the mixed form's FP64 residual, in the order of the kernel it
// replaces: packed columns against the value table and b', else L's own row against b.
__device__ __forceinline__ double true_residual(const SolveArgs<float>& A, const double* ltab,
                                                const double* x, int s, int lane) {
  const int i = s * 32 + lane;
  if (A.lidx) {
    const uint4 d = __ldg(A.op.delta + i);
    const unsigned w = __ldg(A.lidx + i);
    if (!__ldg(A.op.plain + s)) {
      int c[8];
      packed_cols(A.op.base, s, d, c);
      double xv[8], sum = 0.0;
#pragma unroll
      for (int j = 0; j < 8; ++j) xv[j] = x[c[j]];
#pragma unroll
      for (int j = 0; j < 8; ++j) sum = dadd(sum, dmul(xv[j], ltab[(w >> (4 * j)) & 15u]));
      return i < A.n ? A.bp[i] - sum : 0.0;
    }
  }
  long long base;
  int len;
  slice_range(A.L, s, base, len);
  double sum = 0.0;
  for (int j = 0; j < len; ++j) {
    const int c = __ldg(A.L.col + base + 32LL * j + lane);
    if (c >= 0) sum = dadd(sum, dmul(x[c], __ldg(A.L.val + base + 32LL * j + lane)));
  }
  return i < A.n ? A.b[i] - sum : 0.0;
}

// ------------------------------------------------------------------ scalars (thread 0)
__device__ __forceinline__ void mixed_residual_finish(const SolveArgs<float>& A, State& T, int first,
                                                      bool amg, const double (&t)[5]) {
  if (first) T.bb = t[2];
  T.rr = t[0];
  double rz = t[1];
  T.kappa_c = 0.0;
  const int pin = A.pin_row;
  if (pin >= 0) {
    const float old = (float)t[4];
    const float nw = (float)((double)old - A.scale[pin] * t[3]);
    rz = rz - (double)old * (double)old + (double)nw * (double)nw;
    T.kappa_c = t[3] / A.pin_val;
  }
  if (!first) {
    if (!amg) T.beta = rz / T.rz;
    T.outer += 1;
  }
  if (!amg) T.rz = rz;
  T.maxr2 = rz;
  const double goal = 0.5 * A.tol * sqrt(T.bb);
  T.trig = (t[0] > 0.0) ? rz * (goal * goal) / t[0] : 0.0;
  const bool finite = isfinite(t[0]) && isfinite(T.bb);
  const bool conv = finite && !(sqrt(t[0]) > A.tol * sqrt(T.bb));
  if (conv || !finite || T.total >= A.maxit || T.outer >= A.max_outer) {
    if (!conv) T.status = finite ? GIPB200_ERR_NOT_CONVERGED : GIPB200_ERR_BREAKDOWN;
    T.done = 1;
  }
}

// sum of rd[0..n) in the order of the separate residual kernel's grid reduction (vblocks
// blocks of 256 threads, a row per thread and pass).  This sum over the pin's small value
// becomes a constant added to x, and the rounding of b - L x at that constant decides the last
// bit of the next FP32 residual: a different order of this one sum makes other iterates (to
// 1e-9 of the smallest velocity component on the 63^3 cavity), the same order the same ones.
// Every thread of the team receives it; rd's writes are ordered by a barrier before the call.
template <class Team>
__device__ __forceinline__ bool ordered_sum(const double* rd, double* part, int n, int vblocks,
                                            Team& g, double& total) {
  __shared__ double sh[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kAtOnce = kThreads / 256;
  const int ns = (n + 31) / 32, vw = vblocks * 8;
  for (int v0 = g.rank() * kAtOnce; v0 < vblocks; v0 += g.ncta() * kAtOnce) {
    const int v = v0 + (warp >> 3);
    double acc = 0.0;
    if (v < vblocks)
      for (int s = v * 8 + (warp & 7); s < ns; s += vw) {
        const int i = s * 32 + lane;
        if (i < n) acc += rd[i];
      }
    acc = warp_reduce<SumOp>(acc);
    __syncthreads();
    if (lane == 0) sh[warp] = acc;
    __syncthreads();
    if ((warp & 7) == 0) {
      const double t = warp_reduce<SumOp>(lane < 8 ? sh[warp + lane] : 0.0);
      if (lane == 0 && v < vblocks) part[v] = t;
    }
  }
  if (!barrier(g)) return false;
  double a = 0.0;
  if (threadIdx.x < 256)
    for (int b = threadIdx.x; b < vblocks; b += 256) a = dadd(a, part[b]);
  a = warp_reduce<SumOp>(a);
  __syncthreads();
  if (lane == 0) sh[warp] = a;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < 8; ++w) t = dadd(t, sh[w]);
  total = t;
  return true;
}

__device__ __forceinline__ void cycle_finish(State& T, double rz, bool first) {
  if (!(rz > 0.0) || !isfinite(rz)) {  // preconditioner lost definiteness: restart CG
    T.beta = 0.0;
    T.rz = 0.0;
    return;
  }
  T.beta = (!first && T.rz > 0.0) ? rz / T.rz : 0.0;
  T.rz = rz;
}

// z = M r: level 0's residual from zero, the products below, level 0's smoothing with r.z.
// `W` holds the first level-0 words on entry and on exit.  False: a barrier gave up.
template <typename T, class Team>
__device__ __forceinline__ bool vcycle(const SolveArgs<T>& A, const CycleOp<T>* ops, const T* tab,
                                       Team& g, Words& W, double& rz) {
  const int n = A.n;
  const T* d0 = A.dinv0;
  const T w0 = A.w0;
  {  // t = r - A D^-1 r
    const T* r = A.r;
    T* t0 = A.t0;
    if (d0)
      op0_rows<T, false>(A.op, A.nib, n, tab, g, W,
                         [&](int c) {
                           typename Pair2<T>::type q;
                           q.x = __ldg(d0 + c);
                           q.y = r[c];
                           return q;
                         },
                         [](typename Pair2<T>::type q) { return mulr(q.x, q.y); },
                         [&](int i) { return r[i]; },
                         [&](int i, T sum, T ri) { t0[i] = ri - sum; });
    else
      op0_rows<T, false>(A.op, A.nib, n, tab, g, W, [&](int c) { return r[c]; },
                         [](T q) { return q; }, [&](int i) { return r[i]; },
                         [&](int i, T sum, T ri) { t0[i] = fmat(-w0, sum, ri); });
  }
  Ahead<T> w;
  for (int k = 0; k < A.nops; ++k) {
    g.arrive();
    product_ahead<T>(ops[k], g, w);
    if (!g.wait()) return false;
    product_run<T>(ops[k], w);
  }
  g.arrive();
  words_ahead(A.op, A.nib, g, W);
  if (!g.wait()) return false;
  double acc[1] = {0.0};
  {
    const T* x = A.xc0;
    const T* r = A.r;
    typename Pair2<T>::type* pair = A.pair;
    struct Own {
      T r, x, d;
    };
    op0_rows<T, false>(A.op, A.nib, n, tab, g, W, [&](int c) { return x[c]; }, [](T q) { return q; },
                       [&](int i) {
                         return Own{r[i], x[i], d0 ? __ldg(d0 + i) : w0};
                       },
                       [&](int i, T sum, Own o) {
                         const T zi = fmat(o.d, o.r - sum, o.x);
                         pair[i].x = zi;
                         acc[0] += (double)o.r * (double)zi;
                       });
  }
  words_ahead(A.op, A.nib, g, W);
  if (!g.template sum<1, true>(acc)) return false;
  rz = acc[0];
  return true;
}

// ------------------------------------------------------------------ mixed form
template <bool AMG, class Team>
__device__ __forceinline__ void mixed_solve(const SolveArgs<float>& A, Team& g) {
  __shared__ State T;
  __shared__ float tab[256];
  __shared__ double ltab[16];
  __shared__ CycleOp<float> ops[AMG ? kMaxOps : 1];
  for (int t = threadIdx.x; t < (1 << A.nib) && A.nib; t += kThreads) tab[t] = A.op.table[t];
  if (AMG && (int)threadIdx.x < A.nops) ops[threadIdx.x] = A.ops[threadIdx.x];
  if (A.lidx && threadIdx.x < 16) ltab[threadIdx.x] = A.ltable[threadIdx.x];
  if (threadIdx.x == 0) {
    T = State{};
    T.status = GIPB200_OK;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, nw = kThreads >> 5;
  const int s0 = from(g, A.op.A.nslices), s1 = to(g, A.op.A.nslices), sb = s0 + (int)(threadIdx.x >> 5);
  const int n = A.n, gt = g.rank() * kThreads + (int)threadIdx.x, nt = g.ncta() * kThreads;
  const bool lead = threadIdx.x == 0;
  float2* pair = A.pair;
  Words W;

  // the FP64 true residual replaces the FP32 one (first: and starts y, the direction)
  auto residual = [&](int first) -> bool {
    double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    const double* x = first ? A.x0 : A.x;
    for (int s = sb; s < s1; s += nw) {
      const int i = s * 32 + lane;
      const double ri = true_residual(A, ltab, x, s, lane);
      if (i < n) {
        const float rh = (float)(ri * A.scale[i]);
        const double bi = A.b[i];
        if (AMG) A.r[i] = rh;
        if (first) A.y[i] = 0.f;
        if (!AMG || first) pair[i] = make_float2(rh, first ? (AMG ? rh : 0.f) : pair[i].y);
        acc[0] += ri * ri;
        acc[1] += (double)rh * (double)rh;
        acc[2] += bi * bi;
        if (A.pin_row >= 0) A.rd[i] = ri;
        if (i == A.pin_row) acc[4] = rh;
      }
    }
    if (!g.template sum<5, true>(acc)) return false;
    if (A.pin_row >= 0 && !ordered_sum(A.rd, A.rpart, n, A.vblocks, g, acc[3])) return false;
    if (lead) mixed_residual_finish(A, T, first, AMG, acc);
    if (A.pin_row >= 0) {
      // the pinned entry, adjusted by the thread that owns its row before anyone gathers it
      const int pin = A.pin_row, ps = pin >> 5;
      if (ps >= s0 && ps < s1 && (ps - s0) % nw == (int)(threadIdx.x >> 5) && lane == (pin & 31)) {
        const float old = (float)acc[4];
        const float nv = (float)((double)old - A.scale[pin] * acc[3]);
        if (AMG) A.r[pin] = nv;
        else pair[pin].x = nv;
        if (AMG && first) pair[pin].y = nv;
      }
      g.arrive();
      words_ahead(A.op, A.nib, g, W);
      const bool ok = g.wait();
      __syncthreads();  // T, for the cluster's threads
      return ok;
    }
    words_ahead(A.op, A.nib, g, W);
    __syncthreads();
    return true;
  };
  auto precondition = [&]() -> bool {
    if constexpr (AMG) {
      double rz;
      if (!vcycle<float>(A, ops, tab, g, W, rz)) return false;
      if (lead) cycle_finish(T, rz, false);
      __syncthreads();
    }
    return true;
  };

  bool ok = residual(1);
  if (ok && A.x != A.x0)  // (every row has read x0)
    for (int i = gt; i < A.n_all; i += nt) A.x[i] = A.x0[i];
  if (ok && !T.done) ok = precondition();
  while (ok && !T.done) {
    // A p and p.Ap
    const float beta = (float)T.beta;
    double d[1] = {0.0};
    {
      float* q = A.q;
      op0_rows<float, true>(A.op, A.nib, n, tab, g, W, [&](int c) { return pair[c]; },
                            [&](float2 q) { return dir(q, beta); },
                            [&](int i) { return dir(pair[i], beta); },
                            [&](int i, float sum, float pi) {
                              q[i] = sum;
                              d[0] += (double)pi * (double)sum;
                            });
    }
    if (!(ok = g.template sum<1, false>(d))) break;
    if (lead) {
      T.pAp = d[0];
      T.alpha = T.rz / d[0];
      if (!(d[0] > 0.0) || !isfinite(T.alpha)) T.alpha = 0.0;  // direction lost: replace
    }
    __syncthreads();
    // y += alpha p, r -= alpha A p, r.r
    const float alpha = (float)T.alpha;
    double e[2] = {0.0, 0.0};
    {
      float* y = A.y;
      float* r = A.r;
      const float* q = A.q;
      const int pin = A.pin_row;
      constexpr int U = 4;  // slices whose loads are in flight together
      for (int s = sb; s < s1; s += U * nw) {
        float2 zp[U];
        float yv[U], qv[U], rv[U];
#pragma unroll
        for (int h = 0; h < U; ++h) {
          const int i = min((s + h * nw) * 32 + lane, n - 1);
          zp[h] = pair[i];
          yv[h] = y[i];
          qv[h] = q[i];
          rv[h] = AMG ? r[i] : 0.f;
        }
#pragma unroll
        for (int h = 0; h < U; ++h) {
          const int i = (s + h * nw) * 32 + lane;
          if (s + h * nw >= s1 || i >= n) continue;
          const float pi = dir(zp[h], beta);
          const float yi = fmaf(alpha, pi, yv[h]);
          const float ri = fmaf(-alpha, qv[h], AMG ? rv[h] : zp[h].x);
          y[i] = yi;
          if (AMG) r[i] = ri;
          pair[i] = make_float2(AMG ? zp[h].x : ri, pi);
          e[0] += (double)ri * (double)ri;
          if (i == pin) e[1] = yi;
        }
      }
    }
    words_ahead(A.op, A.nib, g, W);
    if (!(ok = g.template sum<2, true>(e))) break;
    if (lead) {
      T.total += 1;
      const double rzn = e[0];
      if (rzn > T.maxr2) T.maxr2 = rzn;
      T.upd = !(rzn > T.trig) || !(rzn > A.delta * A.delta * T.maxr2) || T.alpha == 0.0 ||
              T.total >= A.maxit || !isfinite(rzn);
      if (T.upd) {
        T.kappa = (A.pin_row >= 0) ? T.kappa_c - A.scale[A.pin_row] * e[1] : 0.0;
      } else if (!AMG) {
        T.beta = rzn / T.rz;
        T.rz = rzn;
      }
    }
    __syncthreads();
    if (T.upd) {  // x += S y + kappa, y = 0, then the true residual
      const double kappa = T.kappa;
      for (int s = sb; s < s1; s += nw) {
        const int i = s * 32 + lane;
        if (i >= n) continue;
        A.x[i] += A.scale[i] * (double)A.y[i] + kappa;
        A.y[i] = 0.f;
      }
      if (!(ok = barrier(g))) break;
      if (!(ok = residual(0))) break;
      if (T.done) break;
    }
    ok = precondition();
  }
  if (!ok && lead) report_gave_up(A.gave_up);
  if (g.rank() == 0 && lead) {
    PcgScalars* S = A.S;
    S->rz = T.rz;
    S->pAp = T.pAp;
    S->alpha = T.alpha;
    S->beta = T.beta;
    S->rr = T.rr;
    S->bb = T.bb;
    S->iter = T.total;
    S->done = 1;
    S->inner_done = 1;
    S->status = ok ? T.status : GIPB200_ERR_TIMEOUT;
    S->outer = T.outer;
    S->total_inner = T.total;
    S->kernels = A.count;
    S->kappa_c = T.kappa_c;
    S->kappa = T.kappa;
    S->maxr2 = T.maxr2;
    S->trig = T.trig;
    S->upd = 0;
    S->one_launch = 1;
  }
}

__device__ __forceinline__ ClusterTeam cluster_team(
    double (*red)[kGridSums][kThreads / 32 * ClusterTeam::kMaxCtas]) {
  cluster_barrier();  // every CTA runs before its shared memory is written
  return ClusterTeam{red, (int)cluster_rank(), (int)cluster_size(), 0};
}

template <bool AMG>
__global__ void __launch_bounds__(kThreads, 1) k_mixed_grid(const __grid_constant__ SolveArgs<float> A) {
  GridTeam g{grid_begin(A.slots)};
  mixed_solve<AMG>(A, g);
}
template <bool AMG>
__global__ void __launch_bounds__(kThreads, 1) k_mixed_cluster(const __grid_constant__ SolveArgs<float> A) {
  __shared__ double red[2][kGridSums][kThreads / 32 * ClusterTeam::kMaxCtas];
  ClusterTeam g = cluster_team(red);
  mixed_solve<AMG>(A, g);
  cluster_barrier();  // no CTA leaves while another may still write its sums
}

// One CTA of a group that claims two: a solve without rows, whose first sum waits for a CTA that
// does not exist, or a barrier of that group.
__global__ void __launch_bounds__(kThreads, 1) k_mixed_wait_check(const __grid_constant__ SolveArgs<float> A,
                                                                  int barrier_only) {
  GridTeam g{grid_begin(A.slots, 0, 2, kCheckSpinCycles)};
  if (!barrier_only) {
    mixed_solve<false>(A, g);
  } else if (!barrier(g) && threadIdx.x == 0) {
    report_gave_up(A.gave_up);
    A.S->status = GIPB200_ERR_TIMEOUT;
  }
}

// The solves of a batch in one launch, a group of CTAs per instance; groups never wait on one
// another and leave when their instance has converged.
struct GroupSolve {
  SolveArgs<float> A;
  int cta0, ncta;
};
__global__ void __launch_bounds__(kThreads, 1) k_mixed_groups(const GroupSolve* __restrict__ all,
                                                              const int* __restrict__ owner) {
  __shared__ GroupSolve I;
  const int who = owner[blockIdx.x];
  if (who < 0) return;  // the groups do not fill the grid
  static_assert(sizeof(GroupSolve) % 4 == 0, "copied in words");
  for (int k = threadIdx.x; k < (int)(sizeof(GroupSolve) / 4); k += kThreads)
    reinterpret_cast<unsigned*>(&I)[k] = reinterpret_cast<const unsigned*>(all + who)[k];
  __syncthreads();
  GridTeam g{grid_begin(I.A.slots, (int)blockIdx.x - I.cta0, I.ncta)};
  mixed_solve<true>(I.A, g);
}

// ------------------------------------------------------------------ FP64 tolerance mode, AMG
template <class Team>
__device__ __forceinline__ void tol_amg_solve(const SolveArgs<double>& A, Team& g) {
  __shared__ State T;
  __shared__ double tab[256];
  __shared__ CycleOp<double> ops[kMaxOps];
  for (int t = threadIdx.x; t < (1 << A.nib) && A.nib; t += kThreads) tab[t] = A.op.table[t];
  if ((int)threadIdx.x < A.nops) ops[threadIdx.x] = A.ops[threadIdx.x];
  if (threadIdx.x == 0) {
    T = State{};
    T.status = GIPB200_OK;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, nw = kThreads >> 5;
  const int s1 = to(g, A.op.A.nslices), sb = from(g, A.op.A.nslices) + (int)(threadIdx.x >> 5);
  const int n = A.n;
  const bool lead = threadIdx.x == 0;
  double2* pair = A.pair;
  Words W;
  bool ok = true;
  {  // r = b - L x0 (ghost columns included), p = 0
    double acc[2] = {0.0, 0.0};
    for (int s = sb; s < s1; s += nw) {
      const int i = s * 32 + lane;
      long long base;
      int len;
      slice_range(A.L, s, base, len);
      double sum = 0.0;
      for (int j = 0; j < len; ++j) {
        const int c = __ldg(A.L.col + base + 32LL * j + lane);
        if (c >= 0) sum = dadd(sum, dmul(A.x0[c], __ldg(A.L.val + base + 32LL * j + lane)));
      }
      if (i < A.n) {
        const double bi = A.b[i];
        const double ri = dadd(bi, dmul(-1.0, sum));
        A.r[i] = ri;
        pair[i] = make_double2(0.0, 0.0);
        acc[0] = dadd(acc[0], dmul(ri, ri));
        acc[1] = dadd(acc[1], dmul(bi, bi));
      }
    }
    words_ahead(A.op, A.nib, g, W);
    ok = g.template sum<2, true>(acc);
    if (lead) {
      T.rr = acc[0];
      T.bb = acc[1];
      T.done = (A.maxit <= 0) ? 1 : 0;
      if (!(sqrt(acc[0]) > A.tol * sqrt(acc[1]))) T.done = 1;
      if (!(isfinite(acc[0]) && isfinite(acc[1]))) {
        T.status = GIPB200_ERR_BREAKDOWN;
        T.done = 1;
      }
    }
    __syncthreads();
  }
  if (ok && A.x != A.x0)
    for (int i = g.rank() * kThreads + (int)threadIdx.x; i < A.n_all; i += g.ncta() * kThreads)
      A.x[i] = A.x0[i];
  bool first = true;
  while (ok && !T.done) {
    double rz;
    if (!(ok = vcycle<double>(A, ops, tab, g, W, rz))) break;
    if (lead) cycle_finish(T, rz, first);
    first = false;
    __syncthreads();
    const double beta = T.beta;
    double d[1] = {0.0};
    {
      double* q = A.q;
      op0_rows<double, true>(A.op, A.nib, n, tab, g, W, [&](int c) { return pair[c]; },
                             [&](double2 q) { return dir(q, beta); },
                             [&](int i) { return dir(pair[i], beta); },
                             [&](int i, double sum, double pi) {
                               q[i] = sum;
                               d[0] = dadd(d[0], dmul(pi, sum));
                             });
    }
    if (!(ok = g.template sum<1, false>(d))) break;
    if (lead) {
      T.pAp = d[0];
      T.alpha = ddiv(T.rz, d[0]);
      if (!(d[0] > 0.0) || !isfinite(T.alpha)) {
        T.status = GIPB200_ERR_BREAKDOWN;
        T.done = 1;
      }
    }
    __syncthreads();
    if (T.done) break;
    const double alpha = T.alpha, malpha = dmul(-1.0, alpha);
    double e[1] = {0.0};
    {
      double* x = A.x;
      double* r = A.r;
      const double* q = A.q;
      constexpr int U = 2;  // slices whose loads are in flight together
      for (int s = sb; s < s1; s += U * nw) {
        double2 zp[U];
        double xv[U], qv[U], rv[U];
#pragma unroll
        for (int h = 0; h < U; ++h) {
          const int i = min((s + h * nw) * 32 + lane, n - 1);
          zp[h] = pair[i];
          xv[h] = x[i];
          qv[h] = q[i];
          rv[h] = r[i];
        }
#pragma unroll
        for (int h = 0; h < U; ++h) {
          const int i = (s + h * nw) * 32 + lane;
          if (s + h * nw >= s1 || i >= n) continue;
          const double pi = dir(zp[h], beta);
          x[i] = dadd(xv[h], dmul(alpha, pi));
          const double ri = dadd(rv[h], dmul(malpha, qv[h]));
          r[i] = ri;
          pair[i] = make_double2(zp[h].x, pi);
          e[0] = dadd(e[0], dmul(ri, ri));
        }
      }
    }
    words_ahead(A.op, A.nib, g, W);
    if (!(ok = g.template sum<1, true>(e))) break;
    if (lead) {
      T.rr = e[0];
      T.total += 1;
      if (!isfinite(e[0])) {
        T.status = GIPB200_ERR_BREAKDOWN;
        T.done = 1;
      } else if (!(sqrt(e[0]) > A.tol * sqrt(T.bb))) {
        T.done = 1;
      }
      if (T.total >= A.maxit) {
        if (!T.done) T.status = GIPB200_ERR_NOT_CONVERGED;
        T.done = 1;
      }
    }
    __syncthreads();
  }
  if (!ok && lead) report_gave_up(A.gave_up);
  if (g.rank() == 0 && lead) {
    PcgScalars* S = A.S;
    S->rz = T.rz;
    S->pAp = T.pAp;
    S->alpha = T.alpha;
    S->beta = T.beta;
    S->rr = T.rr;
    S->bb = T.bb;
    S->iter = T.total;
    S->done = 1;
    S->status = ok ? T.status : GIPB200_ERR_TIMEOUT;
    S->kernels = 0;
    S->one_launch = 1;
  }
}

__global__ void __launch_bounds__(kThreads, 1) k_tol_amg_grid(const __grid_constant__ SolveArgs<double> A) {
  GridTeam g{grid_begin(A.slots)};
  tol_amg_solve(A, g);
}
__global__ void __launch_bounds__(kThreads, 1) k_tol_amg_cluster(const __grid_constant__ SolveArgs<double> A) {
  __shared__ double red[2][kGridSums][kThreads / 32 * ClusterTeam::kMaxCtas];
  ClusterTeam g = cluster_team(red);
  tol_amg_solve(A, g);
  cluster_barrier();
}

// ------------------------------------------------------------------ small levels
// The V-cycle's small levels and the dense coarsest solve in one launch of one cluster, for
// cycles whose other levels run kernel by kernel.  Every product costs latency only: in a
// captured step about 3 us as a kernel of its own, 2 to 3 us here, a cluster barrier after the
// last; the launches they no longer need are what a batch's branches compete for.
template <typename T>
__global__ void __launch_bounds__(kThreads, 1) k_amg_small(const CycleOp<T>* __restrict__ all, int nops,
                                                           PcgScalars* S) {
  __shared__ CycleOp<T> ops[kMaxOps];
  for (int k = threadIdx.x; k < (int)(nops * sizeof(CycleOp<T>) / 4); k += kThreads)
    reinterpret_cast<unsigned*>(ops)[k] = reinterpret_cast<const unsigned*>(all)[k];
  __syncthreads();
  ClusterTeam g{nullptr, (int)blockIdx.x, (int)gridDim.x, 0};
  Ahead<T> w;
  product_ahead<T>(ops[0], g, w);
  dep_begin();
  if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&S->kernels, 1);
  if (S->done != 0) return;
  product_run<T>(ops[0], w);
  for (int k = 1; k < nops; ++k) {
    g.arrive();
    product_ahead<T>(ops[k], g, w);
    g.wait();
    product_run<T>(ops[k], w);
  }
}

}  // namespace

// ------------------------------------------------------------------ set-up
namespace {

// The cycle's products between level 0's residual and its smoothing; false: an operator has a
// form these kernels do not run (16-bit columns, FP16 coarse values, aggregate order).
template <typename T>
bool cycle_ops(const AmgT<T>& M, const T* r, int warps, std::vector<CycleOp<T>>* out) {
  const int L = (int)M.lv.size();
  if (L < 2 || M.nc <= 0 || M.perm0.p) return false;
  bool ok = true;
  auto add = [&](const SellT<T>& A, int mode, const T* x, const T* b, const T* dinv, const T* xs,
                 T* y, T w) {
    ok = ok && !A.short_cols && (!A.half || !xs);
    CycleOp<T> o{};
    o.form = A.lanes > 0 ? kCsr : kSell;
    o.mode = mode;
    o.nrows = A.nrows;
    o.lanes = A.lanes;
    if (A.lanes == 0) {  // threads per sliced row: what covers an average row in one pass,
                         // while the operator still fits the grid's warps in two passes
      o.lanes = 1;
      while (o.lanes < 4 && (double)A.nnz > 8.0 * o.lanes * A.nrows &&
             (long long)A.nslices * o.lanes <= (long long)warps)
        o.lanes *= 2;
    }
    o.units = A.lanes == 0 ? A.nslices * o.lanes : (A.nrows + 32 / o.lanes - 1) / (32 / o.lanes);
    o.half = A.half ? 1 : 0;
    o.scaled = xs ? 1 : 0;
    o.sptr = A.sptr.p;
    o.rp = A.rp.p;
    o.col = A.col.p;
    o.val = A.half ? (const void*)A.hval.p : (const void*)A.val.p;
    o.x = x;
    o.b = b;
    o.dinv = dinv;
    o.xs = xs;
    o.y = y;
    o.w = w;
    out->push_back(o);
  };
  for (int l = 0; l < L - 1; ++l) {
    const AmgLevel<T>& V = *M.lv[l];
    if (l > 0) add(V.A, kOpResid, V.b.p, V.b.p, nullptr, V.dinv.p, V.t.p, T(1));
    add(V.R, kOpPlain, V.t.p, nullptr, nullptr, nullptr, M.lv[l + 1]->b.p, T(1));
  }
  {
    const AmgLevel<T>& C = *M.lv[L - 1];
    CycleOp<T> o{};
    o.form = kDense;
    o.mode = kOpPlain;
    o.nrows = M.nc;
    o.lanes = 32;
    o.units = M.nc;
    o.val = M.cinv.p;
    o.x = C.b.p;
    o.y = C.x.p;
    out->push_back(o);
  }
  for (int l = L - 2; l >= 0; --l) {
    const AmgLevel<T>& V = *M.lv[l];
    const T* xc = (l + 1 == L - 1) ? M.lv[l + 1]->x.p : M.lv[l + 1]->t.p;
    if (l == 0 && M.unit0) add(V.P, kOpScaleAdd, xc, r, nullptr, nullptr, V.x.p, (T)M.omega0);
    else add(V.P, kOpDiagAdd, xc, l == 0 ? r : V.b.p, V.dinv.p, nullptr, V.x.p, T(1));
    if (l > 0) add(V.A, kOpSmooth, V.x.p, V.b.p, V.dinv.p, nullptr, V.t.p, T(1));
  }
  return ok && (int)out->size() <= kMaxOps;
}

template <typename T>
void cycle_args(const AmgT<T>& M, SolveArgs<T>* A) {
  A->t0 = M.lv[0]->t.p;
  A->xc0 = M.lv[0]->x.p;
  A->dinv0 = M.unit0 ? nullptr : M.lv[0]->dinv.p;
  A->w0 = (T)M.omega0;
}

template <class K>
void solve_config(K kern, const OneLaunch& o, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at) {
  *cfg = cudaLaunchConfig_t{};
  cfg->gridDim = dim3((unsigned)o.ctas);
  cfg->blockDim = dim3(kThreads);
  if (o.cluster) {
    if (o.ctas > 8) (void)cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = (unsigned)o.ctas;
    at->val.clusterDim.y = 1;
    at->val.clusterDim.z = 1;
  } else {
    at->id = cudaLaunchAttributeCooperative;
    at->val.cooperative = 1;
  }
  cfg->attrs = at;
  cfg->numAttrs = 1;
}

template <class K>
bool cluster_fits(K kern, const OneLaunch& o) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[1];
  solve_config(kern, o, &cfg, at);
  int most = 0;
  if (cudaOccupancyMaxActiveClusters(&most, kern, &cfg) == cudaSuccess) return most >= 1;
  (void)cudaGetLastError();
  return false;
}

template <class K, typename T>
int launch_solve(K kern, const OneLaunch& o, const SolveArgs<T>& A, cudaStream_t s) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[1];
  solve_config(kern, o, &cfg, at);
  cfg.stream = s;
  GIPB_CUDA(cudaLaunchKernelEx(&cfg, kern, A));
  return GIPB200_OK;
}

}  // namespace

int Pcg::plan_solve_launch(cudaStream_t s) {
  const bool mixed = prm.mode == GIPB200_PCG_MIXED, with_amg = prm.precond == GIPB200_PRECOND_AMG;
  // Where the lines lie (us per iteration, one launch against kernel by kernel, host-driven;
  // in the engine's graph the mixed AMG iteration took 75 at 63^3):
  //   mixed AMG    63^3 63 / 131, 75^3 73 / 150, 128^3 244 / 189 (dependent launches)
  //   FP64 AMG     33^3 35 / 94, 63^3 57 / 135, 128^3 275 / 368, 200^3 1004 / 1061
  //   mixed Jacobi 33^3 8 / 23, 75^3 11 / 28, 128^3 34 / 45, 160^3 73 / 66
  // The 16 warps of a resident CTA per SM gather slower than the 64 of the separate kernels, which
  // is what large systems are bound by: mixed AMG crosses between 75^3 and 128^3 and mixed Jacobi
  // between 128^3 and 160^3, sizes between them not measured; FP64 AMG is 5% ahead at 200^3 still,
  // and shares mixed Jacobi's line.
  const int most = mixed && with_amg ? 700000 : 2500000;
  if (n <= 0 || n > most || !L->rows_nonempty || getenv("GIPB200_NO_ONE_LAUNCH")) return GIPB200_OK;
  DeviceInfo di;
  GIPB_TRY(device_info(&di));
  // one cluster while its SMs' share of the rows costs less than the grid's barriers (mixed
  // AMG 12^3 19 against 29 us, 24^3 32 / 41, 33^3 46 / 41; mixed Jacobi 24^3 6.6 / 8.7)
  one.cluster = n <= 20000;
  one.ctas = one.cluster ? (n <= 4096 ? 8 : 16) : std::min(di.nsm, kGridCtasMax);
  if (one.cluster) {
    const bool fits = !mixed     ? cluster_fits(k_tol_amg_cluster, one)
                      : with_amg ? cluster_fits(k_mixed_cluster<true>, one)
                                 : cluster_fits(k_mixed_cluster<false>, one);
    if (!fits) {
      one.cluster = false;
      one.ctas = std::min(di.nsm, kGridCtasMax);
    }
  }
  const int warps = one.ctas * (kThreads / 32);
  size_t bytes = 0;
  std::vector<unsigned char> raw;
  if (mixed) {
    if (rec || (counted && !amg)) return GIPB200_OK;
    if (amg) {
      std::vector<CycleOp<float>> ops;
      if (!cycle_ops<float>(*amg, r32.p, warps, &ops)) return GIPB200_OK;
      one.nops = (int)ops.size();
      bytes = ops.size() * sizeof(ops[0]);
      raw.assign((unsigned char*)ops.data(), (unsigned char*)ops.data() + bytes);
    }
    GIPB_TRY(one.pair.alloc(((size_t)n + 1) / 2));
    if (pin_row >= 0) GIPB_TRY(one.rd.alloc((size_t)n + kMaxReduceBlocks));
  } else {
    if (!amg64 || prm.mode != GIPB200_PCG_TOL) return GIPB200_OK;
    std::vector<CycleOp<double>> ops;
    if (!cycle_ops<double>(*amg64, r.p, warps, &ops)) return GIPB200_OK;
    bool zero = true;
    GIPB_TRY(ghosts_zero(s, &zero));
    if (!zero) return GIPB200_OK;
    GIPB_TRY(build_packed64(s));
    if (counted) return GIPB200_OK;  // the loop reads the packed operator too
    one.nops = (int)ops.size();
    bytes = ops.size() * sizeof(ops[0]);
    raw.assign((unsigned char*)ops.data(), (unsigned char*)ops.data() + bytes);
    GIPB_TRY(one.pair.alloc((size_t)n));
  }
  if (bytes) GIPB_TRY(one.ops.upload(raw.data(), bytes, s));
  GIPB_CUDA(cudaStreamSynchronize(s));
  one.form = OneLaunch::kSolve;
  return one.slots.alloc(grid_slot_count(one.ctas));
}

namespace {
SolveArgs<float> mixed_args(Pcg& P, const double* b, const double* bp, double* x, const double* x0) {
  SolveArgs<float> A{};
  const PackedView pk = P.packed();
  A.op = {P.a32(), pk.delta, pk.idx, pk.base, pk.plain, pk.table, pk.slots, P.n};
  A.L = P.L->view();
  A.lidx = P.lpacked ? P.lidx4.p : nullptr;
  A.ltable = P.ltable.p;
  A.bp = bp;
  A.b = b;
  A.x0 = x0;
  A.x = x;
  A.scale = P.scale.p;
  A.pair = reinterpret_cast<float2*>(P.one.pair.p);
  A.r = P.r32.p;
  A.q = P.Ap32.p;
  A.y = P.y32.p;
  A.rd = P.one.rd.p;
  A.rpart = P.one.rd.p + P.n;
  A.vblocks = P.blocks_spmv;
  A.S = P.sc.p;
  A.gave_up = P.gave_up;
  A.slots = P.one.slots.p;
  A.ops = reinterpret_cast<const CycleOp<float>*>(P.one.ops.p);
  A.nops = P.one.nops;
  if (P.amg) cycle_args<float>(*P.amg, &A);
  A.tol = P.prm.tol;
  A.delta = P.prm.inner_tol;
  A.pin_val = P.pin_val;
  A.n = P.n;
  A.n_all = P.n_all;
  A.maxit = P.prm.maxit;
  A.max_outer = P.prm.max_outer;
  A.pin_row = P.pin_row;
  A.nib = pk.on ? pk.nib : 0;
  A.count = 1;
  return A;
}
}  // namespace

void Pcg::launch_wait_check(bool barrier_only, ulonglong2* slots, cudaStream_t s) {
  SolveArgs<float> A{};
  A.pin_row = -1;
  A.S = sc.p;
  A.gave_up = gave_up;
  A.slots = slots;
  A.maxit = A.max_outer = 1;
  k_mixed_wait_check<<<1, kThreads, 0, s>>>(A, barrier_only ? 1 : 0);
}

int Pcg::enqueue_solve_launch(const double* b, double* x, const double* x0, cudaStream_t s) {
  if (!one.cluster)
    GIPB_CUDA(cudaMemsetAsync(one.slots.p, 0, one.slots.n * sizeof(ulonglong2), s));
  launches += 1;
  if (prm.mode == GIPB200_PCG_MIXED) {
    const double* bp = b;
    if (lpacked) GIPB_TRY(enqueue_ghost_rhs(b, x0, s, &bp));
    const SolveArgs<float> A = mixed_args(*this, b, bp, x, x0);
    if (one.cluster)
      return amg ? launch_solve(k_mixed_cluster<true>, one, A, s)
                 : launch_solve(k_mixed_cluster<false>, one, A, s);
    return amg ? launch_solve(k_mixed_grid<true>, one, A, s)
               : launch_solve(k_mixed_grid<false>, one, A, s);
  }
  SolveArgs<double> A{};
  const Packed64& o = op64;
  A.op = {L->view(), o.delta.p, o.bits == 4 ? (const void*)o.idx4.p : (const void*)o.idx8.p,
          o.base.p,  o.plain.p, o.table.p, o.slots, n};
  A.L = L->view();
  A.b = b;
  A.x0 = x0;
  A.x = x;
  A.pair = one.pair.p;
  A.r = r.p;
  A.q = Ap.p;
  A.S = sc.p;
  A.gave_up = gave_up;
  A.slots = one.slots.p;
  A.ops = reinterpret_cast<const CycleOp<double>*>(one.ops.p);
  A.nops = one.nops;
  cycle_args<double>(*amg64, &A);
  A.tol = prm.tol;
  A.n = n;
  A.n_all = n_all;
  A.maxit = prm.maxit;
  A.pin_row = -1;
  A.nib = o.bits;
  return one.cluster ? launch_solve(k_tol_amg_cluster, one, A, s)
                     : launch_solve(k_tol_amg_grid, one, A, s);
}

// ------------------------------------------------------------------ small levels
template <typename T>
int plan_small_levels(AmgT<T>& M, cudaStream_t s) {
  M.small_from = -1;
  const int L = (int)M.lv.size();
  if (L < 3 || M.nc <= 0 || getenv("GIPB200_NO_ONE_LAUNCH")) return GIPB200_OK;
  // Levels whose operator streams at most 1 MB: 16 SMs read a larger one slower than the whole
  // GPU.  Restart, steps and reads in ms by largest operator, none / 0.3 / 1 / 2 / 4 / 16 MB: 12
  // cavities of 24..64 edges 10.3 / 10.0 / 10.0 / 10.1 / 10.2 / 10.5, 100^3 19.7 / 19.6 / 18.9 /
  // 18.8 / 18.6 / 18.8, 160^3 28.0 / 28.0 / 28.0 / 28.0 / 28.8 / 28.7; a cluster of 8 is slower
  // (19.3 at 100^3).
  constexpr double most = 1e6;
  int t = L - 1;
  while (t - 1 >= 1 && stream_bytes(M.lv[t - 1]->A) <= most) --t;
  if (t > L - 2) return GIPB200_OK;
  OneLaunch o;
  o.cluster = true;
  o.ctas = ClusterTeam::kMaxCtas;
  if (!cluster_fits(k_amg_small<T>, o)) return GIPB200_OK;
  std::vector<CycleOp<T>> ops;
  if (!cycle_ops<T>(M, (const T*)nullptr, o.ctas * (kThreads / 32), &ops)) return GIPB200_OK;
  const int first = 2 * t - 1, count = (int)ops.size() - 2 * first;
  const int st = M.small_ops.upload(reinterpret_cast<const unsigned char*>(ops.data() + first),
                                    count * sizeof(CycleOp<T>), s);
  if (st == GIPB200_ERR_NOMEM) return GIPB200_OK;  // without this launch, a kernel per product
  GIPB_TRY(st);
  GIPB_CUDA(cudaStreamSynchronize(s));
  const double w = sizeof(T), nc = M.nc;
  M.small_bytes = (nc * nc + 2.0 * nc) * w;
  for (int l = t; l < L - 1; ++l) {  // residual, restriction, prolongation, smoothing
    const AmgLevel<T>& V = *M.lv[l];
    const double n = V.n, nn = M.lv[l + 1]->n;
    M.small_bytes += 2.0 * stream_bytes(V.A) + stream_bytes(V.R) + stream_bytes(V.P) +
                     (11.0 * n + 2.0 * nn) * w;
  }
  M.small_nops = count;
  M.small_ctas = o.ctas;
  M.small_from = t;
  return GIPB200_OK;
}

template <typename T>
int launch_small_levels(const AmgT<T>& M, PcgScalars* S, cudaStream_t s) {
  OneLaunch o;
  o.cluster = true;
  o.ctas = M.small_ctas;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  solve_config(k_amg_small<T>, o, &cfg, at);
  if (dependent_launches(s)) {
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
  }
  cfg.stream = s;
  GIPB_CUDA(cudaLaunchKernelEx(&cfg, k_amg_small<T>, reinterpret_cast<const CycleOp<T>*>(M.small_ops.p),
                               M.small_nops, S));
  return GIPB200_OK;
}
template int plan_small_levels(AmgT<float>&, cudaStream_t);
template int plan_small_levels(AmgT<double>&, cudaStream_t);
template int launch_small_levels(const AmgT<float>&, PcgScalars*, cudaStream_t);
template int launch_small_levels(const AmgT<double>&, PcgScalars*, cudaStream_t);

// ------------------------------------------------------------------ groups
int SolveGroups::plan(const std::vector<Pcg*>& solvers, const std::vector<const double*>& b,
                      const std::vector<double*>& x, const std::vector<const double*>& x0,
                      cudaStream_t s) {
  on = false;
  const int ni = (int)solvers.size();
  DeviceInfo di;
  GIPB_TRY(device_info(&di));
  ctas = std::min(di.nsm, kGridCtasMax);
  if (ni > ctas) return GIPB200_OK;
  double rows = 0.0;
  for (const Pcg* P : solvers) {
    if (P->prm.mode != GIPB200_PCG_MIXED || !P->amg || P->one.form != OneLaunch::kSolve)
      return GIPB200_OK;
    rows += P->n;
  }
  // Batches of small systems, or a small batch: the branches' kernels reach a higher rate once
  // they fill the chip.  Measured per step, branches / groups: 3 of 12..20 edges 0.63 / 0.46
  // ms, 8 of 20..30 1.4 / 1.0, 32 of 16..48 (37k rows on average) 6.0 / 4.2, 2 of 44 1.08 /
  // 0.82; 12 of 24..64 (103k) 3.8 / 3.7, 16 of 32..64 (120k) 4.5 / 5.2, 6 of 64..77 4.1 / 6.0.
  if (rows > 600000.0 && rows > 60000.0 * ni) return GIPB200_OK;
  // CTAs by rows (the instances' iteration counts are close with AMG): at least one each
  std::vector<int> share(ni);
  int used = 0;
  for (int i = 0; i < ni; ++i) {
    share[i] = std::max(1, (int)((double)ctas * solvers[i]->n / rows));
    used += share[i];
  }
  for (; used > ctas; --used) *std::max_element(share.begin(), share.end()) -= 1;
  for (; used < ctas; ++used) {  // the rest to the instances with the most rows per CTA
    int k = 0;
    for (int i = 1; i < ni; ++i)
      if ((double)solvers[i]->n * share[k] > (double)solvers[k]->n * share[i]) k = i;
    share[k] += 1;
  }
  size_t need = 0;
  for (int i = 0; i < ni; ++i) need += grid_slot_count(share[i]);
  GIPB_TRY(slots.alloc(need));
  std::vector<GroupSolve> h(ni);
  std::vector<int> own(ctas, -1);
  size_t at = 0;
  int c = 0;
  for (int i = 0; i < ni; ++i) {
    Pcg& P = *solvers[i];
    const bool ghosts = P.lpacked && !P.ghost_rows.empty();
    h[i].A = mixed_args(P, b[i], ghosts ? P.bprime.p : b[i], x[i], x0[i]);
    h[i].A.slots = slots.p + at;
    h[i].A.count = i == 0 ? 1 : 0;
    h[i].cta0 = c;
    h[i].ncta = share[i];
    for (int k = 0; k < share[i]; ++k) own[c + k] = i;
    c += share[i];
    at += grid_slot_count(share[i]);
  }
  GIPB_TRY(items.upload(reinterpret_cast<const unsigned char*>(h.data()), ni * sizeof(GroupSolve), s));
  GIPB_TRY(owner.upload(own.data(), own.size(), s));
  GIPB_CUDA(cudaStreamSynchronize(s));
  on = true;
  return GIPB200_OK;
}

int SolveGroups::launch(cudaStream_t s) const {
  GIPB_CUDA(cudaMemsetAsync(slots.p, 0, slots.n * sizeof(ulonglong2), s));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  GIPB_CUDA(cudaLaunchKernelEx(&cfg, k_mixed_groups, reinterpret_cast<const GroupSolve*>(items.p),
                               (const int*)owner.p));
  return GIPB200_OK;
}

}  // namespace gipb200
