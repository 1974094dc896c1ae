// FP64 Jacobi-PCG (GIP_LinearSolver::solve, src/Algorithms/GIP_LinearSolver.h:44-117) as one
// launch.
//
// The three-kernel loop of pcg.cu spends a launch, a drain and a ticket reduction per kernel:
// 4.1 us each on the 12^3 cavity, whose work is a fraction of a microsecond.  Here the whole
// solve is one kernel whose CTAs stay resident, and an iteration is
//   A: Ap = L p with p_j = z_j + beta p_j formed where it is gathered (the IEEE operations
//      of the separate update, so the same values)                       -> p.Ap, alpha
//   B: x += alpha p, r -= alpha Ap, z = dinv r, (z, p) published           -> r.z, r.r, beta
// with two reductions over all CTAs and no other barrier.  Every row belongs to one thread
// for the whole solve, which keeps x, r, p, dinv and the row's operator in registers; only
// the pair (z, p) of a row is ever written, for the threads that gather it.
//   block form: up to 1920 rows (480 threads, 4 rows each), one CTA; below;
//   cluster form: up to 16384 rows (16 CTAs of 256 threads, 4 rows each), the pairs in the
//     cluster's shared memory, the reductions over hardware cluster barriers;
//   grid form: up to 4 rows per thread of 256 on every SM (151552 rows on 148 SMs), the pairs
//     in global memory (L2), the reductions over epoch-stamped slots (persist.cuh);
//   streamed form: more rows, while r and Ap fit the SMs' shared memory (2.1 million rows on
//     148 SMs), for operators that pack; below.
// Measured per iteration against the three-kernel loop inside a step graph (host-driven it
// took 20 us or more): 8^3 1.4 (block; cluster 2.0), 12^3 2.5 against 12.2 us (block; cluster
// of 4 2.7; grid 4.9), 24^3 4.2 (cluster of 16; grid 5.2), 48^3 6.0 against 16.7 (streamed 9.1), 64^3 10.6 against 23
// (host-driven), 128^3 32.5 against 84.
// Element operations are GIP's (no FMA contraction); only the order of the dot products' sums
// differs from the other forms.  Columns of ghost cells hold stored zeros in these operators
// (checked at set-up; a later change of the values ends these forms, Pcg::follow_values): they
// enter the initial residual like every column, and the iterations, where their entries of p
// stay fixed, drop them.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

#include "persist.cuh"

namespace gipb200 {
namespace {

constexpr int kRowSlots = 8;  // longest row of the register forms

struct Args64 {
  SellView<double> L;
  const double* b;
  const double* x0;
  const double* dinv;
  double* x;
  double2* pair;      // grid form: (z, p) of every row
  ulonglong2* slots;  // grid forms: reduction slots (zero at launch)
  PcgScalars* S;
  int* gave_up;       // host flag: a wait gave up
  double tol;
  int n, n_all, mode, maxit;
};

// The solve's scalars, held identically by every thread.
struct Scal64 {
  double rz, pAp, alpha, beta, rr, bb;
  double goal;  // tol sqrt(b.b), what sqrt(r.r) is compared with
  int iter, done, status;
};

// After the initial residual (PcgInitFinish of the three-kernel loop).
__device__ __forceinline__ void start64(Scal64& T, const double (&t)[3], int mode, int maxit,
                                        double tol) {
  T.rz = t[0];
  T.rr = t[1];
  T.bb = t[2];
  T.pAp = T.alpha = T.beta = 0.0;
  T.iter = 0;
  T.status = GIPB200_OK;
  T.done = (maxit <= 0) ? 1 : 0;
  T.goal = mode == GIPB200_PCG_TOL ? tol * sqrt(t[2]) : 0.0;
  if (mode == GIPB200_PCG_TOL && !(sqrt(t[1]) > T.goal)) T.done = 1;
  if (mode != GIPB200_PCG_FIXED && !(isfinite(t[1]) && isfinite(t[2]))) {
    T.status = GIPB200_ERR_BREAKDOWN;
    T.done = 1;
  }
}

// After p.Ap; false: breakdown, the iteration ends before its update.
__device__ __forceinline__ bool alpha64(Scal64& T, double pAp, int mode) {
  T.pAp = pAp;
  T.alpha = ddiv(T.rz, pAp);
  if (mode != GIPB200_PCG_FIXED && (!(pAp > 0.0) || !isfinite(T.alpha))) {
    T.status = GIPB200_ERR_BREAKDOWN;
    T.done = 1;
    return false;
  }
  return true;
}

// After r.z and r.r.
__device__ __forceinline__ void beta64(Scal64& T, const double (&t)[2], int mode, int maxit) {
  const double r0 = T.rz;
  T.rz = t[0];
  T.rr = t[1];
  T.beta = ddiv(t[0], r0);
  T.iter += 1;
  if (mode == GIPB200_PCG_TOL && !(sqrt(t[1]) > T.goal)) T.done = 1;
  if (T.iter >= maxit) {
    if (mode == GIPB200_PCG_TOL && !T.done) T.status = GIPB200_ERR_NOT_CONVERGED;
    T.done = 1;
  }
}

__device__ __forceinline__ void store64(PcgScalars* S, const Scal64& T) {
  S->rz = T.rz;
  S->pAp = T.pAp;
  S->alpha = T.alpha;
  S->beta = T.beta;
  S->rr = T.rr;
  S->bb = T.bb;
  S->iter = T.iter;
  S->done = 1;
  S->status = T.status;
  S->kernels = 0;
  S->one_launch = 1;
}

// The end of a solve over several CTAs (one thread of each).
__device__ __forceinline__ void finish64(const Args64& A, Scal64& T, int rank, bool ok) {
  if (!ok) {
    T.status = GIPB200_ERR_TIMEOUT;
    report_gave_up(A.gave_up);
  }
  if (rank == 0) store64(A.S, T);
}

// ------------------------------------------------------------------ register forms
// Where a row's (z, p) pair lives and how the sums travel.
struct ClusterPairs {
  static constexpr int kMaxCtas = 16;
  unsigned rank, size;
  int rows;                  // rows of one CTA
  unsigned pairs;            // shared address of this CTA's pairs
  double (*red)[3][8 * kMaxCtas];  // [parity][sum][warp of the cluster]
  int par = 0;
  __device__ __forceinline__ unsigned where(int row) const {
    return map_shared(pairs + 16u * (unsigned)(row % rows), (unsigned)(row / rows));
  }
  __device__ __forceinline__ double2 load(unsigned a) const {
    double2 v;
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
    return v;
  }
  __device__ __forceinline__ void publish(int row, double z, double p) const {
    asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(pairs + 16u * (unsigned)(row - (int)rank * rows)),
                 "d"(z), "d"(p)
                 : "memory");
  }
  // Each warp sends its partial sums to every CTA; after one barrier every warp adds all of
  // them in the same order.  The barrier also publishes the pairs.
  template <int W, bool FENCE>
  __device__ __forceinline__ bool sum(double (&v)[W]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < W; ++k) {
      const double t = warp_reduce<SumOp>(v[k]);
      if (lane < (int)size)
        st_cluster(map_shared(smem_u32(&red[par][k][rank * nw + warp]), (unsigned)lane), t);
    }
    cluster_barrier();
    const int total = nw * (int)size;
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

struct GridPairs {
  double2* pairs;
  GridScope G;
  __device__ __forceinline__ int where(int row) const { return row; }
  // plain loads: the reduction that published the pairs is an acquire for the whole CTA
  __device__ __forceinline__ double2 load(int row) const { return pairs[row]; }
  __device__ __forceinline__ void publish(int row, double z, double p) const {
    pairs[row] = make_double2(z, p);
  }
  template <int W, bool FENCE>
  __device__ __forceinline__ bool sum(double (&v)[W]) {
    return grid_sum<W, FENCE>(v, G);
  }
};

// K rows per thread: rows first + k * blockDim.x + threadIdx.x of the CTA's K * blockDim.x.
template <int K, class Pairs>
__device__ __forceinline__ void solve_rows(const Args64& A, Pairs& Q, int rank, int ncta) {
  using Addr = decltype(Q.where(0));
  const int lane = threadIdx.x & 31;
  const int i0 = rank * K * (int)blockDim.x + (int)threadIdx.x;
  // the rows' operator and the initial residual r = b - L x0, z = dinv r, p = z
  Addr at[K][kRowSlots];
  double v[K][kRowSlots];
  double x[K], r[K], z[K], p[K], q[K], di[K];
  double acc3[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int i = i0 + k * (int)blockDim.x;
    const bool own = i < A.n;
    long long base = 0;
    int len = 0;
    const int s = i >> 5;
    if (s < A.L.nslices) slice_range(A.L, s, base, len);
    double sum = 0.0;
#pragma unroll
    for (int j = 0; j < kRowSlots; ++j) {
      const int c = (j < len) ? A.L.col[base + 32LL * j + lane] : -1;
      v[k][j] = (c >= 0) ? A.L.val[base + 32LL * j + lane] : 0.0;
      if (c >= 0) sum = dadd(sum, dmul(A.x0[c], v[k][j]));
      // padding and ghost columns: the row's own pair times a zero
      at[k][j] = Q.where((c >= 0 && c < A.n) ? c : (own ? i : 0));
    }
    x[k] = r[k] = z[k] = p[k] = q[k] = di[k] = 0.0;
    if (own) {
      const double bi = A.b[i];
      x[k] = A.x0[i];
      di[k] = A.dinv[i];
      r[k] = dadd(bi, dmul(-1.0, sum));
      z[k] = dadd(0.0, dmul(r[k], di[k]));
      acc3[0] = dadd(acc3[0], dmul(r[k], z[k]));
      acc3[1] = dadd(acc3[1], dmul(r[k], r[k]));
      acc3[2] = dadd(acc3[2], dmul(bi, bi));
      Q.publish(i, z[k], 0.0);
    }
  }
  Scal64 T;
  bool ok = Q.template sum<3, true>(acc3);
  start64(T, acc3, A.mode, A.maxit, A.tol);
  if (A.x != A.x0)  // (after the reduction: every row has read x0)
    for (int g = A.n + rank * (int)blockDim.x + (int)threadIdx.x; g < A.n_all;
         g += ncta * (int)blockDim.x)
      A.x[g] = A.x0[g];
  while (ok && !T.done) {
    double d[1] = {0.0};
#pragma unroll
    for (int k = 0; k < K; ++k) {
      double2 zp[kRowSlots];
#pragma unroll
      for (int j = 0; j < kRowSlots; ++j) zp[j] = Q.load(at[k][j]);
      double sum = 0.0;
#pragma unroll
      for (int j = 0; j < kRowSlots; ++j)
        sum = dadd(sum, dmul(dadd(zp[j].x, dmul(T.beta, zp[j].y)), v[k][j]));
      q[k] = sum;
      p[k] = dadd(z[k], dmul(T.beta, p[k]));
      d[0] = dadd(d[0], dmul(p[k], q[k]));  // (a thread without a row adds zeros)
    }
    if (!(ok = Q.template sum<1, false>(d))) break;
    if (!alpha64(T, d[0], A.mode)) break;
    double e[2] = {0.0, 0.0};
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = i0 + k * (int)blockDim.x;
      r[k] = dadd(r[k], dmul(dmul(-1.0, T.alpha), q[k]));
      z[k] = dadd(0.0, dmul(r[k], di[k]));
      if (i < A.n) Q.publish(i, z[k], p[k]);
      e[0] = dadd(e[0], dmul(r[k], z[k]));
      e[1] = dadd(e[1], dmul(r[k], r[k]));
      x[k] = dadd(x[k], dmul(T.alpha, p[k]));
    }
    if (!(ok = Q.template sum<2, true>(e))) break;
    beta64(T, e, A.mode, A.maxit);
  }
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (i0 + k * (int)blockDim.x < A.n) A.x[i0 + k * (int)blockDim.x] = x[k];
  if (threadIdx.x == 0) finish64(A, T, rank, ok);
}

constexpr int kRegThreads = 256;  // CTA size of the register forms

// Bound by latency: per iteration the gathers, the warp reductions and two cluster barriers.
template <int K>
__global__ void __launch_bounds__(kRegThreads, 1) k_pcg64_cluster(const __grid_constant__ Args64 A) {
  __shared__ __align__(16) double2 pairs[K * kRegThreads];
  __shared__ double red[2][3][8 * ClusterPairs::kMaxCtas];
  ClusterPairs Q;
  Q.rank = cluster_rank();
  Q.size = cluster_size();
  Q.rows = K * (int)blockDim.x;
  Q.pairs = smem_u32(pairs);
  Q.red = red;
  cluster_barrier();  // every CTA runs before its shared memory is written
  solve_rows<K>(A, Q, (int)Q.rank, (int)Q.size);
  cluster_barrier();  // no CTA leaves while another may still read its pairs
}

template <int K>
__global__ void __launch_bounds__(kRegThreads, 1) k_pcg64_grid(const __grid_constant__ Args64 A) {
  GridPairs Q;
  Q.pairs = A.pair;
  Q.G = grid_begin(A.slots);
  solve_rows<K>(A, Q, (int)blockIdx.x, (int)gridDim.x);
}

// One CTA of a group that claims two and has no rows: its first sum waits for a CTA that does
// not exist and gives up.
__global__ void __launch_bounds__(kRegThreads, 1) k_pcg64_wait_check(const __grid_constant__ Args64 A) {
  GridPairs Q;
  Q.pairs = A.pair;
  Q.G = grid_begin(A.slots, 0, 2, kCheckSpinCycles);
  solve_rows<1>(A, Q, 0, 1);
}

// ------------------------------------------------------------------ block form
// Small systems in one CTA: p in shared memory, a row's operator in its thread's registers
// (columns as 16-bit rows), no cluster barriers (370 cycles each) and no remote gathers, at the
// price of one more block barrier (30 to 60 cycles), between the update of p and its gathers.
// Few warps with up to four rows a thread: the shuffles of the reductions, an instruction a
// cycle for the whole SM, would bound a CTA of 1024 threads.  One thread keeps the scalars.
constexpr int kBlockThreads = 480;  // 128 registers a thread, 48 KB for four rows each

// Sums over the CTA; the first thread of the CTA receives them (finish), before a barrier.
template <int W, class F>
__device__ __forceinline__ void block_sum(double (&v)[W], double (*part)[kBlockThreads / 32], F finish) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < W; ++k) {
    const double t = warp_reduce<SumOp>(v[k]);
    if (lane == 0) part[k][warp] = t;
  }
  __syncthreads();
  if (warp == 0) {
    double t[W];
#pragma unroll
    for (int k = 0; k < W; ++k) t[k] = warp_reduce<SumOp>(lane < nw ? part[k][lane] : 0.0);
    if (lane == 0) finish(t);
  }
  __syncthreads();
}

// K rows per thread of at most SLOTS entries.
template <int K, int SLOTS>
__global__ void __launch_bounds__(kBlockThreads, 1) k_pcg64_block(const __grid_constant__ Args64 A) {
  constexpr bool kLean = K > 2;  // x and dinv in shared memory: registers
  __shared__ double sp[K * kBlockThreads];
  __shared__ double sx[kLean ? K * kBlockThreads : 1], sd[kLean ? K * kBlockThreads : 1];
  __shared__ double part[3][kBlockThreads / 32];
  __shared__ Scal64 T;
  const int lane = threadIdx.x & 31, nt = blockDim.x;
  unsigned at[K][(SLOTS + 1) / 2];  // two columns a word
  double v[K][SLOTS];
  double xr[kLean ? 1 : K], dr[kLean ? 1 : K], r[K], z[K], p[K], q[K];
  auto X = [&](int k) -> double& { return kLean ? sx[k * nt + (int)threadIdx.x] : xr[kLean ? 0 : k]; };
  auto D = [&](int k) -> double& { return kLean ? sd[k * nt + (int)threadIdx.x] : dr[kLean ? 0 : k]; };
  double acc3[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int i = k * nt + (int)threadIdx.x;
    const bool own = i < A.n;
    long long base = 0;
    int len = 0;
    const int s = i >> 5;
    if (s < A.L.nslices) slice_range(A.L, s, base, len);
    double sum = 0.0;
#pragma unroll
    for (int j = 0; j < (SLOTS + 1) / 2; ++j) at[k][j] = 0u;
#pragma unroll
    for (int j = 0; j < SLOTS; ++j) {
      const int c = (j < len) ? A.L.col[base + 32LL * j + lane] : -1;
      v[k][j] = (c >= 0) ? A.L.val[base + 32LL * j + lane] : 0.0;
      if (c >= 0) sum = dadd(sum, dmul(A.x0[c], v[k][j]));
      // padding and ghost columns: the row's own p times a zero
      at[k][j / 2] |= (unsigned)((c >= 0 && c < A.n) ? c : (own ? i : 0)) << (16 * (j & 1));
    }
    r[k] = z[k] = p[k] = q[k] = 0.0;
    X(k) = 0.0;
    D(k) = 0.0;
    if (own) {
      const double bi = A.b[i];
      X(k) = A.x0[i];
      D(k) = A.dinv[i];
      r[k] = dadd(bi, dmul(-1.0, sum));
      z[k] = dadd(0.0, dmul(r[k], D(k)));
      acc3[0] = dadd(acc3[0], dmul(r[k], z[k]));
      acc3[1] = dadd(acc3[1], dmul(r[k], r[k]));
      acc3[2] = dadd(acc3[2], dmul(bi, bi));
    }
  }
  block_sum(acc3, part, [&](const double (&t)[3]) { start64(T, t, A.mode, A.maxit, A.tol); });
  if (A.x != A.x0)  // (after the reduction: every row has read x0)
    for (int g = A.n + (int)threadIdx.x; g < A.n_all; g += nt) A.x[g] = A.x0[g];
  while (!T.done) {
    const double beta = T.beta;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      p[k] = dadd(z[k], dmul(beta, p[k]));
      sp[k * nt + (int)threadIdx.x] = p[k];
    }
    __syncthreads();
    double d[1] = {0.0};
#pragma unroll
    for (int k = 0; k < K; ++k) {
      double pv[SLOTS];
#pragma unroll
      for (int j = 0; j < SLOTS; ++j) pv[j] = sp[(at[k][j / 2] >> (16 * (j & 1))) & 0xffffu];
      double sum = 0.0;
#pragma unroll
      for (int j = 0; j < SLOTS; ++j) sum = dadd(sum, dmul(pv[j], v[k][j]));
      q[k] = sum;
      d[0] = dadd(d[0], dmul(p[k], q[k]));  // (a thread without a row adds zeros)
    }
    block_sum(d, part, [&](const double (&t)[1]) { alpha64(T, t[0], A.mode); });
    if (T.done) break;  // breakdown
    const double alpha = T.alpha, malpha = dmul(-1.0, alpha);
    double e[2] = {0.0, 0.0};
#pragma unroll
    for (int k = 0; k < K; ++k) {
      r[k] = dadd(r[k], dmul(malpha, q[k]));
      z[k] = dadd(0.0, dmul(r[k], D(k)));
      e[0] = dadd(e[0], dmul(r[k], z[k]));
      e[1] = dadd(e[1], dmul(r[k], r[k]));
      X(k) = dadd(X(k), dmul(alpha, p[k]));
    }
    block_sum(e, part, [&](const double (&t)[2]) { beta64(T, t, A.mode, A.maxit); });
  }
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (k * nt + (int)threadIdx.x < A.n) A.x[k * nt + (int)threadIdx.x] = X(k);
  if (threadIdx.x == 0) store64(A.S, T);
}

// ------------------------------------------------------------------ streamed form
// Several rows per thread: a CTA owns a contiguous range of slices; r and Ap (then z) of its
// rows stay in shared memory, p, x and dinv in global memory, and the operator streams from
// its packed layout (21 bytes a row) each iteration.  x += alpha p waits for the pass that
// forms the next p, which reads p anyway.
struct Stream64 {
  const uint4* delta;
  const void* idx;
  const int* base;
  const unsigned char* plain;
  const double* table;
  double* p;   // n_all entries, ghosts as x0 has them
};

// Operator words are read every iteration and meant to stay in L2.
__device__ __forceinline__ uint4 ld_words(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ unsigned ld_word(const unsigned* p) {
  unsigned v;
  asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 ld_word2(const uint2* p) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}

template <int NIB>
__device__ __forceinline__ void words64(const Stream64& M, int s, int lane, PackedWords& w) {
  const int i = s * 32 + lane;
  w.plain = __ldg(M.plain + s);
  w.d = ld_words(M.delta + i);
  if (NIB == 4) {
    w.w0 = ld_word(static_cast<const unsigned*>(M.idx) + i);
    w.w1 = 0u;
  } else {
    const uint2 t = ld_word2(static_cast<const uint2*>(M.idx) + i);
    w.w0 = t.x;
    w.w1 = t.y;
  }
}

// sum of row i of a sliced slice with plain loads of x (written inside the launch)
__device__ __forceinline__ double row_plain(const SellView<double>& L, const double* x, int s,
                                            int lane) {
  long long base;
  int len;
  slice_range(L, s, base, len);
  double sum = 0.0;
  for (int j = 0; j < len; ++j) {
    const int c = L.col[base + 32LL * j + lane];
    if (c >= 0) sum = dadd(sum, dmul(x[c], L.val[base + 32LL * j + lane]));
  }
  return sum;
}

template <int NIB>
__global__ void __launch_bounds__(1024, 1) k_pcg64_stream(const __grid_constant__ Args64 A,
                                                          const __grid_constant__ Stream64 M) {
  extern __shared__ __align__(16) double onchip[];
  __shared__ double tab[NIB == 4 ? 16 : 256];
  for (int t = threadIdx.x; t < (NIB == 4 ? 16 : 256); t += blockDim.x) tab[t] = M.table[t];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int rank = blockIdx.x, ncta = gridDim.x;
  const int ns = A.L.nslices;
  const int s0 = (int)((long long)ns * rank / ncta), s1 = (int)((long long)ns * (rank + 1) / ncta);
  const int first = s0 * 32, rows = min(A.n, s1 * 32) - first;  // this CTA's rows
  double* sr = onchip;                       // r
  double* sq = onchip + (size_t)(s1 - s0) * 32;  // A p, then z
  double* p = M.p;
  GridScope G = grid_begin(A.slots);
  double acc3[3] = {0.0, 0.0, 0.0};
  for (int s = s0 + warp; s < s1; s += nw) {
    const int i = s * 32 + lane;
    const double sum = row_plain(A.L, A.x0, s, lane);
    if (i < A.n) {
      const double bi = A.b[i];
      const double ri = dadd(bi, dmul(-1.0, sum));
      const double zi = dadd(0.0, dmul(ri, A.dinv[i]));
      sr[i - first] = ri;
      p[i] = zi;
      acc3[0] = dadd(acc3[0], dmul(ri, zi));
      acc3[1] = dadd(acc3[1], dmul(ri, ri));
      acc3[2] = dadd(acc3[2], dmul(bi, bi));
    }
  }
  for (int g = A.n + rank * (int)blockDim.x + (int)threadIdx.x; g < A.n_all;
       g += ncta * (int)blockDim.x)
    p[g] = A.x0[g];
  Scal64 T;
  bool ok = grid_sum<3, true>(acc3, G);
  start64(T, acc3, A.mode, A.maxit, A.tol);
  if (A.x != A.x0) {  // (after the reduction: every row has read x0)
    for (int k = threadIdx.x; k < rows; k += blockDim.x) A.x[first + k] = A.x0[first + k];
    for (int g = A.n + rank * (int)blockDim.x + (int)threadIdx.x; g < A.n_all;
         g += ncta * (int)blockDim.x)
      A.x[g] = A.x0[g];
  }
  while (ok && !T.done) {
    // A: Ap = L p, p.Ap
    double d[1] = {0.0};
    PackedWords w;
    if (s0 + warp < s1) words64<NIB>(M, s0 + warp, lane, w);
    for (int s = s0 + warp; s < s1; s += nw) {
      const int i = s * 32 + lane;
      PackedWords nx;
      if (s + nw < s1) words64<NIB>(M, s + nw, lane, nx);
      double sum = 0.0;
      if (w.plain) {
        sum = row_plain(A.L, p, s, lane);
      } else {
        int c[8];
        packed_cols(M.base, s, w.d, c);
        double xv[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) xv[j] = p[c[j]];
#pragma unroll
        for (int j = 0; j < 8; ++j) sum = dadd(sum, dmul(xv[j], tab[packed_index<NIB>(w, j)]));
      }
      if (i < A.n) {
        sq[i - first] = sum;
        d[0] = dadd(d[0], dmul(p[i], sum));
      }
      w = nx;
    }
    if (!(ok = grid_sum<1, false>(d, G))) break;
    if (!alpha64(T, d[0], A.mode)) break;
    // B: r -= alpha Ap, z = dinv r (over Ap), r.z, r.r
    const double malpha = dmul(-1.0, T.alpha);
    double e[2] = {0.0, 0.0};
#pragma unroll 4
    for (int k = threadIdx.x; k < rows; k += 1024) {
      const double ri = dadd(sr[k], dmul(malpha, sq[k]));
      const double zi = dadd(0.0, dmul(ri, __ldg(A.dinv + first + k)));
      sr[k] = ri;
      sq[k] = zi;
      e[0] = dadd(e[0], dmul(ri, zi));
      e[1] = dadd(e[1], dmul(ri, ri));
    }
    if (!(ok = grid_sum<2, false>(e, G))) break;
    beta64(T, e, A.mode, A.maxit);
    // C: x += alpha p; p = z + beta p (not after the last iteration)
    if (T.done) {
#pragma unroll 4
      for (int k = threadIdx.x; k < rows; k += 1024)
        A.x[first + k] = dadd(A.x[first + k], dmul(T.alpha, p[first + k]));
      break;
    }
#pragma unroll 4
    for (int k = threadIdx.x; k < rows; k += 1024) {
      const double pk = p[first + k];
      A.x[first + k] = dadd(A.x[first + k], dmul(T.alpha, pk));
      p[first + k] = dadd(sq[k], dmul(T.beta, pk));
    }
    double none[1] = {0.0};
    ok = grid_sum<1, true>(none, G);
  }
  if (threadIdx.x == 0) finish64(A, T, rank, ok);
}

struct AlphaFinish64 {
  PcgScalars* S;
  int mode;
  __device__ void operator()(const double* t) const {
    S->pAp = t[0];
    S->alpha = ddiv(S->rz, t[0]);
    if (mode != GIPB200_PCG_FIXED && (!(t[0] > 0.0) || !isfinite(S->alpha))) {
      S->status = GIPB200_ERR_BREAKDOWN;
      S->done = 1;
    }
  }
};

// Ap = L p and p.Ap of the three-kernel loop (grids whose r and Ap do not fit on chip) from
// the packed layout: 37 bytes a row instead of 100.
template <int NIB>
__global__ void __launch_bounds__(256, 8) k_pcg64_spmv_dot(SellView<double> L, Stream64 M,
                                                           double* __restrict__ Ap, PcgScalars* S,
                                                           ReduceScratch rs, int mode) {
  if (S->done) return;
  __shared__ double tab[NIB == 4 ? 16 : 256];
  for (int t = threadIdx.x; t < (NIB == 4 ? 16 : 256); t += blockDim.x) tab[t] = M.table[t];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  const double* __restrict__ p = M.p;
  double acc[1] = {0.0};
  for (int s = gw; s < L.nslices; s += nw) {
    PackedWords w;
    packed_words<NIB>(M.delta, M.idx, M.plain, s, lane, w);
    const int i = s * 32 + lane;
    double sum = 0.0;
    if (w.plain) {
      sum = row_plain(L, p, s, lane);
    } else {
      int c[8];
      packed_cols(M.base, s, w.d, c);
#pragma unroll
      for (int h = 0; h < 8; h += 4) {  // four gathers in flight at 32 registers
        double xv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) xv[j] = __ldg(p + c[h + j]);
#pragma unroll
        for (int j = 0; j < 4; ++j) sum = dadd(sum, dmul(xv[j], tab[packed_index<NIB>(w, h + j)]));
      }
    }
    if (i < L.nrows) {
      Ap[i] = sum;
      acc[0] = dadd(acc[0], dmul(p[i], sum));
    }
  }
  grid_reduce<SumOp, 1>(acc, rs, AlphaFinish64{S, mode});
}

}  // namespace

// ------------------------------------------------------------------ set-up
int Pcg::build_packed64(cudaStream_t s) { return pack64(*L, n, false, &op64, s); }

// L's values changed since they were looked at: the FP64 solves read them as they are now, as
// the kernel-by-kernel loop does.  What was made from the old ones lapses for good: the packed
// copy, and with ghost columns every form that drops them because they held zeros.  (The mixed
// form keeps its own copies of L's values, in one launch and kernel by kernel alike.)
void Pcg::follow_values() {
  if (prm.mode == GIPB200_PCG_MIXED || (L->version == planned_version && !L->values_in_graph)) return;
  if (op64.bits || n_all > n) one.form = OneLaunch::kNone;
  op64.bits = 0;
}

namespace {

size_t stream_shared(int nslices, int ncta) {
  return (size_t)((nslices + ncta - 1) / ncta) * 32 * 2 * sizeof(double);
}

template <class K>
bool stream_fits(K kern, size_t shared) {
  int dev = 0, most = 0;
  cudaFuncAttributes fa;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
      cudaFuncGetAttributes(&fa, kern) != cudaSuccess)
    return false;
  // the limit belongs to the kernel, not to this solver: always the device's, so that planning
  // one solver never lowers it below what another launches with
  const int limit = most - (int)fa.sharedSizeBytes;
  return shared <= (size_t)std::max(limit, 0) &&
         cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, limit) ==
             cudaSuccess;
}

template <class K>
void one_launch_attr(K kern, const OneLaunch& o, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at,
                     bool cluster) {
  *cfg = cudaLaunchConfig_t{};
  cfg->gridDim = dim3((unsigned)o.ctas);
  cfg->blockDim = dim3((unsigned)o.threads);
  cfg->dynamicSmemBytes = o.shared;
  if (cluster) {
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
  one_launch_attr(kern, o, &cfg, at, true);
  int most = 0;
  if (cudaOccupancyMaxActiveClusters(&most, kern, &cfg) == cudaSuccess) return most >= 1;
  (void)cudaGetLastError();
  return false;
}

}  // namespace

int Pcg::ghosts_zero(cudaStream_t s, bool* zero) const {
  *zero = true;
  if (n_all <= n) return GIPB200_OK;
  std::vector<double> hval((size_t)std::max(L->nnz, 1));
  GIPB_CUDA(cudaMemcpyAsync(hval.data(), L->csr_val.p, (size_t)L->nnz * 8, cudaMemcpyDeviceToHost, s));
  GIPB_CUDA(cudaStreamSynchronize(s));
  for (int k = 0; k < L->nnz && *zero; ++k) *zero = L->h_col[k] < n || hval[k] == 0.0;
  return GIPB200_OK;
}

void Pcg::join_batch() {
  in_batch = true;
  if (one.form == OneLaunch::kGrid || one.form == OneLaunch::kStream) one.release();
}

int Pcg::solve_form() {
  follow_values();
  if (!one_launch()) return GIPB200_SOLVE_LOOP;
  switch (one.form) {
    case OneLaunch::kBlock: return GIPB200_SOLVE_BLOCK;
    case OneLaunch::kCluster: return GIPB200_SOLVE_CLUSTER;
    case OneLaunch::kGrid: return GIPB200_SOLVE_GRID;
    case OneLaunch::kStream: return GIPB200_SOLVE_STREAM;
    default: return one.cluster ? GIPB200_SOLVE_PRECOND_CLUSTER : GIPB200_SOLVE_PRECOND_GRID;
  }
}

// A solver that found no memory for its one-launch form solves kernel by kernel.
int Pcg::plan_one_launch(cudaStream_t s) {
  one.release();
  planned_version = L->version;
  int st;
  try {
    st = choose_one_launch(s);
  } catch (const std::bad_alloc&) {
    st = GIPB200_ERR_NOMEM;
  }
  if (st == GIPB200_OK) return GIPB200_OK;
  one.release();
  return st == GIPB200_ERR_NOMEM ? GIPB200_OK : st;
}

// Which one-launch form runs this solver's solves.
int Pcg::choose_one_launch(cudaStream_t s) {
  if (prm.mode == GIPB200_PCG_MIXED || prm.precond != GIPB200_PRECOND_JACOBI)
    return plan_solve_launch(s);
  if (n <= 0 || !L->rows_nonempty || getenv("GIPB200_NO_ONE_LAUNCH")) return GIPB200_OK;
  int longest = 0;
  for (int i = 0; i < n; ++i) longest = std::max(longest, L->h_rowptr[i + 1] - L->h_rowptr[i]);
  bool zero = true;  // the iterations drop ghost columns: all of them stored zeros
  GIPB_TRY(ghosts_zero(s, &zero));
  if (!zero) return GIPB200_OK;
  DeviceInfo di;
  GIPB_TRY(device_info(&di));
  const int ctas = std::min(di.nsm, kGridCtasMax);
  // One CTA as far as its threads hold the rows; above, a second SM's arithmetic is worth the
  // cluster's barriers (12^3 2.45 against 2.66 us per iteration, but 1.9 / 2.5 at 11^3 and
  // 1.4 / 2.0 at 8^3).
  if (longest <= kRowSlots && n <= 4 * kBlockThreads) {
    one.form = OneLaunch::kBlock;
    one.per_thread = (n + kBlockThreads - 1) / kBlockThreads;
    one.row_slots = longest;
    one.ctas = 1;
    one.threads = ((n + one.per_thread - 1) / one.per_thread + 31) / 32 * 32;
    return GIPB200_OK;
  }
  if (longest <= kRowSlots && n <= kRegThreads * 4 * ClusterPairs::kMaxCtas) {
    // the fewest CTAs that leave a thread at most 4 rows, fewer rows while 8 CTAs (the
    // portable cluster size) hold them
    const int k = n <= kRegThreads * 2 * 8 ? 2 : 4;
    int c = 1;
    while (c * kRegThreads * k < n) c *= 2;
    one.ctas = c;
    one.per_thread = k;
    one.threads = ((n + c * k - 1) / (c * k) + 31) / 32 * 32;
    const bool fits = k == 2 ? cluster_fits(k_pcg64_cluster<2>, one)
                             : cluster_fits(k_pcg64_cluster<4>, one);
    if (fits) {
      one.form = OneLaunch::kCluster;
      return GIPB200_OK;
    }
  }
  if (longest <= kRowSlots && n <= kRegThreads * 4 * ctas) {
    const int k = (n + kRegThreads * ctas - 1) / (kRegThreads * ctas);
    one.form = OneLaunch::kGrid;
    one.per_thread = k;
    one.threads = kRegThreads;
    one.ctas = (n + kRegThreads * k - 1) / (kRegThreads * k);
    GIPB_TRY(one.pair.alloc((size_t)n));
    return one.slots.alloc(grid_slot_count(one.ctas));
  }
  GIPB_TRY(build_packed64(s));
  if (op64.bits) {
    const size_t sh = stream_shared(L->nslices, ctas);
    if (op64.bits == 4 ? stream_fits(k_pcg64_stream<4>, sh) : stream_fits(k_pcg64_stream<8>, sh)) {
      one.form = OneLaunch::kStream;
      one.threads = 1024;
      one.ctas = ctas;
      one.shared = sh;
      return one.slots.alloc(grid_slot_count(ctas));
    }
  }
  return GIPB200_OK;
}

namespace {
template <int K>
int launch_block(const OneLaunch& o, const Args64& A, cudaStream_t s) {
  if (o.row_slots <= 7) k_pcg64_block<K, 7><<<1, o.threads, 0, s>>>(A);
  else k_pcg64_block<K, 8><<<1, o.threads, 0, s>>>(A);
  GIPB_LAUNCH_CHECK();
  return GIPB200_OK;
}

template <class K, class... Args>
int launch_one(K kern, const OneLaunch& o, cudaStream_t s, const Args&... args) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[1];
  one_launch_attr(kern, o, &cfg, at, o.form == OneLaunch::kCluster);
  cfg.stream = s;
  GIPB_CUDA(cudaLaunchKernelEx(&cfg, kern, args...));
  return GIPB200_OK;
}
}  // namespace

// The FP64 register form and the preconditioned form (persist_amg.cu), one after the other.
int Pcg::check_bounded_wait(cudaStream_t s, int* status) {
  DevBuf<ulonglong2> slots;
  GIPB_TRY(slots.alloc(grid_slot_count(2)));
  Args64 A{};
  A.slots = slots.p;
  A.S = sc.p;
  A.gave_up = gave_up;
  A.maxit = 1;
  *status = GIPB200_ERR_TIMEOUT;
  for (int k = 0; k < 3; ++k) {
    GIPB_TRY(slots.zero(s));
    GIPB_TRY(sc.zero(s));
    clear_gave_up();
    if (k == 0) k_pcg64_wait_check<<<1, kRegThreads, 0, s>>>(A);
    else launch_wait_check(k == 2, slots.p, s);
    GIPB_LAUNCH_CHECK();
    GIPB_TRY(result(s, nullptr));
    if (h_sc->status != GIPB200_ERR_TIMEOUT || !wait_gave_up()) *status = GIPB200_OK;
  }
  return GIPB200_OK;
}

static Stream64 stream64(const Pcg& P) {
  const Packed64& o = P.op64;
  return {o.delta.p, o.bits == 4 ? (const void*)o.idx4.p : (const void*)o.idx8.p, o.base.p,
          o.plain.p, o.table.p, P.p.p};
}

int Pcg::enqueue_one_launch(const double* b, double* x, const double* x0, cudaStream_t s) {
  if (one.form == OneLaunch::kSolve) return enqueue_solve_launch(b, x, x0, s);
  Args64 A{L->view(), b,     x0,    dinv.p,   x,        one.pair.p, one.slots.p, sc.p,
           gave_up,   prm.tol, n, n_all, prm.mode, prm.maxit};
  launches += 1;
  if (one.form != OneLaunch::kBlock && one.form != OneLaunch::kCluster)
    GIPB_CUDA(cudaMemsetAsync(one.slots.p, 0, one.slots.n * sizeof(ulonglong2), s));
  const int k = one.per_thread;
  switch (one.form) {
    case OneLaunch::kBlock:
      return k == 1   ? launch_block<1>(one, A, s)
             : k == 2 ? launch_block<2>(one, A, s)
             : k == 3 ? launch_block<3>(one, A, s)
                      : launch_block<4>(one, A, s);
    case OneLaunch::kCluster:
      return k == 2 ? launch_one(k_pcg64_cluster<2>, one, s, A)
                    : launch_one(k_pcg64_cluster<4>, one, s, A);
    case OneLaunch::kGrid:
      return k == 1   ? launch_one(k_pcg64_grid<1>, one, s, A)
             : k == 2 ? launch_one(k_pcg64_grid<2>, one, s, A)
             : k == 3 ? launch_one(k_pcg64_grid<3>, one, s, A)
                      : launch_one(k_pcg64_grid<4>, one, s, A);
    default: {
      const Stream64 M = stream64(*this);
      return op64.bits == 4 ? launch_one(k_pcg64_stream<4>, one, s, A, M)
                            : launch_one(k_pcg64_stream<8>, one, s, A, M);
    }
  }
}

void Pcg::launch_packed64_spmv(double* q, PcgScalars* S, int mode, cudaStream_t s) {
  const Stream64 M = stream64(*this);
  if (op64.bits == 4)
    k_pcg64_spmv_dot<4><<<blocks_spmv, 256, 0, s>>>(L->view(), M, q, S, rs, mode);
  else
    k_pcg64_spmv_dot<8><<<blocks_spmv, 256, 0, s>>>(L->view(), M, q, S, rs, mode);
}

}  // namespace gipb200
