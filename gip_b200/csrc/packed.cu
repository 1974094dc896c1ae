// FP64 operators packed in their stored slot order: the lossless layout of internal.cuh's
// Packed64, its builder, and the standalone products from it.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <new>

#include "device.cuh"
#include "internal.cuh"

namespace gipb200 {

namespace {

// cols: columns below it are kept; entries of later ones (ghost cells whose stored values the
// caller knows to be zeros) become padding.  keep_zeros: a stored zero is an entry with a
// table value of its own (its product with an infinity is a NaN, as in the sliced layout);
// else it is padding that gathers its column and multiplies by table entry 0.
int build(const Sell& S, int cols, bool keep_zeros, Packed64* out, cudaStream_t s) {
  const int ns = S.nslices;
  const long long nslots = S.nslots;
  if (ns == 0 || nslots == 0) return GIPB200_OK;
  std::vector<long long> sptr((size_t)ns + 1);
  std::vector<int> col((size_t)nslots);
  std::vector<double> val((size_t)nslots);
  GIPB_CUDA(cudaMemcpyAsync(sptr.data(), S.sptr.p, sptr.size() * 8, cudaMemcpyDeviceToHost, s));
  GIPB_CUDA(cudaMemcpyAsync(val.data(), S.val.p, val.size() * 8, cudaMemcpyDeviceToHost, s));
  GIPB_CUDA(cudaStreamSynchronize(s));
  std::vector<double> tab;
  if (!value_table(val.data(), nslots, 255, &tab)) return GIPB200_OK;
  GIPB_CUDA(cudaMemcpyAsync(col.data(), S.col.p, col.size() * 4, cudaMemcpyDeviceToHost, s));
  GIPB_CUDA(cudaStreamSynchronize(s));
  std::vector<unsigned long long> keys;
  for (double t : tab) {
    unsigned long long k;
    memcpy(&k, &t, 8);
    if (k != 0ull || keep_zeros) keys.push_back(k);
  }
  if (keys.size() > 255) return GIPB200_OK;
  const int nib = keys.size() <= 15 ? 4 : 8;
  std::vector<double> table((size_t)1 << nib, 0.0);
  for (size_t t = 0; t < keys.size(); ++t) memcpy(&table[t + 1], &keys[t], 8);
  const size_t rows = (size_t)ns * 32;
  std::vector<uint4> delta(rows, make_uint4(0u, 0u, 0u, 0u));
  std::vector<unsigned> idx4(nib == 4 ? rows : 0, 0u);
  std::vector<uint2> idx8(nib == 8 ? rows : 0, make_uint2(0u, 0u));
  std::vector<int> base((size_t)ns * 8, 0);
  std::vector<unsigned char> plain((size_t)ns, 1);
  long long packed = 0;
  int longest = 0;
#pragma omp parallel for schedule(static) reduction(+ : packed) reduction(max : longest)
  for (int sl = 0; sl < ns; ++sl) {
    const long long b0 = sptr[sl];
    const int len = (int)((sptr[sl + 1] - b0) >> 5);
    if (len > 8) continue;
    int lo[8], hi[8];
    bool ok = true;
    for (int j = 0; j < len && ok; ++j) {
      lo[j] = 0x7fffffff;
      hi[j] = -1;
      for (int l = 0; l < 32; ++l) {
        const int c = col[b0 + 32LL * j + l];
        if (c < 0 || c >= cols) continue;
        lo[j] = std::min(lo[j], c);
        hi[j] = std::max(hi[j], c);
      }
      ok = hi[j] < 0 || hi[j] - lo[j] <= 65535;
    }
    if (!ok) continue;
    plain[sl] = 0;
    packed += 1;
    longest = std::max(longest, len);
    for (int j = 0; j < len; ++j) base[(size_t)sl * 8 + j] = hi[j] >= 0 ? lo[j] : 0;
    for (int l = 0; l < 32; ++l) {
      unsigned dw[4] = {0u, 0u, 0u, 0u};
      unsigned long long iw = 0ull;
      for (int j = 0; j < len; ++j) {
        const long long k = b0 + 32LL * j + l;
        if (col[k] < 0 || col[k] >= cols) continue;
        dw[j >> 1] |= (unsigned)(col[k] - lo[j]) << (16 * (j & 1));
        unsigned long long bits;
        memcpy(&bits, &val[k], 8);
        if (bits == 0ull && !keep_zeros) continue;
        const unsigned t =
            1u + (unsigned)(std::lower_bound(keys.begin(), keys.end(), bits) - keys.begin());
        iw |= (unsigned long long)t << (nib * j);
      }
      const size_t r = (size_t)sl * 32 + l;
      delta[r] = make_uint4(dw[0], dw[1], dw[2], dw[3]);
      if (nib == 4) idx4[r] = (unsigned)iw;
      else idx8[r] = make_uint2((unsigned)iw, (unsigned)(iw >> 32));
    }
  }
  if (packed * 2 < ns) return GIPB200_OK;  // not worth a second layout
  GIPB_TRY(out->delta.upload(delta.data(), delta.size(), s));
  if (nib == 4) GIPB_TRY(out->idx4.upload(idx4.data(), idx4.size(), s));
  else GIPB_TRY(out->idx8.upload(idx8.data(), idx8.size(), s));
  GIPB_TRY(out->base.upload(base.data(), base.size(), s));
  GIPB_TRY(out->plain.upload(plain.data(), plain.size(), s));
  GIPB_TRY(out->table.upload(table.data(), table.size(), s));
  GIPB_CUDA(cudaStreamSynchronize(s));
  out->bits = nib;
  out->slots = longest <= 7 ? 7 : 8;
  return GIPB200_OK;
}

}  // namespace

// The packed copy is a second one: where there is no memory for it the operator is used without.
int pack64(const Sell& S, int cols, bool keep_zeros, Packed64* out, cudaStream_t s) {
  out->release();
  int st;
  try {
    st = build(S, cols, keep_zeros, out, s);
  } catch (const std::bad_alloc&) {
    st = GIPB200_ERR_NOMEM;
  }
  if (st == GIPB200_OK) return GIPB200_OK;
  out->release();
  return st == GIPB200_ERR_NOMEM ? GIPB200_OK : st;
}

namespace {

struct PackedArgs {
  const uint4* delta;
  const void* idx;
  const int* base;
  const unsigned char* plain;
  const double* table;
};

struct StorePackedDot {
  double* out;
  __device__ void operator()(const double* t) const { *out = t[0]; }
};

// y = A x (mode 1: alpha A x + beta y) with GIP's row semantics; DOT: also out = x.y over the
// first n_dot rows (mode 0).  Entry 0 of the table is padding: such a slot gathers nothing.
// Streams 37 bytes a row (operator words 21, x, y) where the sliced layout streams 100, and is
// bound by its gathers: at 8 CTAs per SM the 200^3 pressure operator took 56 us (5.3 TB/s of
// those bytes) against 131 us sliced; with the next slice's words loaded ahead at 4 CTAs 64
// us, with a contiguous range of slices per CTA 66 us.
template <int NIB, bool DOT>
__global__ void __launch_bounds__(256, 8) k_packed_spmv(SellView<double> A, PackedArgs M,
                                                        const double* __restrict__ x,
                                                        double* __restrict__ y, double alpha,
                                                        double beta, int mode, int n_dot,
                                                        ReduceScratch rs, double* out) {
  dep_begin();
  __shared__ double tab[NIB == 4 ? 16 : 256];
  for (int t = threadIdx.x; t < (NIB == 4 ? 16 : 256); t += blockDim.x) tab[t] = M.table[t];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  double acc[1] = {0.0};
  for (int s = gw; s < A.nslices; s += nw) {
    const int i = s * 32 + lane;
    double sum = 0.0;
    bool any = false;
    PackedWords cur;
    packed_words<NIB>(M.delta, M.idx, M.plain, s, lane, cur);
    if (!cur.plain) {
      int c[8];
      packed_cols(M.base, s, cur.d, c);
      double xv[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) xv[j] = packed_index<NIB>(cur, j) ? __ldg(x + c[j]) : 0.0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const unsigned k = packed_index<NIB>(cur, j);
        if (k) sum = dadd(sum, dmul(xv[j], tab[k]));
      }
      any = (cur.w0 | cur.w1) != 0u;
    } else {
      sell_row_f64<double, double, 2>(A, x, s, lane, sum, any);
    }
    if (i < A.nrows) {
      if (DOT) {
        const double v = any ? sum : y[i];
        if (any) y[i] = v;
        if (i < n_dot) acc[0] = dadd(acc[0], dmul(x[i], v));
      } else if (any) {
        y[i] = mode ? dadd(dmul(alpha, sum), dmul(beta, y[i])) : sum;
      }
    }
  }
  if (DOT) grid_reduce<SumOp, 1>(acc, rs, StorePackedDot{out});
}

PackedArgs args_of(const Packed64& P) {
  return {P.delta.p, P.bits == 4 ? (const void*)P.idx4.p : (const void*)P.idx8.p, P.base.p,
          P.plain.p, P.table.p};
}

template <bool DOT>
int launch(const Sell& A, const Packed64& P, const double* x, double* y, double alpha, double beta,
           int mode, int n_dot, ReduceScratch rs, double* out, cudaStream_t s) {
  if (A.nrows == 0) return GIPB200_OK;
  int blocks = 1;
  GIPB_TRY(P.bits == 4 ? one_wave(k_packed_spmv<4, DOT>, (A.nslices * 32 + 255) / 256, &blocks)
                       : one_wave(k_packed_spmv<8, DOT>, (A.nslices * 32 + 255) / 256, &blocks));
  if (P.bits == 4)
    launch_dep(k_packed_spmv<4, DOT>, blocks, 256, s, A.view(), args_of(P), x, y, alpha, beta,
               mode, n_dot, rs, out);
  else
    launch_dep(k_packed_spmv<8, DOT>, blocks, 256, s, A.view(), args_of(P), x, y, alpha, beta,
               mode, n_dot, rs, out);
  GIPB_LAUNCH_CHECK();
  return GIPB200_OK;
}

}  // namespace

int launch_packed_spmv(const Sell& A, const Packed64& P, const double* x, double* y, double alpha,
                       double beta, int mode, cudaStream_t s) {
  return launch<false>(A, P, x, y, alpha, beta, mode, 0, ReduceScratch{}, nullptr, s);
}

int launch_packed_spmv_dot(const Sell& A, const Packed64& P, const double* x, double* y, int n_dot,
                           ReduceScratch rs, double* out, cudaStream_t s) {
  return launch<true>(A, P, x, y, 0.0, 0.0, 0, n_dot, rs, out, s);
}

}  // namespace gipb200
