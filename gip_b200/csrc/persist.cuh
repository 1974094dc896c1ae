// Building blocks of the solvers that run as one launch: reductions and barriers over a
// thread-block cluster (shared memory of its CTAs) or over a cooperative grid (epoch-stamped
// slots in global memory, every wait bounded).
#pragma once

#include "device.cuh"
#include "pcg.cuh"

namespace gipb200 {

// A grid wait that would never end gives up after about 2 s of SM clock (a check of that: 20 ms).
constexpr long long kGridSpinCycles = 4000000000LL, kCheckSpinCycles = 40000000LL;
constexpr int kGridSums = 5;       // sums per grid reduction
constexpr int kGridCtasMax = 256;  // CTAs of a grid reduction (each polled by one thread)
// 16-byte slots of one grid's reductions: [2 parities][kGridSums][CTA], then the arrival
// counter; all zero at launch
inline size_t grid_slot_count(int ncta) { return (size_t)2 * kGridSums * ncta + 1; }

// One 16-byte slot {value, epoch}, written and read as one access, so a reader that sees the
// epoch sees its value: the arrival flag and the partial sum travel together.
__device__ __forceinline__ void slot_store(ulonglong2* p, double v, unsigned long long epoch) {
  asm volatile(
      "{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
      "l"(__double_as_longlong(v)), "l"(epoch)
      : "memory");
}
__device__ __forceinline__ void slot_load(const ulonglong2* p, double& v, unsigned long long& epoch) {
  long long a;
  asm volatile(
      "{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
      : "=l"(a), "=l"(epoch)
      : "l"(p)
      : "memory");
  v = __longlong_as_double(a);
}

// Sums over a cooperative grid of at most kGridCtasMax CTAs (and at most blockDim.x).  Every
// CTA writes its partial sums to its slots and counts its arrival; one thread of each CTA
// polls the counter, then thread t reads CTA t's slots and checks their epochs.  The counter
// only says when to look: without FENCE nothing orders it after the slots, so no store has to
// be waited for (a fence behind a store costs 0.4 to 0.6 us here), and a slot that is not
// there yet is polled.  Measured on 148 CTAs of 256 threads: 1.5 us, with FENCE 2.0 us; slots
// behind a fenced counter 1.9, all-to-all mailboxes 2.5 / 3.3, CTA 0 adding for all 2.9 /
// 4.3, every CTA polling every slot 3.9 us.
// Every CTA adds the partials in the same order: the totals are identical everywhere and
// depend only on the launch shape.  Two slot sets alternate: a CTA overwrites a set only
// after every CTA has passed the next reduction, so nobody still waits for the old epoch.
struct GridScope {
  ulonglong2* slots;
  unsigned* count;
  unsigned epoch;
  int ncta, rank;
  long long spin;  // cycles after which a wait gives up
  bool ok;  // false: a wait gave up (the same in every thread after the call that noticed)
};

__device__ __forceinline__ GridScope grid_begin(ulonglong2* slots, int rank, int ncta,
                                                 long long spin = kGridSpinCycles) {
  return GridScope{slots, reinterpret_cast<unsigned*>(slots + (size_t)2 * kGridSums * ncta), 0u,
                   ncta, rank, spin, true};
}
__device__ __forceinline__ GridScope grid_begin(ulonglong2* slots) {
  return grid_begin(slots, (int)blockIdx.x, (int)gridDim.x);
}

// A solve one of whose waits gave up tells the host, whoever enqueued it (pinned memory).
__device__ __forceinline__ void report_gave_up(int* flag) {
  *static_cast<volatile int*>(flag) = 1;
  __threadfence_system();
}

// FENCE: the reduction is also a barrier for global memory (what any thread of the grid wrote
// before it is visible to every thread after it); without it only the sums are exchanged.
template <int W, bool FENCE>
__device__ __forceinline__ bool grid_sum(double (&v)[W], GridScope& G) {
  static_assert(W <= kGridSums, "too many sums");
  __shared__ double sh1[W][32];
  __shared__ double sh2[W][kGridCtasMax / 32];
  __shared__ int s_fail;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  ulonglong2* set = G.slots + (size_t)(G.epoch & 1u) * kGridSums * G.ncta;
  G.epoch += 1u;
#pragma unroll
  for (int k = 0; k < W; ++k) {
    const double t = warp_reduce<SumOp>(v[k]);
    if (lane == 0) sh1[k][warp] = t;
  }
  __syncthreads();
  if (warp == 0) {
    double t[W];
#pragma unroll
    for (int k = 0; k < W; ++k) t[k] = warp_reduce<SumOp>(lane < nw ? sh1[k][lane] : 0.0);
    if (lane == 0) {
      if (FENCE) __threadfence();
#pragma unroll
      for (int k = 0; k < W; ++k) slot_store(set + (size_t)k * G.ncta + G.rank, t[k], G.epoch);
      asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(G.count) : "memory");
      const unsigned target = G.epoch * (unsigned)G.ncta;
      const long long t0 = clock64();
      unsigned c;
      s_fail = 0;
      while (true) {
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(G.count) : "memory");
        if ((int)(c - target) >= 0) break;
        if (clock64() - t0 > G.spin) {
          s_fail = 1;
          break;
        }
      }
      if (FENCE) __threadfence();
    }
  }
  __syncthreads();
  const int nwait = (G.ncta + 31) >> 5;  // warps that read the slots
  if (warp < nwait) {
    double t[W];
#pragma unroll
    for (int k = 0; k < W; ++k) t[k] = 0.0;
    if ((int)threadIdx.x < G.ncta && !s_fail) {
      const long long t0 = clock64();
#pragma unroll
      for (int k = 0; k < W; ++k) {
        unsigned long long e;
        while (true) {
          slot_load(set + (size_t)k * G.ncta + threadIdx.x, t[k], e);
          if (e == G.epoch) break;
          if (clock64() - t0 > G.spin) {
            s_fail = 1;
            break;
          }
        }
      }
    }
#pragma unroll
    for (int k = 0; k < W; ++k) {
      const double a = warp_reduce<SumOp>(t[k]);
      if (lane == 0) sh2[k][warp] = a;
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < W; ++k) {
    double a = sh2[k][0];
    for (int i = 1; i < nwait; ++i) a = dadd(a, sh2[k][i]);
    v[k] = a;
  }
  if (s_fail) G.ok = false;
  return G.ok;
}

// A grid barrier in two halves: between them a CTA may load what no CTA of the grid writes.
__device__ __forceinline__ void grid_arrive(GridScope& G) {
  G.epoch += 1u;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(G.count) : "memory");
  }
}
// Every thread of the grid has arrived and what it wrote before is visible; false: gave up.
__device__ __forceinline__ bool grid_wait(GridScope& G) {
  __shared__ int s_fail;
  if (threadIdx.x == 0) {
    const unsigned target = G.epoch * (unsigned)G.ncta;
    const long long t0 = clock64();
    unsigned c;
    s_fail = 0;
    while (true) {
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(G.count) : "memory");
      if ((int)(c - target) >= 0) break;
      if (clock64() - t0 > G.spin) {
        s_fail = 1;
        break;
      }
    }
    __threadfence();
  }
  __syncthreads();
  if (s_fail) G.ok = false;
  return G.ok;
}

// ------------------------------------------------------------------ clusters
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// Every thread of the cluster; release/acquire over its shared memory.
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
// The address of CTA `rank`'s copy of a shared variable of this CTA.
__device__ __forceinline__ unsigned map_shared(unsigned addr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

}  // namespace gipb200
