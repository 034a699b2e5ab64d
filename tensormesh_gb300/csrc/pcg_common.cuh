// Pieces shared by the persistent PCG kernels (CSR and SELL-32): the solver
// record at the head of the workspace, the bounded grid barrier, the block
// and per-CTA-partial reductions, and the double-float storage pair.
#pragma once
#include "tm_common.cuh"
#include "../../include/tensormesh_gb300.h"

namespace tmg {

struct PcgState {
  unsigned int count;
  unsigned int gen;
  int status;
  int iters;
  double res;   // final recurrence residual norm
  double bnorm;
};

constexpr long long kGridSpinLimit = 1ll << 25;  // ~1 s with the 32 ns back-off

__device__ __forceinline__ bool grid_sync(PcgState* st, unsigned nblocks, unsigned& my_gen,
                                          long long spin_limit = kGridSpinLimit) {
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned g = my_gen;
    __threadfence();
    unsigned arrived = atomicAdd(&st->count, 1u);
    if (arrived == nblocks - 1) {
      atomicExch(&st->count, 0u);
      __threadfence();
      atomicAdd(&st->gen, 1u);
    } else {
      volatile unsigned* gen = &st->gen;
      long long spins = 0;
      while (*gen == g) {
        if (++spins > spin_limit) {
          atomicExch(&st->status, TM_ERR_TIMEOUT);
          break;
        }
        __nanosleep(32);
      }
    }
    __threadfence();
  }
  ++my_gen;
  __syncthreads();
  return *((volatile int*)&st->status) == TM_OK;
}

// Grid-wide sums that are also the barrier.  A CTA publishes its sums as
// tagged words -- a double's halves with the barrier's number in the low 32
// bits of each 8-byte word --, CTA 0 reads every CTA's words until they carry
// that number, adds them and publishes the totals the same way, and every CTA
// waits for those.  So the data are their own flags: no counter, no generation
// word, no second read of partial sums.  (All CTAs reading all words took 6.5
// us for 152 CTAs: their requests queue at the few L2 lines.)  Two sets of
// words alternate: a CTA writes set k + 2 only after the totals of k + 1, which
// CTA 0 published after reading set k + 1 of every CTA, that is, after every
// CTA had read the totals of k.  Bounded: about a second without progress ends
// the wait.
struct GridSlots {
  ulonglong2* w;   // [2 sets][nb][2 sums], then the totals [2 sets][kTotals][8]
  unsigned nb;
};
constexpr unsigned kTotals = 8;                  // copies of the totals, 128 bytes apart
__host__ __device__ inline size_t grid_slot_bytes(unsigned nb) {
  return ((size_t)nb * 4 + 2 * kTotals * 8 + 8) * sizeof(ulonglong2);
}
constexpr long long kSlotSpinLimit = 1ll << 20;  // polls of about a microsecond
constexpr int kSlotThreads = 512;                // threads of the calling CTA

__device__ __forceinline__ ulonglong2 slot_load(const ulonglong2* p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void slot_store(ulonglong2* p, double d, unsigned tag) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(d);
  const unsigned long long x = (b & 0xffffffff00000000ull) | tag, y = (b << 32) | tag;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(x), "l"(y) : "memory");
}

__device__ __forceinline__ double slot_value(ulonglong2 v) {
  return __longlong_as_double((long long)((v.x & 0xffffffff00000000ull) | (v.y >> 32)));
}

// Sums of doubles in integers.  FP64 additions issue at one warp instruction
// per ~70 cycles and SM partition, and a sum of 512 values with its second one
// took 1.9 us as a chain of them.  Here the values are written in units of
// 2^-63 of twice the largest one (fixed point, 21-bit limbs, so that 512 of
// them add without overflow) and the limbs are added by the warp's integer
// reductions.  The result is exact up to the truncation of each value, below
// 2^-62 of the largest (a double's own rounding is 2^-53 of the sum), and does
// not depend on the order.
struct Limbs {
  int h, m, l;
};
__device__ __forceinline__ int fix_exp(double d) { return (int)(((unsigned)__double2hiint(d) >> 20) & 0x7ffu); }
__device__ __forceinline__ Limbs fix_limbs(double d, int emax) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(d);
  const int e = (int)((b >> 52) & 0x7ff), sh = emax - e;
  const unsigned long long x = ((b & 0xfffffffffffffull) | 0x10000000000000ull) << 10;
  const unsigned long long y = (e != 0 && sh < 64) ? x >> sh : 0ull;
  Limbs r{(int)(y >> 42), (int)((y >> 21) & 0x1fffffull), (int)(y & 0x1fffffull)};
  if ((long long)b < 0) r = Limbs{-r.h, -r.m, -r.l};
  return r;
}
__device__ __forceinline__ Limbs fix_add(Limbs a, Limbs b) { return Limbs{a.h + b.h, a.m + b.m, a.l + b.l}; }
__device__ __forceinline__ Limbs fix_warp(Limbs a) {
  return Limbs{__reduce_add_sync(0xffffffffu, a.h), __reduce_add_sync(0xffffffffu, a.m),
               __reduce_add_sync(0xffffffffu, a.l)};
}
// The double nearest to (h 2^42 + m 2^21 + l) 2^(emax - 1085); nan when a value
// was nan or inf (emax = 2047).
__device__ __forceinline__ double fix_value(Limbs a, int emax) {
  if (emax >= 2047) return __longlong_as_double(0x7ff8000000000000ll);
  // t = h 2^21 + m (|t| < 2^53), total = t 2^21 + l
  const long long t = ((long long)a.h << 21) + a.m;
  long long hi = t >> 20, lo = ((t & 0xfffffll) << 21) + a.l;   // total = hi 2^41 + lo, |lo| < 2^42
  hi += lo >> 41;
  lo &= 0x1ffffffffffll;                                        // 0 <= lo < 2^41
  const bool neg = hi < 0;
  if (neg) {
    hi = ~hi;
    lo = 0x20000000000ll - lo;
    hi += lo >> 41;
    lo &= 0x1ffffffffffll;
  }
  if ((hi | lo) == 0) return 0.0;
  // magnitude hi 2^41 + lo (hi < 2^33), normalised into 64 bits
  unsigned long long v;
  int top;   // the leading bit's weight is 2^top
  if (hi) {
    const int z = __clzll(hi);
    top = 63 - z + 41;
    // lo's 41 bits follow hi's: hi < 2^33, so z >= 31 and the shift is 31 .. 63 less 41
    v = ((unsigned long long)hi << z) | (z >= 41 ? (unsigned long long)lo << (z - 41) : (unsigned long long)lo >> (41 - z));
  } else {
    const int z = __clzll(lo);
    top = 63 - z;
    v = (unsigned long long)lo << z;
  }
  const int ex = top + emax - 1085 + 1023;   // biased exponent of the result
  if (ex < 1) return neg ? -0.0 : 0.0;
  const unsigned long long r = (v >> 11) + ((v >> 10) & 1ull);   // 53 bits, rounded half up
  const unsigned long long bits = ((unsigned long long)(ex - 1) << 52) + r;
  return __longlong_as_double((long long)(neg ? bits | 0x8000000000000000ull : bits));
}

// Sums of a and b (b with kTwo) over the threads of the CTA, valid in warp 0;
// every thread calls it (two barriers inside).
template <bool kTwo>
__device__ __forceinline__ void cta_sum(double& a, double& b, int* s_red /* [8][kSlotThreads / 32] */) {
  constexpr int NW = kSlotThreads / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  {
    const int ea = __reduce_max_sync(0xffffffffu, fix_exp(a));
    const int eb = kTwo ? __reduce_max_sync(0xffffffffu, fix_exp(b)) : 0;
    if (lane == 0) {
      s_red[warp] = ea;
      if (kTwo) s_red[NW + warp] = eb;
    }
  }
  __syncthreads();
  const int ea = __reduce_max_sync(0xffffffffu, lane < NW ? s_red[lane] : 0);
  const int eb = kTwo ? __reduce_max_sync(0xffffffffu, lane < NW ? s_red[NW + lane] : 0) : 0;
  {
    const Limbs la = fix_warp(fix_limbs(a, ea));
    Limbs lb{0, 0, 0};
    if (kTwo) lb = fix_warp(fix_limbs(b, eb));
    if (lane == 0) {
      s_red[2 * NW + warp] = la.h;
      s_red[3 * NW + warp] = la.m;
      s_red[4 * NW + warp] = la.l;
      if (kTwo) {
        s_red[5 * NW + warp] = lb.h;
        s_red[6 * NW + warp] = lb.m;
        s_red[7 * NW + warp] = lb.l;
      }
    }
  }
  __syncthreads();
  if (warp != 0) return;
  auto total = [&](int at, int e) {
    Limbs v{0, 0, 0};
    if (lane < NW) v = Limbs{s_red[at * NW + lane], s_red[(at + 1) * NW + lane], s_red[(at + 2) * NW + lane]};
    return fix_value(fix_warp(v), e);
  };
  a = total(2, ea);
  if (kTwo) b = total(5, eb);
}

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The same over a cluster: every CTA writes its sums into the shared memory of
// all of them (s_slot[2 sets][16][2], alternating like the grid's words) and
// one hardware cluster barrier, which also orders the CTAs' global stores,
// stands between the writes and the reads.  The caller has passed a cluster
// barrier before its first sum, so that all of them have started.
template <bool kTwo>
__device__ __forceinline__ void cluster_sum(unsigned gen, unsigned nb, double& a, double& b, int* s_red,
                                            double* s_slot) {
  const int lane = threadIdx.x & 31;
  cta_sum<kTwo>(a, b, s_red);
  double* set = s_slot + (gen & 1u) * 32;
  if (threadIdx.x < 32 && lane < (int)nb) {
    unsigned rank, at = (unsigned)__cvta_generic_to_shared(set), dst;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(at + rank * 16), "r"((unsigned)lane));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(dst), "d"(a) : "memory");
    if (kTwo) asm volatile("st.shared::cluster.f64 [%0+8], %1;" ::"r"(dst), "d"(b) : "memory");
  }
  cluster_barrier();
  if (threadIdx.x < 32) {
    auto sum = [&](int k) {
      const double d = lane < (int)nb ? set[2 * lane + k] : 0.0;
      const int e = __reduce_max_sync(0xffffffffu, fix_exp(d));
      return fix_value(fix_warp(fix_limbs(d, e)), e);
    };
    a = sum(0);
    if (kTwo) b = sum(1);
  }
}

// a and b (b with kTwo) become their sums over all threads of the grid, valid in
// warp 0 of every CTA, the same bits everywhere.  Every thread of the CTA calls
// it; the caller's __syncthreads after it completes the barrier.  Returns false
// in warp 0 when the wait ran out (st->status is set).  kFence = false: only
// the sums are exchanged; what the CTAs stored before becomes visible at the
// next sum with fences.
template <bool kTwo, bool kFence = true>
__device__ __forceinline__ bool grid_sum(PcgState* st, const GridSlots& sl, unsigned gen, double& a, double& b,
                                         int* s_red, long long spin_limit = kSlotSpinLimit) {
  cta_sum<kTwo>(a, b, s_red);
  const int lane = threadIdx.x & 31;
  if (threadIdx.x >= 32) return true;
  ulonglong2* set = sl.w + (gen & 1u) * 2 * (size_t)sl.nb;
  {
    if (lane == 0) {
      if (kFence) __threadfence();   // the CTA's vector stores before its words
      slot_store(set + 2 * blockIdx.x, a, gen);
      if (kTwo) slot_store(set + 2 * blockIdx.x + 1, b, gen);
    }
  }
  __syncwarp();
  bool ok = true;
  // the totals of this set, on a 128-byte boundary
  ulonglong2* tot = reinterpret_cast<ulonglong2*>((reinterpret_cast<uintptr_t>(sl.w + 4 * (size_t)sl.nb) + 127) & ~uintptr_t(127)) +
                    (gen & 1u) * kTotals * 8;
  if (blockIdx.x == 0) {
    constexpr int U = 5;   // slots of a lane in flight
    a = b = 0.0;
    for (unsigned i0 = 0; i0 < sl.nb; i0 += 32 * U) {
      ulonglong2 va[U], vb[U];
      long long spins = 0;
      for (;;) {
        bool ready = true;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const unsigned i = i0 + 32 * u + lane;
          va[u] = make_ulonglong2(gen, gen);   // an absent slot adds zero
          if (i < sl.nb) va[u] = slot_load(set + 2 * i);
          if (kTwo) {
            vb[u] = make_ulonglong2(gen, gen);
            if (i < sl.nb) vb[u] = slot_load(set + 2 * i + 1);
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          ready = ready && (unsigned)va[u].x == gen && (unsigned)va[u].y == gen;
          if (kTwo) ready = ready && (unsigned)vb[u].x == gen && (unsigned)vb[u].y == gen;
        }
        if (__all_sync(0xffffffffu, ready)) break;
        if (++spins > spin_limit) {
          ok = false;
          break;
        }
      }
      if (!ok) break;
      auto sum = [&](const ulonglong2 (&v)[U]) {
        double d[U];
        int e = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          d[u] = slot_value(v[u]);
          e = max(e, fix_exp(d[u]));
        }
        e = __reduce_max_sync(0xffffffffu, e);
        Limbs t = fix_limbs(d[0], e);
#pragma unroll
        for (int u = 1; u < U; ++u) t = fix_add(t, fix_limbs(d[u], e));
        return fix_value(fix_warp(t), e);
      };
      const double x = sum(va);
      a = i0 ? a + x : x;
      if (kTwo) {
        const double y = sum(vb);
        b = i0 ? b + y : y;
      }
    }
    if (ok) {
      if (kFence) __threadfence();   // the other CTAs' stores before the totals
      if (lane < (int)kTotals) {
        slot_store(tot + lane * 8, a, gen);
        if (kTwo) slot_store(tot + lane * 8 + 1, b, gen);
      }
    }
  } else {
    const ulonglong2* t = tot + (blockIdx.x % kTotals) * 8;
    long long spins = 0;
    for (;;) {
      const ulonglong2 x = slot_load(t), y = kTwo ? slot_load(t + 1) : make_ulonglong2(gen, gen);
      const bool ready = (unsigned)x.x == gen && (unsigned)x.y == gen && (unsigned)y.x == gen && (unsigned)y.y == gen;
      if (__all_sync(0xffffffffu, ready)) {
        a = slot_value(x);
        b = slot_value(y);
        break;
      }
      if (++spins > spin_limit) {
        ok = false;
        break;
      }
    }
  }
  if (kFence) __threadfence();     // what the other CTAs stored before their words
  if (!ok && lane == 0) atomicExch(&st->status, TM_ERR_TIMEOUT);
  return ok;
}

template <class T>
__device__ __forceinline__ T block_sum(T v, T* s_red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if (lane == 0) s_red[warp] = v;
  __syncthreads();
  T t = 0;
  if (warp == 0) {
    t = lane < (blockDim.x >> 5) ? s_red[lane] : T(0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
  }
  __syncthreads();
  return t;  // valid in thread 0
}

// Sum the per-CTA partials (same order in every CTA).
template <class T>
__device__ __forceinline__ T sum_partials(const T* part, int n, T* s_red) {
  T v = 0;
  if (threadIdx.x < 32) {
    for (int i = threadIdx.x; i < n; i += 32) v += ((volatile T*)part)[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) s_red[0] = v;
  }
  __syncthreads();
  T r = s_red[0];
  __syncthreads();
  return r;
}

// FP64 systems: values and vectors are held as double-float pairs (same bytes
// as double) and every operation runs on the FP32 pipe; GB300's native FP64
// FMA rate (~0.5 T/s) would otherwise bound the SpMV.
struct F2 {
  float hi, lo;
};
TM_D df64 ld2(const F2* a, int64_t i) {
  F2 v = a[i];
  return {v.hi, v.lo};
}
TM_D void st2(F2* a, int64_t i, df64 v) { a[i] = F2{v.hi, v.lo}; }

}  // namespace tmg
