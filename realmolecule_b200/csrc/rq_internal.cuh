// rq_internal.cuh -- shared definitions of the librq CUDA kernels (sm_100a).
//
// Layout in HBM: every field is one flat array of S^3 elements, id = i*S^2 + j*S + k
// (k fastest), exactly the reference layout (cloud/solver.py:24-26,
// molecule.js:273-276), so host buffers copy in and out without repacking.
//
// Arithmetic: kernels whose results feed an integer decision (labels) or whose
// outputs are compared bit-for-bit with the reference's own kernels use the
// explicitly rounded intrinsics below (F_ADD ...), which the compiler never
// contracts into FMAs; the order of operations is the reference's.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "exact_sum.h"

#define F_ADD(a, b) __fadd_rn((a), (b))
#define F_SUB(a, b) __fsub_rn((a), (b))
#define F_MUL(a, b) __fmul_rn((a), (b))
#define F_DIV(a, b) __fdiv_rn((a), (b))
#define F_SQRT(a) __fsqrt_rn((a))

// F_SQRT where 0 is a usual argument (the gradient of a front is 0 in most of a box): 0 takes the square
// root's slow path, a call of its own per element
__device__ __forceinline__ float sqrt0(float a) {
  const float r = __fsqrt_rn(a == 0.0f ? 1.0f : a);
  return a == 0.0f ? a : r;
}

namespace rq {

constexpr int kThreadsK = 32;  // threads along k (contiguous) per block
constexpr int kThreadsJ = 8;   // threads along j per block
constexpr int kMarch = 16;     // planes along i marched by one thread
constexpr int kNmPD = 5;       // new flavour: readout sums per domain (norm, T, V_eK, P rho, P A P)

// bits of the same-label neighbour mask of a point: set when neighbour +i, -i, +j, -j, +k, -k carries the
// point's label; kNmIn on every interior point (the mask of a face point is 0)
constexpr int kNmIp = 1, kNmIm = 2, kNmJp = 4, kNmJm = 8, kNmKp = 16, kNmKm = 32, kNmIn = 64;

struct Geo {
  int S;      // points per axis
  int NN;     // S - 1
  long long S2, S3;
};

inline Geo make_geo(int S) {
  Geo g;
  g.S = S;
  g.NN = S - 1;
  g.S2 = (long long)S * S;
  g.S3 = g.S2 * S;
  return g;
}

// Interior march launch: blocks of 32(k) x 8(j) threads, each thread walking kMarch planes in i.
inline dim3 march_grid(const Geo& g, int march = kMarch) {
  int n = g.NN - 1;  // interior points per axis
  return dim3((n + kThreadsK - 1) / kThreadsK, (n + kThreadsJ - 1) / kThreadsJ, (n + march - 1) / march);
}
inline dim3 march_block() { return dim3(kThreadsK, kThreadsJ, 1); }

// ---------------------------------------------------------------------------------------
// Label-keyed FP64 block aggregation.  Each thread carries a running (label, NQ sums)
// pair while it marches; when the label changes the pair is merged into a small
// open-addressing table in shared memory; at block end every used slot is added to the
// global per-domain array with one FP64 atomic per quantity.  A label that finds no free
// slot goes straight to global memory, so the result is exact for any label count.
// ---------------------------------------------------------------------------------------
template <int NQ, int NSLOT = 128>
struct DomTable {
  int keys[NSLOT];
  double vals[NSLOT * NQ];
};

template <int NQ, int NSLOT>
__device__ __forceinline__ void dom_table_init(DomTable<NQ, NSLOT>& t) {
  const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
  const int nt = blockDim.x * blockDim.y * blockDim.z;
  for (int s = tid; s < NSLOT; s += nt) t.keys[s] = -1;
  for (int s = tid; s < NSLOT * NQ; s += nt) t.vals[s] = 0.0;
}

template <int NQ, int NSLOT>
__device__ __forceinline__ void dom_table_add(DomTable<NQ, NSLOT>& t, int label, const double* v, double* global) {
  unsigned slot = ((unsigned)label * 2654435761u) & (NSLOT - 1);
  for (int p = 0; p < NSLOT; ++p) {
    int old = atomicCAS(&t.keys[slot], -1, label);
    if (old == -1 || old == label) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) atomicAdd(&t.vals[slot * NQ + q], v[q]);
      return;
    }
    slot = (slot + 1) & (NSLOT - 1);
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q) atomicAdd(&global[(long long)label * NQ + q], v[q]);
}

template <int NQ, int NSLOT>
__device__ __forceinline__ void dom_table_flush(DomTable<NQ, NSLOT>& t, double* global) {
  const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
  const int nt = blockDim.x * blockDim.y * blockDim.z;
  for (int s = tid; s < NSLOT; s += nt) {
    int k = t.keys[s];
    if (k >= 0) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) atomicAdd(&global[(long long)k * NQ + q], t.vals[s * NQ + q]);
    }
  }
}

// lane of the calling thread in its warp (blocks of any shape)
__device__ __forceinline__ int lane_id() {
  int l;
  asm("mov.u32 %0, %%laneid;" : "=r"(l));
  return l;
}

// Per-thread running sum keyed by label; flushes into the block table on label change.
template <int NQ>
struct RunSum {
  int label;
  double v[NQ];
  __device__ __forceinline__ void reset() {
    label = -1;
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = 0.0;
  }
  template <int NSLOT>
  __device__ __forceinline__ void add(int l, const double* x, DomTable<NQ, NSLOT>& t, double* global) {
    if (l != label) {
      if (label >= 0) dom_table_add(t, label, v, global);
      label = l;
#pragma unroll
      for (int q = 0; q < NQ; ++q) v[q] = x[q];
    } else {
#pragma unroll
      for (int q = 0; q < NQ; ++q) v[q] += x[q];
    }
  }
  template <int NSLOT>
  __device__ __forceinline__ void finish(DomTable<NQ, NSLOT>& t, double* global) {
    if (label >= 0) dom_table_add(t, label, v, global);
  }
  // Same as finish, but must be called by every lane of the warp together: lanes holding the
  // same label first combine their sums with shuffles, so one lane per distinct label touches
  // the shared table (neighbouring k values almost always share a label).
  template <int NSLOT>
  __device__ __forceinline__ void finish_warp(DomTable<NQ, NSLOT>& t, double* global) {
    const unsigned peers = __match_any_sync(0xffffffffu, label);
    const int lane = lane_id();
    double s[NQ];
    if (__all_sync(0xffffffffu, peers == 0xffffffffu)) {
      // one label over the warp (the common case): a butterfly
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        double x = v[q];
        x += __shfl_xor_sync(0xffffffffu, x, 16);
        x += __shfl_xor_sync(0xffffffffu, x, 8);
        x += __shfl_xor_sync(0xffffffffu, x, 4);
        x += __shfl_xor_sync(0xffffffffu, x, 2);
        x += __shfl_xor_sync(0xffffffffu, x, 1);
        s[q] = x;
      }
      if (label >= 0 && lane == 0) dom_table_add(t, label, s, global);
      return;
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) s[q] = 0.0;
    for (int l = 0; l < 32; ++l) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const double x = __shfl_sync(0xffffffffu, v[q], l);
        if ((peers >> l) & 1u) s[q] += x;
      }
    }
    if (label >= 0 && lane == __ffs(peers) - 1) dom_table_add(t, label, s, global);
  }
};

// acc += v for an accumulator of exact_sum.h in global memory, from any number of threads
__device__ __forceinline__ void exact_add(long long* acc, double v) {
  long long p[3];
  const int w = exact_split(v, p);
  auto* a = reinterpret_cast<unsigned long long*>(acc) + w;
  if (w == kExFlags) {
    atomicOr(a, (unsigned long long)p[0]);
    return;
  }
#pragma unroll
  for (int q = 0; q < 3; ++q)
    if (p[q]) atomicAdd(a + q, (unsigned long long)p[q]);
}

// The double next to an accumulator, by a warp (every lane gets it)
__device__ __forceinline__ double exact_value_warp(const long long* __restrict__ acc) {
  const int lane = lane_id();
  const long long a = acc[lane], b = acc[lane + 32], c = lane < kExWords - 64 ? acc[lane + 64] : 0;
  const unsigned na = __ballot_sync(0xffffffffu, a != 0), nb = __ballot_sync(0xffffffffu, b != 0),
                 nc = __ballot_sync(0xffffffffu, c != 0) & ((1u << (kExLimbs - 64)) - 1u);
  const long long flags = __shfl_sync(0xffffffffu, c, kExFlags - 64);
  const int first = na ? __ffs(na) - 1 : nb ? 31 + __ffs(nb) : nc ? 63 + __ffs(nc) : 0;
  const int last = nc ? 95 - __clz(nc) : nb ? 63 - __clz(nb) : na ? 31 - __clz(na) : 0;
  return exact_round([&](int i) { return __shfl_sync(0xffffffffu, i < 32 ? a : i < 64 ? b : c, i & 31); }, first, last,
                     flags);
}

// Where the sums of a walk go (RunSumL).  TableSums: the block table, then the global array, FP64 adds
// in the order in which the warps come.  ExactSums: one accumulator per domain and quantity, the same whatever the
// order.  The sums that fp32 fields are scaled by are exact ones: a last bit that depends on the order turns
// roundings of psi and of the reverse sweep's fields, so two runs of one evaluation differed by 2e-9 in
// the forces, and by 1e-7 where a value of psi beside a nucleus was turned.
template <int NQ, int NSLOT = 128>
struct TableSums {
  DomTable<NQ, NSLOT>& t;
  double* global;
  static constexpr bool kBlock = false;
  __device__ __forceinline__ void add(int l, const double* v) const { dom_table_add(t, l, v, global); }
};
// A warp's first four entries meet those of the other seven in one more butterfly: a big grid of few
// domains otherwise has 8 x as many additions to the same words (320^3, one domain: 165 us without it, 66 with), and
// merging all entries, a scan per entry, costs more than the additions (64^3, 13 domains: 21.5 us against 8.2; with
// block tables of FP64 sums the passes took 66 and 9.4 us).
template <int NQ>
struct BlockSums {
  int label[32];
  double v[NQ][32];
};
template <int NQ>
struct ExactSums {
  BlockSums<NQ>& sm;
  long long* global;  // NQ accumulators per domain
  static constexpr bool kBlock = true;
  __device__ __forceinline__ void add(int l, const double* v) const {
#pragma unroll
    for (int q = 0; q < NQ; ++q) exact_add(global + ((long long)l * NQ + q) * kExWords, v[q]);
  }
};

// Running sums of threads that walk columns across many domains.  A thread that meets a new label parks the
// finished (label, sums) in its own list in shared memory; at the end of the walk the warp goes through the
// lists together, one entry per lane at a time: a butterfly merges lanes of one label, and the leaders hold
// what is added.  Adding to the table on the spot cost a compare-and-swap loop per lane (the table's
// FP64 adds are such loops, and a warp's lanes cross a domain face together), and a butterfly on every
// plane 130 instructions a point.  A thread that meets more than CAP labels adds the rest on the spot.
template <int NQ, int CAP>
struct RunList {
  int label[CAP][256];
  double v[CAP][NQ][256];
};

template <int NQ, int CAP>
struct RunSumL {
  int label, n;
  double v[NQ];
  __device__ __forceinline__ void reset() {
    label = -1;
    n = 0;
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = 0.0;
  }
  // l = -1: nothing to add
  template <class Sums>
  __device__ __forceinline__ void add(int l, const double* x, RunList<NQ, CAP>& list, int tid, const Sums& sums) {
    if (l != label) {
      if (label >= 0) {
        if (n < CAP) {
          list.label[n][tid] = label;
#pragma unroll
          for (int q = 0; q < NQ; ++q) list.v[n][q][tid] = v[q];
          ++n;
        } else {
          sums.add(label, v);
        }
      }
      label = l;
#pragma unroll
      for (int q = 0; q < NQ; ++q) v[q] = x[q];
    } else {
#pragma unroll
      for (int q = 0; q < NQ; ++q) v[q] += x[q];
    }
  }
  // lanes of one label that a butterfly brings together leave the sum with the lower one; fl = -1: none
  static __device__ __forceinline__ void merge(int& fl, double (&v)[NQ], int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int ol = __shfl_xor_sync(0xffffffffu, fl, o);
      const bool same = ol == fl;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const double y = __shfl_xor_sync(0xffffffffu, v[q], o);
        if (same && !(lane & o)) v[q] += y;
      }
      if (same && (lane & o)) fl = -1;
    }
  }
  // every thread of the block (of 256) together
  template <class Sums>
  __device__ __forceinline__ void finish(RunList<NQ, CAP>& list, int tid, const Sums& sums) {
    const int lane = lane_id();
    int cnt = 0;  // entries that the warp has had
    for (int s = -1; s < CAP; ++s) {  // the running entry, then the parked ones
      int fl = label;
      if (s >= 0) {
        fl = s < n ? list.label[s][tid] : -1;
#pragma unroll
        for (int q = 0; q < NQ; ++q) v[q] = fl >= 0 ? list.v[s][q][tid] : 0.0;
        if (!__any_sync(0xffffffffu, fl >= 0)) break;
      }
      merge(fl, v, lane);
      if constexpr (Sums::kBlock) {  // the first four entries of a warp wait for the block's other warps
        const unsigned bal = __ballot_sync(0xffffffffu, fl >= 0);
        const int o = cnt + __popc(bal & ((1u << lane) - 1u));
        cnt += __popc(bal);
        if (fl >= 0 && o < 4) {
          sums.sm.label[4 * (tid >> 5) + o] = fl;
#pragma unroll
          for (int q = 0; q < NQ; ++q) sums.sm.v[q][4 * (tid >> 5) + o] = v[q];
          fl = -1;
        }
      }
      if (fl >= 0) sums.add(fl, v);
    }
    if constexpr (Sums::kBlock) {
      if (lane >= cnt && lane < 4) sums.sm.label[4 * (tid >> 5) + lane] = -1;
      __syncthreads();
      if (tid >= 32) return;
      int fl = sums.sm.label[lane];
#pragma unroll
      for (int q = 0; q < NQ; ++q) v[q] = fl >= 0 ? sums.sm.v[q][lane] : 0.0;
      merge(fl, v, lane);
      if (fl >= 0) sums.add(fl, v);
    }
  }
};

// Weight Z/N that turns a domain's energy partials (each linear in its density for a fixed P)
// into those of the exactly normalised domain; 1 when Z or the measured norm N is not positive.
inline double domain_norm_weight(double Z, double N) { return (Z > 0.0 && N > 0.0) ? Z / N : 1.0; }

}  // namespace rq
