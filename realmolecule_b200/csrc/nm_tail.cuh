// nm_tail.cuh -- the small levels of the new flavour's V(1,1) cycle, and of its transpose, in one block.
//
// Below ~16 intervals a level is a few thousand points: its six kernels (eight transposed) are launches of
// 2-5 us whose work is a fraction of that, and the coarsest solve waits for all of them.  One block of 1024
// threads runs every level of at most 16 intervals through the coarsest and back in shared memory, a
// barrier where a launch was.  Half a warp takes a row.  Arithmetic and roundings are those of the kernels
// it stands for (nm_vrbgs_body, nm_vresidual_body, nm_restrict_tile_body, nm_prolong_cells_body, nm_coarsest_body; k_adj_half,
// k_adj_other, k_adj_prolong, k_adj_restrict, k_adj_res, k_adj_muf, k_adj_coarsest), bit for bit.
// Bound by the barriers and the dependent FP64 chain of the coarsest sweeps.
#pragma once
#include "nm_bodies.cuh"

namespace rq {

constexpr int kTailNN = 16;     // intervals of the first level at most
constexpr int kTailLevels = 5;  // 16, 8, 4, 2, 1
constexpr int kTailThreads = 1024;
struct NmTail {
  int n;                   // levels, the coarsest last
  int NN[kTailLevels];
  int off[kTailLevels];    // byte offset of the level's arrays (three of T; the coarsest: two of double)
  double h2[kTailLevels];  // squared spacings
  int sweeps;              // of the coarsest level
};

// f(id, i, j, k) for every interior point (color < 0) or those with (i + j + k) % 2 == color of a level of at
// most 16 intervals; half a warp takes a row.  Small code throughout: a pass runs only a few iterations and one
// SM fetches every instruction once (with the loop unrolled by three the cycle's kernel took 28 us at 16 intervals).
template <class F>
__device__ __forceinline__ void tail_map(int NN, int color, F&& f) {
  const int n = NN - 1, S = NN + 1;
  const int hw = (int)threadIdx.x >> 4, lane = (int)threadIdx.x & 15;
  const int total = n * n;
  const unsigned inv = 65536u / (unsigned)n + 1u;  // row / n = (row inv) >> 16 for row < 65536 / n
#pragma unroll 1
  for (int row = hw; row < total; row += kTailThreads / 16) {
    const int i0 = (int)(((unsigned)row * inv) >> 16);
    const int i = 1 + i0, j = 1 + row - i0 * n;
    const int k = color < 0 ? 1 + lane : 1 + ((i + j + 1 + color) & 1) + 2 * lane;
    if (k < NN) f((i * S + j) * S + k, i, j, k);
  }
}

template <typename T>
__device__ __noinline__ void tail_smooth(T* P, const T* f, int NN, T h2) {
  using A = Ar<T>;
  const int S = NN + 1, S2 = S * S;
#pragma unroll 1
  for (int color = 0; color < 2; ++color) {
    tail_map(NN, color, [&](int id, int, int, int) {
      const T s = A::add(A::add(A::add(A::add(A::add(P[id + S2], P[id - S2]), P[id + S]), P[id - S]), P[id + 1]), P[id - 1]);
      P[id] = sixth(A::add(s, A::mul(h2, f[id])));
    });
    __syncthreads();
  }
}

// The coarsest sweeps (of a level of at most 8 intervals, whose colours hold fewer points than the block has
// threads): phase(color, id) for each of `phases` half sweeps of alternating colour, first colour `first`.  Only the warps that hold points take
// part, and a barrier of their own (number 1) separates the phases; the others wait at the block's.
template <class F>
__device__ __forceinline__ void tail_phases(int NN, int phases, int first, F&& phase) {
  const int n = NN - 1, S = NN + 1, hk = (n + 1) / 2;
  const int threads = (n * n * hk + 31) / 32 * 32;
  if ((int)threadIdx.x < threads) {
    const int r = (int)threadIdx.x / hk, kk = (int)threadIdx.x % hk, i = 1 + r / n, j = 1 + r % n;
    int id[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int k = 1 + ((i + j + 1 + c) & 1) + 2 * kk;
      id[c] = (i < NN && k < NN) ? (i * S + j) * S + k : -1;
    }
    for (int s = 0; s < phases; ++s) {
      const int c = (first + s) & 1, q = c ? id[1] : id[0];
      if (q >= 0) phase(s, q);
      asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
    }
  }
  __syncthreads();
}
static_assert((kTailNN / 2 - 1) * (kTailNN / 2 - 1) * (kTailNN / 4) <= kTailThreads, "a point per thread and colour");

// src (global) into a, zeros into b and c; four loads at a time
template <typename T>
__device__ __forceinline__ void tail_input(const T* __restrict__ src, T* a, T* b, T* c, int n) {
#pragma unroll 1
  for (int q = threadIdx.x; q < n; q += 4 * kTailThreads) {
    T v[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = src[min(q + e * kTailThreads, n - 1)];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int x = q + e * kTailThreads;
      if (x < n) { a[x] = v[e]; b[x] = T(0); c[x] = T(0); }
    }
  }
}

// V(1,1) from level 0 of the tail, whose right-hand side is f0 (global); the correction (which starts from
// 0) goes to P0 (global, interior points).
template <typename T>
__global__ void __launch_bounds__(kTailThreads, 1) k_nm_tail(const NmTail t, const T* __restrict__ f0, T* __restrict__ P0) {
  using A = Ar<T>;
  extern __shared__ __align__(16) unsigned char tail_sm[];
  const int last = t.n - 1;
  auto arr = [&](int l, int q) {  // array q (P, f, residual) of level l
    const int S = t.NN[l] + 1;
    return reinterpret_cast<T*>(tail_sm + t.off[l]) + q * S * S * S;
  };
  auto cube = [](int S) { return S * S * S; };
  tail_input<T>(f0, arr(0, 1), arr(0, 0), arr(0, 2), cube(t.NN[0] + 1));
  __syncthreads();
  for (int l = 0; l < last; ++l) {
    const int NN = t.NN[l], S = NN + 1, S2 = S * S, Sc = t.NN[l + 1] + 1;
    T *P = arr(l, 0), *f = arr(l, 1), *r = arr(l, 2);
    tail_smooth<T>(P, f, NN, (T)t.h2[l]);
    const T inv_h2 = (T)(1.0 / t.h2[l]);
    tail_map(NN, -1, [&](int id, int, int, int) {
      r[id] = nm_residual_value<T>(P[id + S2], P[id - S2], P[id + S], P[id - S], P[id + 1], P[id - 1], P[id], f[id], inv_h2);
    });
    // the next level's arrays cleared (faces), then the full weighting into its right-hand side
    double* cd = reinterpret_cast<double*>(tail_sm + t.off[l + 1]);
    if (l + 1 == last) {
      for (int q = threadIdx.x; q < 2 * cube(Sc); q += kTailThreads) cd[q] = 0.0;
    } else {
      for (int q = threadIdx.x; q < 3 * cube(Sc); q += kTailThreads) arr(l + 1, 0)[q] = T(0);
    }
    __syncthreads();
    tail_map(t.NN[l + 1], -1, [&](int id, int I, int J, int K) {
      T v = T(0);
#pragma unroll 1
      for (int ab = 0; ab < 9; ++ab) {
        const int a = ab / 3, b = ab % 3;
        const T* q = r + (2 * I - 1 + a) * S2 + (2 * J - 1 + b) * S + 2 * K - 1;
        const T w = (T)((a == 1 ? 2 : 1) * (b == 1 ? 2 : 1));
        v = A::add(v, A::mul(w, q[0]));
        v = A::add(v, A::mul(w * T(2), q[1]));
        v = A::add(v, A::mul(w, q[2]));
      }
      v = A::mul(v, T(1.0 / 64));
      if (l + 1 == last) cd[cube(Sc) + id] = (double)v;
      else arr(l + 1, 1)[id] = v;
    });
    __syncthreads();
  }
  {  // the coarsest level in FP64
    const int NN = t.NN[last], S = NN + 1, S2 = S * S;
    double* sP = reinterpret_cast<double*>(tail_sm + t.off[last]);
    const double* sf = sP + cube(S);
    const double h2 = t.h2[last];
    auto value = [&](int id) {
      const double sum = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(sP[id + S2], sP[id - S2]), sP[id + S]),
                                                      sP[id - S]), sP[id + 1]), sP[id - 1]);
      return sixth(__dadd_rn(sum, __dmul_rn(h2, sf[id])));
    };
    tail_phases(NN, 2 * t.sweeps, 0, [&](int, int id) { sP[id] = value(id); });
  }
  for (int l = last - 1; l >= 0; --l) {
    const int NN = t.NN[l], Sc = t.NN[l + 1] + 1;
    T *P = arr(l, 0), *f = arr(l, 1);
    const double* cd = reinterpret_cast<const double*>(tail_sm + t.off[l + 1]);
    const T* ce = arr(l + 1, 0);
    tail_map(NN, -1, [&](int id, int i, int j, int k) {
      const int oi = i & 1, oj = j & 1, ok = k & 1;
      int q = ((i >> 1) * Sc + (j >> 1)) * Sc + (k >> 1);
      T v = T(0);
#pragma unroll 1
      for (int a = 0; a <= oi; ++a, q += Sc * Sc)
#pragma unroll 1
        for (int b = 0; b <= oj; ++b) {
          v = A::add(v, l + 1 == last ? (T)cd[q + b * Sc] : ce[q + b * Sc]);
          if (ok) v = A::add(v, l + 1 == last ? (T)cd[q + b * Sc + 1] : ce[q + b * Sc + 1]);
        }
      v = A::mul(v, T(1) / (T)((1 + oi) * (1 + oj) * (1 + ok)));
      P[id] = A::add(P[id], v);
    });
    __syncthreads();
    tail_smooth<T>(P, f, NN, (T)t.h2[l]);
  }
  const T* P = arr(0, 0);
  tail_map(t.NN[0], -1, [&](int id, int, int, int) { P0[id] = P[id]; });
}

// m0 += (1/6) sum_6 m1 on colour 0, in place
template <typename T>
__device__ __forceinline__ double tail_sum6(const T* m, int id, int S, int S2) {
  return (double)m[id + S2] + (double)m[id - S2] + (double)m[id + S] + (double)m[id - S] + (double)m[id + 1] +
         (double)m[id - 1];
}
template <typename T>
__device__ __noinline__ void tail_adj_half(T* m, int NN) {
  const int S = NN + 1, S2 = S * S;
  tail_map(NN, 0, [&](int id, int, int, int) { m[id] = (T)((double)m[id] + sixth(tail_sum6(m, id, S, S2))); });
  __syncthreads();
}

// The transpose of k_nm_tail: mA0 (global) is the adjoint of level 0's P after the cycle, muf0 (global,
// interior points) receives dE/df of level 0.
template <typename T>
__global__ void __launch_bounds__(kTailThreads, 1) k_adj_tail(const NmTail t, const T* __restrict__ mA0, T* __restrict__ muf0) {
  extern __shared__ __align__(16) unsigned char tail_sm[];
  const int last = t.n - 1;
  auto arr = [&](int l, int q) {  // array q (mA, m2, mur) of level l; mA becomes dE/df of the level on the way back
    const int S = t.NN[l] + 1;
    return reinterpret_cast<T*>(tail_sm + t.off[l]) + q * S * S * S;
  };
  auto cube = [](int S) { return S * S * S; };
  tail_input<T>(mA0, arr(0, 0), arr(0, 1), arr(0, 2), cube(t.NN[0] + 1));
  __syncthreads();
  for (int l = 0; l < last; ++l) {
    const int NN = t.NN[l], S = NN + 1, S2 = S * S, Sc = t.NN[l + 1] + 1;
    T *mA = arr(l, 0), *m2 = arr(l, 1);
    tail_adj_half<T>(mA, NN);
    // colour 0 stays 0
    tail_map(NN, 1, [&](int id, int, int, int) { m2[id] = (T)(0.0 + sixth(tail_sum6(mA, id, S, S2))); });
    double* cd = reinterpret_cast<double*>(tail_sm + t.off[l + 1]);
    if (l + 1 == last) {
      for (int q = threadIdx.x; q < 2 * cube(Sc); q += kTailThreads) cd[q] = 0.0;
    } else {
      for (int q = threadIdx.x; q < 3 * cube(Sc); q += kTailThreads) arr(l + 1, 0)[q] = T(0);
    }
    __syncthreads();
    tail_map(t.NN[l + 1], -1, [&](int id, int I, int J, int K) {
      double v = 0.0;
#pragma unroll 1
      for (int ab = 0; ab < 9; ++ab) {
        const int a = ab / 3, b = ab % 3;
        const T* q = m2 + (2 * I - 1 + a) * S2 + (2 * J - 1 + b) * S + 2 * K - 1;
        const double w = (double)((a == 1 ? 2 : 1) * (b == 1 ? 2 : 1));
        v += w * (double)q[0];
        v += 2.0 * w * (double)q[1];
        v += w * (double)q[2];
      }
      const T w = (T)(v / 8.0);
      if (l + 1 == last) cd[id] = (double)w;
      else arr(l + 1, 0)[id] = w;
    });
    __syncthreads();
  }
  {  // the coarsest sweeps transposed, in reverse order
    const int NN = t.NN[last], S = NN + 1, S2 = S * S;
    double* sP = reinterpret_cast<double*>(tail_sm + t.off[last]);
    double* sf = sP + cube(S);
    const double c6 = t.h2[last] / 6.0;
    // Colour c transposed: the other colour gathers sP += (1/6) sum_6 sP, then c's points go into sf and
    // become 0.  The zero and the sum into sf are taken with the point's next gather: half sweep s updates
    // colour s & 1, and at s = 0 its points have not been through sf yet.
    auto value = [&](int s, int id) {
      double own = sP[id];
      const double x = sixth(tail_sum6(sP, id, S, S2));
      if (s > 0) {
        sf[id] = fma(c6, own, sf[id]);
        own = 0.0;
      }
      return own + x;
    };
    tail_phases(NN, 2 * t.sweeps, 0, [&](int s, int id) { sP[id] = value(s, id); });
    tail_map(NN, 0, [&](int id, int, int, int) { sf[id] = fma(c6, sP[id], sf[id]); });
    __syncthreads();
  }
  for (int l = last - 1; l >= 0; --l) {
    const int NN = t.NN[l], S = NN + 1, S2 = S * S, Sc = t.NN[l + 1] + 1;
    T *mA = arr(l, 0), *m2 = arr(l, 1), *mur = arr(l, 2);
    const double* cd = reinterpret_cast<const double*>(tail_sm + t.off[l + 1]) + cube(Sc);
    const T* ce = arr(l + 1, 0);
    tail_map(NN, -1, [&](int id, int i, int j, int k) {
      const int oi = i & 1, oj = j & 1, ok = k & 1;
      int q = ((i >> 1) * Sc + (j >> 1)) * Sc + (k >> 1);
      double v = 0.0;
#pragma unroll 1
      for (int a = 0; a <= oi; ++a, q += Sc * Sc)
#pragma unroll 1
        for (int b = 0; b <= oj; ++b) {
          v += l + 1 == last ? (double)(T)cd[q + b * Sc] : (double)ce[q + b * Sc];
          if (ok) v += l + 1 == last ? (double)(T)cd[q + b * Sc + 1] : (double)ce[q + b * Sc + 1];
        }
      mur[id] = (T)(v * (0.125 / (double)((1 + oi) * (1 + oj) * (1 + ok))));
    });
    __syncthreads();
    const double inv_h2 = 1.0 / t.h2[l], c6 = t.h2[l] / 6.0;
    tail_map(NN, -1, [&](int id, int, int, int) {
      m2[id] = (T)((double)m2[id] + (tail_sum6(mur, id, S, S2) - 6.0 * (double)mur[id]) * inv_h2);
    });
    __syncthreads();
    tail_adj_half<T>(m2, NN);
    tail_map(NN, -1, [&](int id, int, int, int) {
      T f = (T)(c6 * (double)mA[id]);
      f = (T)((double)f + (double)mur[id]);
      f = (T)fma(c6, (double)m2[id], (double)f);
      if (l == 0) muf0[id] = f;
      else mA[id] = f;
    });
    __syncthreads();
  }
}

// The tail of a hierarchy of `levels` levels (NN and spacing of each): from the first level, at least 1, of at
// most 16 intervals, or none (t.n = 0) if fewer than two levels are that small.  Returns that level, or
// `levels`.  Levels above 16 intervals stay kernels: one SM takes longer over them than the launches cost (at 24
// intervals 48 us for the tail against 17 us from 16).
template <typename T, class GeoAt, class HAt>
inline int nm_tail_plan(int levels, GeoAt geo, HAt h, int sweeps, NmTail& t, size_t& smem) {
  t.n = 0;
  t.sweeps = sweeps;
  int first = 1;
  while (first < levels && geo(first).NN > kTailNN) ++first;
  if (first + 1 >= levels) return levels;
  size_t off = 0;
  t.n = levels - first;
  for (int l = first; l < levels; ++l) {
    const Geo g = geo(l);
    t.NN[l - first] = g.NN;
    t.h2[l - first] = h(l) * h(l);
    t.off[l - first] = (int)off;
    off += l == levels - 1 ? 2 * sizeof(double) * (size_t)g.S3 : (3 * sizeof(T) * (size_t)g.S3 + 15) / 16 * 16;
  }
  smem = off;  // at most 3 x 8 (17^3 + 9^3 + 5^3 + 3^3) bytes, 136 KB
  return first;
}

}  // namespace rq
