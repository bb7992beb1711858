// vec_stencil.cuh -- 7-point stencil passes on 16-byte vectors of an S^3 field with odd S.
//
// The row pitch S = NN + 1 is odd (the flavours that come here take even NN), so rows start at every alignment and a
// scalar pass spends itself on load instructions: 8 per point, each warp load touching 2-4 lines.  Here a
// thread owns one 16-byte group of consecutive ids (W = 4 floats or 2 doubles) of a plane, whatever rows
// it straddles, and lane l of a warp owns the l-th of 32 consecutive groups.  A neighbour row or plane
// is the same run of ids shifted by +-S or +-S^2, which is off alignment by exactly one element (S^2 = 1
// mod 8; S = 1 or 3 mod 4): one aligned vector load plus one element from the next or previous lane.
// Per W points: five vector loads of the field instead of 5 W scalar ones.
#pragma once
#include "rq_internal.cuh"

namespace rq {

template <typename T> struct Vec { static constexpr int W = 16 / (int)sizeof(T); };

template <typename T> struct alignas(16) Quad {
  T v[Vec<T>::W];
};

template <typename T>
__device__ __forceinline__ Quad<T> ldq(const T* __restrict__ p);
template <>
__device__ __forceinline__ Quad<float> ldq<float>(const float* __restrict__ p) {
  const float4 x = __ldg(reinterpret_cast<const float4*>(p));
  return Quad<float>{{x.x, x.y, x.z, x.w}};
}
template <>
__device__ __forceinline__ Quad<double> ldq<double>(const double* __restrict__ p) {
  const double2 x = __ldg(reinterpret_cast<const double2*>(p));
  return Quad<double>{{x.x, x.y}};
}
template <>
__device__ __forceinline__ Quad<int> ldq<int>(const int* __restrict__ p) {
  const int4 x = __ldg(reinterpret_cast<const int4*>(p));
  return Quad<int>{{x.x, x.y, x.z, x.w}};
}
template <typename T>
__device__ __forceinline__ void stq(T* p, const Quad<T>& q) {
  *reinterpret_cast<Quad<T>*>(p) = q;
}

// A thread's group in plane i: ids a .. a + W - 1.  Lanes 0 and 31 of a warp only load: they hold the groups
// before and after the 30 the warp owns, so a shift's odd element always comes from the next lane (edge
// loads by the end lanes, the other way to get it, cost more L1 passes than the 2 spare lanes).
struct VGroup {
  long long a;
  bool own;  // this thread's to store
};
constexpr int kVOwn = 240;  // groups owned by a block of 256 threads
constexpr int kVecPad = 4;  // elements that a field of 3^3 needs behind it (from 5^3 on loads stay inside)

// groups per plane at most (any alignment of the plane)
template <typename T>
inline unsigned vgroups(const Geo& g) {
  constexpr int W = Vec<T>::W;
  return (unsigned)(((long long)(g.NN - 2) * g.S + (g.NN - 2) + (W - 1)) / W + 1);
}
template <typename T>
inline dim3 vgrid(const Geo& g, int planes) {
  return dim3((vgroups<T>(g) + kVOwn - 1) / kVOwn, (unsigned)((g.NN - 1 + planes - 1) / planes));
}

// Planes per block: 4 where the grid still has 16 blocks per SM (the loads of neighbouring planes then hit
// L1), else 1; with per-domain sums always 4, for fewer block tables to flush.
template <typename T>
inline int vplanes(const Geo& g, bool sums) {
  const dim3 q = vgrid<T>(g, 4);
  return sums || (long long)q.x * q.y >= 16 * 148 ? 4 : 1;
}

// The thread's group of plane i.  The owned groups run from the one that holds (i, 1, 1) to the one that
// holds (i, NN - 1, NN - 1); with one more on either side their +-S and +-S^2 shifts stay inside the
// array (S >= 5; of 3^3 points they reach one element behind it, kVecPad).
template <typename T>
__device__ __forceinline__ VGroup vgroup(const Geo& g, int i, int blk) {
  constexpr int W = Vec<T>::W;
  const int lane = (int)threadIdx.x & 31;
  const int q = blk * kVOwn + ((int)threadIdx.x >> 5) * 30 + lane - 1;
  const long long base = (long long)i * g.S2;
  const long long a0 = (base + g.S + 1) & ~(long long)(W - 1);
  const int n = (int)(base + (long long)(g.NN - 1) * g.S + (g.NN - 1) - a0) / W + 1;
  VGroup r;
  r.own = lane >= 1 && lane <= 30 && q < n;
  r.a = a0 + W * min(q, n);
  return r;
}

// Row and column of the group's first element, for passes without the mask's interior bit
struct VRow {
  int j, k;  // k may wrap to the next row inside the group
};
__device__ __forceinline__ VRow vrow(const Geo& g, const VGroup& r, int i) {
  const unsigned x = (unsigned)(r.a - (long long)i * g.S2);
  const int j = (int)(x / (unsigned)g.S);
  return VRow{j, (int)x - j * g.S};
}
__device__ __forceinline__ bool vinterior(const Geo& g, const VRow& r, int e) {
  int k = r.k + e, j = r.j;
  if (k >= g.S) { k -= g.S; ++j; }
  return k >= 1 && k < g.NN && j >= 1 && j < g.NN;
}

// The group's elements with their bit in `in`, the others as the array holds them
__device__ __forceinline__ void vstore(float* p, const VGroup& r, unsigned in, const Quad<float>& q) {
  if (in == 15u) {
    stq(p + r.a, q);
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (in >> e & 1u) p[r.a + e] = q.v[e];
  }
}

// A field on the group and its six neighbours.  A shift by d = 1 mod W is the aligned group at a + d - 1 and
// the next lane's first element; d = -1 mod W the aligned group at a + d + 1 and the previous lane's last.
// Every load is issued by the constructor of VLoad (the shuffles of vstar would otherwise order them), so
// a thread has all its vectors in flight at once.  LDG: through the read-only path (not for a field the
// pass writes).  ROW: the form of the +-S shifts, kRowP for S = 1 mod 4 (+S is the one taken from the next
// lane), kRowM for 3 mod 4, kRowAny decided at run time by a swap (batches, whose grids differ; the two
// forms side by side cost registers).  For W = 2 both forms are the same shift.
constexpr int kRowP = 1, kRowM = 0, kRowAny = 2;
template <typename T, int ROW, bool LDG = true> struct VLoad {
  Quad<T> ip, im, jn, jv, c;  // jn: the row shift taken from the next lane, jv: from the previous
  bool up;                    // jn is +S
  static __device__ __forceinline__ Quad<T> q(const T* p) {
    if (LDG) return ldq<T>(p);
    return *reinterpret_cast<const Quad<T>*>(p);
  }
  __device__ __forceinline__ VLoad(const T* p, const VGroup& r, const Geo& g) {
    const T* x = p + r.a;
    up = ROW == kRowAny ? (g.S & 3) == 1 : ROW == kRowP;
    const int S = up ? (int)g.S : -(int)g.S, S2 = (int)g.S2;  // 32 bits: one multiply-add per address
    c = q(x);
    ip = q(x + S2 - 1);
    im = q(x - S2 + 1);
    jn = q(x + S - 1);
    jv = q(x - S + 1);
  }
};
template <typename T> struct Star {
  Quad<T> ip, im, jp, jm, kp, km, c;  // +i, -i, +j, -j, +k, -k and the centre
};
template <typename T>
__device__ __forceinline__ Quad<T> vnext(const Quad<T>& q) {  // the run shifted by one element up
  constexpr int W = Vec<T>::W;
  Quad<T> o;
#pragma unroll
  for (int e = 0; e < W - 1; ++e) o.v[e] = q.v[e + 1];
  o.v[W - 1] = __shfl_down_sync(0xffffffffu, q.v[0], 1);
  return o;
}
template <typename T>
__device__ __forceinline__ Quad<T> vprev(const Quad<T>& q) {  // the run shifted by one element down
  constexpr int W = Vec<T>::W;
  Quad<T> o;
#pragma unroll
  for (int e = 1; e < W; ++e) o.v[e] = q.v[e - 1];
  o.v[0] = __shfl_up_sync(0xffffffffu, q.v[W - 1], 1);
  return o;
}
template <typename T, int ROW, bool LDG>
__device__ __forceinline__ Star<T> vstar(const VLoad<T, ROW, LDG>& l) {
  Star<T> s;
  s.c = l.c;
  s.ip = vnext(l.ip);
  s.im = vprev(l.im);
  const Quad<T> n = vnext(l.jn), v = vprev(l.jv);
#pragma unroll
  for (int e = 0; e < Vec<T>::W; ++e) {
    s.jp.v[e] = l.up ? n.v[e] : v.v[e];
    s.jm.v[e] = l.up ? v.v[e] : n.v[e];
  }
  s.kp = vnext(l.c);
  s.km = vprev(l.c);
  return s;
}

// the W bytes of a byte field on the group (a is a multiple of W, so the load is aligned)
template <typename T>
__device__ __forceinline__ unsigned vbytes(const unsigned char* __restrict__ m, const VGroup& r) {
  if (Vec<T>::W == 4) return __ldg(reinterpret_cast<const unsigned*>(m + r.a));
  return __ldg(reinterpret_cast<const unsigned short*>(m + r.a));
}

// the W labels of the group
template <typename T>
__device__ __forceinline__ void vlabels(const int* __restrict__ label, const VGroup& r, int (&l)[Vec<T>::W]) {
  if constexpr (Vec<T>::W == 4) {
    const int4 x = __ldg(reinterpret_cast<const int4*>(label + r.a));
    l[0] = x.x; l[1] = x.y; l[2] = x.z; l[3] = x.w;
  } else {
    const int2 x = __ldg(reinterpret_cast<const int2*>(label + r.a));
    l[0] = x.x; l[1] = x.y;
  }
}

// x / 6 correctly rounded, by the two-constant product of Brisebarre, Muller and Raina ("Accelerating
// correctly rounded floating-point division when the divisor is known in advance", 2004): zh + zl is 1/6
// to twice the precision.  For f32 it equals the division for every mantissa at |x| >= 2^-121 (checked
// exhaustively); smaller, zero and infinite arguments divide.
__device__ __forceinline__ float sixth(float x) {
  constexpr float zh = 0x1.555556p-3f, zl = -0x1.555556p-28f;
  const float a = fabsf(x);
  if (a >= 0x1p-100f && a <= 0x1p126f) return __fmaf_rn(x, zh, __fmul_rn(x, zl));
  return x == 0.0f ? x : F_DIV(x, 6.0f);
}
// For f64: x zh + x zl needs one rounding of a value whose error is far below the distance of x / 6 from any
// midpoint (at least 1/6 ulp), as long as x zl is a normal number; 0, infinities and NaN come out as the
// division's.
__device__ __forceinline__ double sixth_in_range(double x) {
  constexpr double zh = 0x1.5555555555555p-3, zl = 0x1.5555555555555p-57;
  return __fma_rn(x, zh, __dmul_rn(x, zl));
}
__device__ __forceinline__ double sixth(double x) {
  // |x| in [2^-900, 2^1000), by the exponent field: FP64 comparisons are as long a wait as the product
  const unsigned ex = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
  if (ex - (1023u - 900u) < 1900u) return sixth_in_range(x);
  return __ddiv_rn(x, 6.0);
}

}  // namespace rq
