// nm_bodies.cuh -- device bodies of the new flavour's kernels.
//
// Each body takes its block coordinates explicitly, so the same code runs in two shapes:
// one grid per instance (nm_kernels.cu: the coordinates are blockIdx) and one launch over the
// (instance, tile) work list of a batch of uneven grids (batch_kernels.cu: the coordinates come
// from the work item).  Templated on the field type T (float: mixed path, double: FP64 path);
// point-wise arithmetic is explicitly rounded in the FP64 oracle's operation order
// (oracle/rq_oracle.c, orc_nm_*).
#pragma once
#include "rq_internal.cuh"
#include "vec_stencil.cuh"

namespace rq {

template <typename T> struct Ar;
template <> struct Ar<float> {
  static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
  static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
  static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
  static __device__ __forceinline__ float div(float a, float b) { return __fdiv_rn(a, b); }
};
template <> struct Ar<double> {
  static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
  static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
  static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
  static __device__ __forceinline__ double div(double a, double b) { return __ddiv_rn(a, b); }
};

constexpr int kNmFlatChunk = 16;     // points per thread of the flat (all S^3) bodies
constexpr int kNmRowPlanes = 4;      // planes i per block of the row-tiled multigrid bodies
constexpr int kNmRowTJ = 8;           // rows j per block of the row-tiled bodies (block 32 x 8)
// Thread coordinates of a body written for a block of W threads along x, from the linear thread
// index: the body runs the same under a 2-D launch of that shape and under a 1-D launch of the
// same thread count (the persistent batch kernel).
template <int W>
__device__ __forceinline__ int tile_x() { return (int)((threadIdx.x + blockDim.x * threadIdx.y) % W); }
template <int W>
__device__ __forceinline__ int tile_y() { return (int)((threadIdx.x + blockDim.x * threadIdx.y) / W); }
// March tile of the new flavour's stencil bodies (update, readout, level set): 2^lgk points along
// k x 256 / 2^lgk rows j per block of 256 threads, each thread walking `march` planes of i.  The
// single-grid kernels use kNmTile (16 x 16 x 16: 16 wide rows waste fewer lanes than 32 on the
// 47..127-point interiors of the cluster grids); a batch uses the tile its autotuner picked.
struct NmTile {
  int lgk, march;
};
constexpr int kNmTK = 16, kNmTJ = 16;
constexpr NmTile kNmTile{4, kMarch};
inline dim3 nm_march_grid(const Geo& g, NmTile t = kNmTile) {
  const int n = g.NN - 1, tk = 1 << t.lgk, tj = 256 >> t.lgk;
  return dim3((n + tk - 1) / tk, (n + tj - 1) / tj, (n + t.march - 1) / t.march);
}
inline dim3 nm_march_block() { return dim3(kNmTK, kNmTJ, 1); }
// a thread's column (k, j) and first plane i0 in march tile (bx, by, bz)
__device__ __forceinline__ void nm_tile_origin(const NmTile& t, int bx, int by, int bz, int& k, int& j, int& i0) {
  const int lin = (int)(threadIdx.x + blockDim.x * threadIdx.y);
  k = 1 + (bx << t.lgk) + (lin & ((1 << t.lgk) - 1));
  j = 1 + by * (256 >> t.lgk) + (lin >> t.lgk);
  i0 = 1 + bz * t.march;
}
constexpr int kCoarsestThreads = 256; // one block solves the coarsest level (<= 29^3 points)

// FP64 1/sqrt(x) for x in the normal FP32 range: the FP32 hardware estimate y0 (relative error
// e0 below 2^-21) refined by the binomial series (1 - e)^(-1/2) = 1 + e/2 + 3e^2/8 + O(e^3),
// e = 1 - x y0^2 (Householder's third-order step for the reciprocal square root).  The truncation
// is 5e^3/16 < 1e-18 relative, below FP64 rounding; the FP64 work is five FMA-pipe operations
// where the FP64 reciprocal square root costs a slow-pipe estimate and Newton steps.
__device__ __forceinline__ double rsqrt_refined(double x) {
  const double y0 = (double)rsqrtf((float)x);
  const double e = fma(-x * y0, y0, 1.0);
  return fma(y0 * e, fma(0.375, e, 0.5), y0);
}

// The scale that brings a domain of norm n to its charge Z (1 for an empty or non-finite domain;
// a non-finite norm also sets bit 0 of *err).
__device__ __forceinline__ double nm_domain_scale(double n, double Z, int* err) {
  if (!isfinite(n)) {
    atomicOr(err, 1);
    return 1.0;
  }
  return (Z > 0.0 && n > 1e-300) ? sqrt(Z / n) : 1.0;
}

// Squared distance from which erf(r / (sqrt2 sigma)) is 1 to double precision (r / (sqrt2
// sigma) >= 6: erfc(6) = 2e-17): beyond it a Gaussian nucleus is a point charge.
__device__ __forceinline__ double nm_point_r2(double sigma) { return 72.0 * sigma * sigma; }

// ---------------------------------------------------------------------------------------
// K = sum Z erf(r/(sqrt2 sigma))/r in FP64 (K(0) = Z sqrt(2/pi)/sigma); boundary planes 0.
// One block of 256 threads covers points [blk*256, blk*256+256); sa: 512 doubles of smem.
// K64 (optional): the same sums kept in FP64 (the fp32 fields' readout copy), from the same
// pass.
// ---------------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void nm_potential_body(T* __restrict__ K, const double* __restrict__ at, int nAt,
                                                  const Geo& g, double h, double sigma, long long blk, double* sa,
                                                  double* __restrict__ K64 = nullptr) {
  const long long id = blk * blockDim.x + threadIdx.x;
  const bool inside = id < g.S3;
  int i = 0, j = 0, k = 0;
  if (inside) { i = (int)(id / g.S2); j = (int)((id / g.S) % g.S); k = (int)(id % g.S); }
  const bool interior = inside && i >= 1 && i < g.NN && j >= 1 && j < g.NN && k >= 1 && k < g.NN;
  const double x = i * h, y = j * h, z = k * h;
  const double inv = 1.0 / (1.4142135623730951 * sigma), c0 = 0.7978845608028654 / sigma;  // sqrt(2/pi)
  const double rp2 = nm_point_r2(sigma);
  double v = 0.0;
  for (int base = 0; base < nAt; base += 128) {
    const int cnt = min(128, nAt - base);
    __syncthreads();
    for (int q = threadIdx.x; q < cnt * 4; q += blockDim.x) sa[q] = at[base * 4 + q];
    __syncthreads();
    if (!interior) continue;
    for (int m = 0; m < cnt; ++m) {
      const double Z = sa[m * 4 + 3];
      if (Z <= 0.0) continue;
      const double dx = x - sa[m * 4 + 0], dy = y - sa[m * 4 + 1], dz = z - sa[m * 4 + 2];
      const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
      if (r2 >= rp2) {  // point charge: Z / r
        v = fma(Z, rsqrt_refined(r2), v);
      } else {
        const double r = sqrt(r2);
        v += (r < 1e-12) ? Z * c0 : Z * erf(r * inv) / r;
      }
    }
  }
  if (inside) {
    K[id] = interior ? (T)v : T(0);
    if (K64) K64[id] = interior ? v : 0.0;
  }
}

// initial state: nearest domain seed (f32 squared distances, first wins ties), psi = exp(-d)
template <typename T>
__device__ __forceinline__ void nm_init_body(T* __restrict__ U, int* __restrict__ label,
                                             const float4* __restrict__ seeds, int nSeed, const Geo& g, float h,
                                             long long blk, float4* ss) {
  const long long id = blk * blockDim.x + threadIdx.x;
  const bool inside = id < g.S3;
  int i = 0, j = 0, k = 0;
  if (inside) { i = (int)(id / g.S2); j = (int)((id / g.S) % g.S); k = (int)(id % g.S); }
  const float x = F_MUL((float)i, h), y = F_MUL((float)j, h), z = F_MUL((float)k, h);
  float best = 3.4e38f;
  int bl = 0;
  for (int base = 0; base < nSeed; base += 256) {
    const int cnt = min(256, nSeed - base);
    __syncthreads();
    if (threadIdx.x < cnt) ss[threadIdx.x] = seeds[base + threadIdx.x];
    __syncthreads();
    for (int m = 0; m < cnt; ++m) {
      const float4 s = ss[m];
      const float dx = F_SUB(x, s.x), dy = F_SUB(y, s.y), dz = F_SUB(z, s.z);
      const float d2 = F_ADD(F_ADD(F_MUL(dx, dx), F_MUL(dy, dy)), F_MUL(dz, dz));
      if (d2 < best) { best = d2; bl = __float_as_int(s.w); }
    }
  }
  if (!inside) return;
  const bool interior = i >= 1 && i < g.NN && j >= 1 && j < g.NN && k >= 1 && k < g.NN;
  label[id] = bl;
  U[id] = interior ? (T)exp(-sqrt((double)best)) : T(0);
}

// Unbiased rounding of the fp32 update.  With round-to-nearest, a change of psi smaller than half
// an ulp is lost at every step and the fp32 iteration stops short of the fixed point.  Instead the
// new value is formed exactly in FP64 and rounded down or up with probability proportional to the
// distance to each neighbour, so its expected value is exact.  The uniform variate is a
// counter-based hash of (grid point, step seed) -- the SplitMix64 finaliser (Steele, Lea and Flood,
// OOPSLA 2014) -- so a run is reproducible.
__device__ __forceinline__ unsigned sr_uniform24(unsigned long long id, unsigned seed) {
  unsigned long long x = id * 0x9E3779B97F4A7C15ull + (unsigned long long)seed * 0xD1B54A32D192ED03ull;
  x ^= x >> 30;
  x *= 0xBF58476D1CE4E5B9ull;
  x ^= x >> 27;
  x *= 0x94D049BB133111EBull;
  x ^= x >> 31;
  return (unsigned)(x >> 40);  // 24 bits
}
__device__ __forceinline__ float sr_round(double v, unsigned u24) {
  const float a = __double2float_rz(v);  // the neighbour toward zero
  const double rem = v - (double)a;      // same sign as v, |rem| < the ulp of a
  if (rem == 0.0) return a;
  const float b = nextafterf(a, v > 0.0 ? 3.0e38f : -3.0e38f);  // the neighbour away from zero
  const double frac = rem / ((double)b - (double)a);             // in (0, 1)
  return (double)u24 * 5.9604644775390625e-08 < frac ? b : a;   // u24 / 2^24
}

// One point of the update from its (already selected) neighbours.  With `scaled` the pending per-domain
// scale multiplies the result, formed in FP64 and rounded once; with SR and `rnd` the exact FP64 value is
// rounded without bias.
template <typename T, bool SR>
__device__ __forceinline__ T nm_update_point(T u_c, T a, T b, T c, T d, T e, T f, T kv, T pv, T half_dv, T dt, bool rnd,
                                             unsigned sd, long long id, double scale, bool scaled) {
  using A = Ar<T>;
  const T lap = A::sub(A::add(A::add(A::add(A::add(A::add(a, b), c), d), e), f), A::mul(T(6), u_c));
  if (SR && sizeof(T) == sizeof(float) && rnd) {
    // the same f32 terms, summed exactly in FP64, scaled, then one unbiased rounding
    double v = ((double)u_c + (double)A::mul(half_dv, lap)) + (double)A::mul(A::mul(dt, A::sub(kv, A::mul(T(2), pv))), u_c);
    if (scaled) v *= scale;
    return (T)sr_round(v, sr_uniform24((unsigned long long)id, sd));
  }
  T out = A::add(A::add(u_c, A::mul(half_dv, lap)), A::mul(A::mul(dt, A::sub(kv, A::mul(T(2), pv))), u_c));
  if (scaled) out = (T)((double)out * scale);
  return out;
}

// ITP update (same-label Neumann Laplacian) on the march tile (bx, by, bz); with ACC the FP64
// norm of the new psi per label goes through the block table (caller inits and flushes it).
// With a non-null `scale` the stored psi is one normalisation behind.  The update is linear in
// psi and reads only neighbours of the centre's label (a neighbour of another label is replaced
// by the centre value), so the pending per-domain scale multiplies the result once: psi' =
// scale[label] * update(psi), formed in FP64 and rounded once -- normalise-then-update up to
// rounding, without a separate pass over psi.  With a non-null `seed` (fp32 fields) the stored
// value is rounded without bias (sr_round) from its exact FP64 form.
// SR: the unbiased rounding of fp32 fields (seed non-null), compiled only where it is asked for.
// This form walks a march tile over the labels; the persistent batch launch runs it (its blocks take march
// tiles), every other launch the vector form below.
template <typename T, bool ACC, bool SR = false>
__device__ __forceinline__ void nm_update_body(const T* __restrict__ U, T* __restrict__ Unew, const T* __restrict__ K,
                                               const T* __restrict__ P, const int* __restrict__ label, const Geo& g,
                                               T half_dv, T dt, double h3, int nDom, double* __restrict__ norms,
                                               DomTable<1, 128>& tab, int bx, int by, int bz,
                                               const double* __restrict__ scale = nullptr,
                                               const unsigned* __restrict__ seed = nullptr,
                                               const NmTile t = kNmTile) {
  using A = Ar<T>;
  RunSum<1> rs;
  rs.reset();
  int k, j, i0;
  nm_tile_origin(t, bx, by, bz, k, j, i0);
  if (k < g.NN && j < g.NN && i0 < g.NN) {
    const int iend = min(i0 + t.march, g.NN);
    const long long S = g.S, S2 = g.S2;
    long long id = (long long)i0 * S2 + j * S + k;
    const unsigned sd = (SR && seed) ? __ldg(seed) : 0u;
    T u_m = __ldg(U + id - S2), u_c = __ldg(U + id);
    int l_m = __ldg(label + id - S2), l_c = __ldg(label + id);
    for (int i = i0; i < iend; ++i, id += S2) {
      const T u_p = __ldg(U + id + S2);
      const T ujp = __ldg(U + id + S), ujm = __ldg(U + id - S), ukp = __ldg(U + id + 1), ukm = __ldg(U + id - 1);
      const T kv = __ldg(K + id), pv = __ldg(P + id);
      const int l_p = __ldg(label + id + S2);
      const int ljp = __ldg(label + id + S), ljm = __ldg(label + id - S), lkp = __ldg(label + id + 1),
                lkm = __ldg(label + id - 1);
      const T a = (l_p == l_c) ? u_p : u_c;
      const T b = (l_m == l_c) ? u_m : u_c;
      const T c = (ljp == l_c) ? ujp : u_c;
      const T d = (ljm == l_c) ? ujm : u_c;
      const T e = (lkp == l_c) ? ukp : u_c;
      const T f = (lkm == l_c) ? ukm : u_c;
      const T out = nm_update_point<T, SR>(u_c, a, b, c, d, e, f, kv, pv, half_dv, dt, seed != nullptr, sd, id,
                                           scale ? __ldg(scale + min(max(l_c, 0), nDom - 1)) : 1.0, scale != nullptr);
      Unew[id] = out;
      if (ACC) {
        const double r = (double)out * (double)out * h3;
        rs.add(min(max(l_c, 0), nDom - 1), &r, tab, norms);
      }
      u_m = u_c; u_c = u_p; l_m = l_c; l_c = l_p;
    }
  }
  if (ACC) rs.finish_warp(tab, norms);  // every lane of the block reaches this point
}

// The update on 16-byte groups (vec_stencil.cuh), planes [i0, iend) of block column bx, label equality from
// the same-label mask (nm_mask of the same labels); the labels are read only where a pending scale applies.
// Same values as nm_update_body.  Traffic 17 B per fp32 point.  The norms of a normalising step are a pass
// of their own (nm_norms_body): in this kernel their running sums cost more registers, and so more of the
// loads in flight, than the second read of psi.
template <typename T, bool SR, int ROW>
__device__ __forceinline__ void nm_vupdate_body(const T* __restrict__ U, T* __restrict__ Unew, const T* __restrict__ K,
                                                const T* __restrict__ P, const int* __restrict__ label,
                                                const unsigned char* __restrict__ mask, const Geo& g, T half_dv, T dt,
                                                int nDom, int bx, int i0, int iend, const double* __restrict__ scale,
                                                const unsigned* __restrict__ seed) {
  constexpr int W = Vec<T>::W;
  const unsigned sd = (SR && seed) ? __ldg(seed) : 0u;
  for (int i = i0; i < iend; ++i) {
    const VGroup r = vgroup<T>(g, i, bx);
    const VLoad<T, ROW> lu(U, r, g);
    const Quad<T> kv = ldq<T>(K + r.a), pv = ldq<T>(P + r.a);
    const unsigned mw = vbytes<T>(mask, r);
    int l[W];
    if (scale) vlabels<T>(label, r, l);
    const Star<T> u = vstar(lu);
    Quad<T> un;
#pragma unroll
    for (int e = 0; e < W; ++e) {
      const unsigned m = mw >> (8 * e);
      const T uc = u.c.v[e];
      const T a = (m & kNmIp) ? u.ip.v[e] : uc, b = (m & kNmIm) ? u.im.v[e] : uc;
      const T c = (m & kNmJp) ? u.jp.v[e] : uc, d = (m & kNmJm) ? u.jm.v[e] : uc;
      const T f = (m & kNmKp) ? u.kp.v[e] : uc, q = (m & kNmKm) ? u.km.v[e] : uc;
      const int lc = scale ? min(max(l[e], 0), nDom - 1) : 0;
      const T out = nm_update_point<T, SR>(uc, a, b, c, d, f, q, kv.v[e], pv.v[e], half_dv, dt, seed != nullptr, sd,
                                           r.a + e, scale ? __ldg(scale + lc) : 1.0, scale != nullptr);
      un.v[e] = (m & kNmIn) ? out : T(0);
    }
    if (r.own) stq(Unew + r.a, un);
  }
}

// Same-label neighbour mask of the interior points (kNmIp ..) of plane i, block column bx: the updates read
// it in place of six neighbour labels while the labels do not change.  The face bytes are 0 from the
// allocation.
template <int ROW>
__device__ __forceinline__ void nm_mask_body(const int* __restrict__ label, unsigned char* __restrict__ mask, const Geo& g,
                                             int bx, int i) {
  const VGroup r = vgroup<int>(g, i, bx);
  const Star<int> l = vstar(VLoad<int, ROW>(label, r, g));
  if (!r.own) return;
  const VRow row = vrow(g, r, i);
  unsigned m4 = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int c = l.c.v[e];
    const unsigned m = (l.ip.v[e] == c ? kNmIp : 0) | (l.im.v[e] == c ? kNmIm : 0) | (l.jp.v[e] == c ? kNmJp : 0) |
                       (l.jm.v[e] == c ? kNmJm : 0) | (l.kp.v[e] == c ? kNmKp : 0) | (l.km.v[e] == c ? kNmKm : 0) | kNmIn;
    if (vinterior(g, row, e)) m4 |= m << (8 * e);
  }
  *reinterpret_cast<unsigned*>(mask + r.a) = m4;
}

// U *= scale[label] (FP64 product, rounded once) for labels in [0, nDom) over kNmFlatChunk*256
// points from blk.  With 16-byte aligned fields each thread moves 16-byte vectors of psi (and the
// matching int4 / int2 of labels), kNmFlatChunk points in all; the block covers the same points
// as the scalar walk and every point gets the same product.
template <typename T>
__device__ __forceinline__ void nm_apply_scale_point(T& u, int l, const double* __restrict__ scale, int nDom) {
  if (l >= 0 && l < nDom) u = (T)((double)u * scale[l]);
}

template <typename T>
__device__ __forceinline__ void nm_apply_scale_body(T* __restrict__ U, const int* __restrict__ label,
                                                    const double* __restrict__ scale, long long S3, int nDom,
                                                    long long blk) {
  const long long base = blk * blockDim.x * kNmFlatChunk;
  if ((((unsigned long long)U | (unsigned long long)label) & 15) == 0) {
    constexpr int W = 16 / (int)sizeof(T);  // points per vector
#pragma unroll
    for (int q = 0; q < kNmFlatChunk / W; ++q) {
      const long long e0 = base + ((long long)q * blockDim.x + threadIdx.x) * W;
      if (e0 + W <= S3) {
        if constexpr (sizeof(T) == sizeof(float)) {
          float4 u = *reinterpret_cast<const float4*>(U + e0);
          const int4 l = *reinterpret_cast<const int4*>(label + e0);
          nm_apply_scale_point(u.x, l.x, scale, nDom);
          nm_apply_scale_point(u.y, l.y, scale, nDom);
          nm_apply_scale_point(u.z, l.z, scale, nDom);
          nm_apply_scale_point(u.w, l.w, scale, nDom);
          *reinterpret_cast<float4*>(U + e0) = u;
        } else {
          double2 u = *reinterpret_cast<const double2*>(U + e0);
          const int2 l = *reinterpret_cast<const int2*>(label + e0);
          nm_apply_scale_point(u.x, l.x, scale, nDom);
          nm_apply_scale_point(u.y, l.y, scale, nDom);
          *reinterpret_cast<double2*>(U + e0) = u;
        }
      } else {
        for (long long e = e0; e < S3; ++e) nm_apply_scale_point(U[e], label[e], scale, nDom);
      }
    }
    return;
  }
  for (int q = 0; q < kNmFlatChunk; ++q) {
    const long long id = base + (long long)q * blockDim.x + threadIdx.x;
    if (id >= S3) break;
    nm_apply_scale_point(U[id], label[id], scale, nDom);
  }
}

constexpr int kNmNormAhead = 8, kNmNormCap = 4;
template <class Sm>
struct NormSmem {
  Sm sums;  // DomTable<1, 128> or BlockSums<1>
  RunList<1, kNmNormCap> list;
};
// FP64 per-label psi^2 h^3 over the interior (label clipped to [0, nDom); psi is 0 on the faces): a thread
// walks the planes [i0, iend) of one column of the 32 x 8 tile (bx, by), so it touches the block table about
// once per domain it crosses.  A flat walk, whose points are 256 apart, touched it at every point: 2.14 ms
// against 0.40 ms for the 96 clusters.
template <typename T, class Sums>
__device__ __forceinline__ void nm_norms_body(const T* __restrict__ U, const int* __restrict__ label, const Geo& g,
                                              double h3, int nDom, const Sums& sums, RunList<1, kNmNormCap>& list, int bx,
                                              int by, int i0, int iend) {
  RunSumL<1, kNmNormCap> rs;
  rs.reset();
  const int tid = (int)(threadIdx.x + blockDim.x * threadIdx.y);
  const int k = 1 + bx * 32 + tile_x<32>(), j = 1 + by * 8 + tile_y<32>();
  const bool in = k < g.NN && j < g.NN;
  const long long col = in ? (long long)j * g.S + k : 0;
  for (int i = i0; i < iend; i += kNmNormAhead) {  // the loads of some planes ahead of their sums, whose table
    T u[kNmNormAhead];                             // atomics the compiler does not move loads across
    int l[kNmNormAhead];
#pragma unroll
    for (int q = 0; q < kNmNormAhead; ++q) {
      const long long id = (long long)min(i + q, g.NN) * g.S2 + col;
      u[q] = __ldg(U + id);
      l[q] = __ldg(label + id);
    }
#pragma unroll
    for (int q = 0; q < kNmNormAhead; ++q) {
      const bool on = in && i + q < iend;
      const double r = on ? (double)u[q] * (double)u[q] * h3 : 0.0;
      rs.add(on ? min(max(l[q], 0), nDom - 1) : -1, &r, list, tid, sums);
    }
  }
  rs.finish(list, tid, sums);
}
constexpr int kNmNormPlanes = 16;
inline dim3 nm_norms_grid(const Geo& g) {
  const unsigned n = (unsigned)(g.NN - 1);
  return dim3((n + 31) / 32, (n + 7) / 8, (n + kNmNormPlanes - 1) / kNmNormPlanes);
}

// fine-level right-hand side f = (2 pi psi) psi formed from psi on the fly
template <typename T, bool FINE>
__device__ __forceinline__ T rhs_at(const T* __restrict__ f, long long id) {
  if (FINE) {
    const T u = f[id];
    return Ar<T>::mul(Ar<T>::mul((T)6.283185307179586, u), u);
  }
  return f[id];
}

// One colour of a red-black sweep for A P = f, A P = (6P - sum_6 P)/h^2, on 16-byte groups: planes
// [i0, iend) of block column bx.  S is odd, so i + j + k and the linear id have the same parity and a
// group's elements alternate colours: the pass updates elements COLOR, COLOR + 2 and needs a shuffle only
// for the one whose neighbour is in the next lane.  The pass is in place: it reads points of the other
// colour only, which it does not write, and stores its own one by one.
template <typename T, bool FINE, int ROW, int COLOR>
__device__ __forceinline__ void nm_vrbgs_body(T* __restrict__ P, const T* __restrict__ f, const Geo& g, T h2, int bx,
                                              int i0, int iend) {
  using A = Ar<T>;
  constexpr int W = Vec<T>::W;
  for (int i = i0; i < iend; ++i) {
    const VGroup r = vgroup<T>(g, i, bx);
    const VLoad<T, ROW, false> l(P, r, g);
    const Quad<T> fq = ldq<T>(f + r.a);
    const VRow row = vrow(g, r, i);
    auto next = [&](const Quad<T>& q, int e) { return e + 1 < W ? q.v[(e + 1) % W] : __shfl_down_sync(0xffffffffu, q.v[0], 1); };
    auto prev = [&](const Quad<T>& q, int e) { return e > 0 ? q.v[(e + W - 1) % W] : __shfl_up_sync(0xffffffffu, q.v[W - 1], 1); };
#pragma unroll
    for (int e = COLOR; e < W; e += 2) {
      const T ip = next(l.ip, e), im = prev(l.im, e);
      const T n = next(l.jn, e), v = prev(l.jv, e);
      const T jp = l.up ? n : v, jm = l.up ? v : n;
      const T kp = next(l.c, e), km = prev(l.c, e);
      const T s = A::add(A::add(A::add(A::add(A::add(ip, im), jp), jm), kp), km);
      T rhs = fq.v[e];
      if (FINE) rhs = A::mul(A::mul((T)6.283185307179586, rhs), rhs);
      if (r.own && vinterior(g, row, e)) P[r.a + e] = sixth(A::add(s, A::mul(h2, rhs)));
    }
  }
}

// one colour of a red-black sweep for A P = f, A P = (6P - sum_6 P)/h^2; block (32, 8): each
// thread owns the pair (k0, k0+1) of row j on the kNmRowPlanes planes i from 1 + bz*kNmRowPlanes,
// and on each plane updates the one of the pair that has the colour.  The pass is in place, so
// the compiler may not move a plane's loads above the previous plane's store; they only read
// points of the other colour, which the pass does not change, so all planes' loads are issued
// first (explicitly) and the updates follow.
template <typename T, bool FINE>
__device__ __forceinline__ void nm_rbgs_body(T* __restrict__ P, const T* __restrict__ f, const Geo& g, T h2, int color,
                                             int bx, int by, int bz) {
  using A = Ar<T>;
  const int k0 = 1 + bx * 64 + 2 * tile_x<32>();
  const int j = 1 + by * kNmRowTJ + tile_y<32>();
  const int i0 = 1 + bz * kNmRowPlanes;
  if (j >= g.NN || k0 >= g.NN) return;
  const int iend = min(i0 + kNmRowPlanes, g.NN);
  const long long S = g.S, S2 = g.S2;
  T s[kNmRowPlanes], rhs[kNmRowPlanes];
  long long ids[kNmRowPlanes];
#pragma unroll
  for (int q = 0; q < kNmRowPlanes; ++q) {
    const int i = i0 + q;
    const int k = k0 + ((i + j + k0 + color) & 1);
    ids[q] = (i < iend && k < g.NN) ? (long long)i * S2 + (long long)j * S + k : -1;
    const long long id = ids[q] >= 0 ? ids[q] : S2 + S + 1;  // an interior point: in bounds, not stored
    s[q] = A::add(A::add(A::add(A::add(A::add(P[id + S2], P[id - S2]), P[id + S]), P[id - S]), P[id + 1]), P[id - 1]);
    rhs[q] = rhs_at<T, FINE>(f, id);
  }
#pragma unroll
  for (int q = 0; q < kNmRowPlanes; ++q)
    if (ids[q] >= 0) P[ids[q]] = A::div(A::add(s[q], A::mul(h2, rhs[q])), T(6));
}

// residual f - A P at one interior point from its P values (+i, -i, +j, -j, +k, -k, centre) and
// its right-hand side
template <typename T>
__device__ __forceinline__ T nm_residual_value(T pip, T pim, T pjp, T pjm, T pkp, T pkm, T pc, T rhs, T inv_h2) {
  using A = Ar<T>;
  if (sizeof(T) == sizeof(float)) {
    // fp32 fields: sum_6 P - 6 P cancels most of its digits (P is smooth), so the residual is
    // formed in FP64 from the fp32 values (each operation rounded to nearest) and rounded once --
    // this is what lets the fp32 multigrid reach the fp32 resolution of P instead of stalling at
    // ~1e-4 relative
    const double sd = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn((double)pip, (double)pim), (double)pjp),
                                                    (double)pjm), (double)pkp), (double)pkm);
    return (T)__dadd_rn((double)rhs, __dmul_rn(__dsub_rn(sd, __dmul_rn(6.0, (double)pc)), (double)inv_h2));
  }
  const T s = A::add(A::add(A::add(A::add(A::add(pip, pim), pjp), pjm), pkp), pkm);
  return A::add(rhs, A::mul(A::sub(s, A::mul(T(6), pc)), inv_h2));
}

// residual r = f - A P at one interior point
template <typename T, bool FINE>
__device__ __forceinline__ void nm_residual_point(const T* __restrict__ P, const T* __restrict__ f, T* __restrict__ r,
                                                  long long id, long long S, long long S2, T inv_h2) {
  r[id] = nm_residual_value<T>(P[id + S2], P[id - S2], P[id + S], P[id - S], P[id + 1], P[id - 1], P[id],
                               rhs_at<T, FINE>(f, id), inv_h2);
}

// Row tiling shared by the residual and the prolongation: block (32, 8) covers 64 points of k
// on 8 rows j of the kNmRowPlanes planes from i = 1 + bz*kNmRowPlanes; thread x takes
// k = 1 + 64 bx + x and k + 32 on each plane.  Every point is independent (no dependent chain
// along i), so levels of every size fill the SMs, and each warp load is one contiguous run of 32
// values.
#define NM_ROWS_PROLOGUE                                  \
  const int j = 1 + by * kNmRowTJ + tile_y<32>();        \
  const int tx = tile_x<32>();                            \
  const int i0 = 1 + bz * kNmRowPlanes;                   \
  if (j >= g.NN) return;                                  \
  const int iend = min(i0 + kNmRowPlanes, g.NN);          \
  const long long S = g.S, S2 = g.S2;

template <typename T, bool FINE>
__device__ __forceinline__ void nm_residual_rows_body(const T* __restrict__ P, const T* __restrict__ f,
                                                      T* __restrict__ r, const Geo& g, T inv_h2, int bx, int by,
                                                      int bz) {
  NM_ROWS_PROLOGUE
#pragma unroll
  for (int q = 0; q < kNmRowPlanes; ++q) {
    const int i = i0 + q;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int k = 1 + bx * 64 + tx + 32 * t;
      if (i < iend && k < g.NN)
        nm_residual_point<T, FINE>(P, f, r, (long long)i * S2 + (long long)j * S + k, S, S2, inv_h2);
    }
  }
}

// Trilinear prolongation + correction, P += I E_c, on the row tiling.  A fine point averages the
// 1, 2, 4 or 8 coarse values around it, summed in the order (a, b, c) = (i, j, k) offsets with
// k fastest, then divided by their count.  The i and j parities are uniform over a warp's row;
// only the k parity alternates between lanes, and it selects whether a second value is added.
template <typename T>
__device__ __forceinline__ void nm_prolong_rows_body(const T* __restrict__ Ec, T* __restrict__ P, const Geo& g,
                                                     const Geo& gc, int bx, int by, int bz) {
  using A = Ar<T>;
  NM_ROWS_PROLOGUE
  const int oj = j & 1;
#pragma unroll
  for (int q = 0; q < kNmRowPlanes * 2; ++q) {
    const int i = i0 + (q >> 1);
    const int k = 1 + bx * 64 + tx + 32 * (q & 1);
    if (i >= iend || k >= g.NN) continue;
    const int oi = i & 1;
    const long long row0 = (long long)(i >> 1) * gc.S2 + (long long)(j >> 1) * gc.S;
    const int ck = k >> 1, ok = k & 1;
    T v = T(0);
    auto add_row = [&](long long row) {
      v = A::add(v, Ec[row + ck]);
      if (ok) v = A::add(v, Ec[row + ck + 1]);
    };
    add_row(row0);
    if (oj) add_row(row0 + gc.S);
    if (oi) {
      add_row(row0 + gc.S2);
      if (oj) add_row(row0 + gc.S2 + gc.S);
    }
    v = A::div(v, (T)((1 + oi) * (1 + oj) * (1 + ok)));
    const long long id = (long long)i * S2 + (long long)j * S + k;
    P[id] = A::add(P[id], v);
  }
}
#undef NM_ROWS_PROLOGUE

// The same prolongation by coarse cells: thread (x, y) of a block of 256 owns the cells (I, J, K) =
// (I0 + t, by * 8 + y, bx * 32 + x) for `planes` values of t and updates the 2 x 2 x 2 fine
// points (2I + a, 2J + b, 2K + c) of each that are interior.  A fine point with offsets (a, b, c)
// averages the coarse values (I + da, J + db, K + dc) with da <= a, db <= b, dc <= c, added in
// the (da, db, dc) order of nm_prolong_rows_body and scaled by the exact reciprocal of their
// count, so the result is the row body's bit for bit.  Every load is unconditional (no branch
// on parities) and each coarse plane is loaded once per march: 4 coarse and 8 fine loads and 8
// fine stores per cell.
constexpr int kNmPrTK = 32, kNmPrTJ = 8;
template <typename T>
__device__ __forceinline__ void nm_prolong_cells_body(const T* __restrict__ Ec, T* __restrict__ P, const Geo& g,
                                                      const Geo& gc, int bx, int by, int bz, int planes) {
  using A = Ar<T>;
  const int nc = gc.NN;  // coarse cells 0..nc-1 along each axis cover the fine interior 1..NN-1
  const int K = bx * kNmPrTK + tile_x<32>(), J = by * kNmPrTJ + tile_y<32>();
  if (K >= nc || J >= nc) return;
  const int I0 = bz * planes;
  const int Iend = min(I0 + planes, nc);
  const long long S = g.S, S2 = g.S2, Sc = gc.S, Sc2 = gc.S2;
  T c0[2][2], c1[2][2];  // coarse values of planes I and I + 1: [db][dc]
#pragma unroll
  for (int db = 0; db < 2; ++db)
#pragma unroll
    for (int dc = 0; dc < 2; ++dc) c0[db][dc] = Ec[(long long)I0 * Sc2 + (long long)(J + db) * Sc + K + dc];
  for (int I = I0; I < Iend; ++I) {
#pragma unroll
    for (int db = 0; db < 2; ++db)
#pragma unroll
      for (int dc = 0; dc < 2; ++dc) c1[db][dc] = Ec[(long long)(I + 1) * Sc2 + (long long)(J + db) * Sc + K + dc];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const int i = 2 * I + a;
      if (i < 1) continue;  // the fine boundary plane
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const int j = 2 * J + b;
        if (j < 1) continue;
        const long long row = (long long)i * S2 + (long long)j * S;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int k = 2 * K + c;
          if (k < 1) continue;
          T v = A::add(T(0), c0[0][0]);
          if (c) v = A::add(v, c0[0][1]);
          if (b) {
            v = A::add(v, c0[1][0]);
            if (c) v = A::add(v, c0[1][1]);
          }
          if (a) {
            v = A::add(v, c1[0][0]);
            if (c) v = A::add(v, c1[0][1]);
            if (b) {
              v = A::add(v, c1[1][0]);
              if (c) v = A::add(v, c1[1][1]);
            }
          }
          v = A::mul(v, (T)(1.0 / ((1 + a) * (1 + b) * (1 + c))));
          P[row + k] = A::add(P[row + k], v);
        }
      }
    }
#pragma unroll
    for (int db = 0; db < 2; ++db)
#pragma unroll
      for (int dc = 0; dc < 2; ++dc) c0[db][dc] = c1[db][dc];
  }
}

// full weighting (1/64)(8,4,2,1) at coarse interior point number q; loop order a, b, c
template <typename T>
__device__ __forceinline__ void nm_restrict_body(const T* __restrict__ fine, T* __restrict__ coarse, const Geo& g,
                                                 const Geo& gc, long long q) {
  using A = Ar<T>;
  const int n = gc.NN - 1;
  if (q >= (long long)n * n * n) return;
  const int K2 = 1 + (int)(q % n), J = 1 + (int)((q / n) % n), I = 1 + (int)(q / ((long long)n * n));
  T v = T(0);
  for (int a = -1; a <= 1; ++a)
    for (int b = -1; b <= 1; ++b)
      for (int c = -1; c <= 1; ++c) {
        const T w = (T)((a == 0 ? 2 : 1) * (b == 0 ? 2 : 1) * (c == 0 ? 2 : 1));
        v = A::add(v, A::mul(w, fine[(long long)(2 * I + a) * g.S2 + (long long)(2 * J + b) * g.S + (2 * K2 + c)]));
      }
  coarse[(long long)I * gc.S2 + (long long)J * gc.S + K2] = A::div(v, T(64));
}

// residual r = f - A P on 16-byte groups: planes [i0, iend) of block column bx
template <typename T, bool FINE, int ROW>
__device__ __forceinline__ void nm_vresidual_body(const T* __restrict__ P, const T* __restrict__ f, T* __restrict__ r,
                                                  const Geo& g, T inv_h2, int bx, int i0, int iend) {
  using A = Ar<T>;
  for (int i = i0; i < iend; ++i) {
    const VGroup q = vgroup<T>(g, i, bx);
    const VLoad<T, ROW> l(P, q, g);
    const Quad<T> fq = ldq<T>(f + q.a);
    const Star<T> u = vstar(l);
    const VRow row = vrow(g, q, i);
    Quad<T> o;
#pragma unroll
    for (int e = 0; e < Vec<T>::W; ++e) {
      T rhs = fq.v[e];
      if (FINE) rhs = A::mul(A::mul((T)6.283185307179586, rhs), rhs);
      const T v = nm_residual_value<T>(u.ip.v[e], u.im.v[e], u.jp.v[e], u.jm.v[e], u.kp.v[e], u.km.v[e], u.c.v[e], rhs, inv_h2);
      o.v[e] = vinterior(g, row, e) ? v : T(0);
    }
    if (q.own) stq(r + q.a, o);
  }
}

// full weighting (1/64)(8,4,2,1) of r at the coarse point (K, J) of a 32 x 8 tile on planes I0 .. Iend - 1, in
// the (a, b, c) order of nm_restrict_body; the coarse correction Pc is cleared on the same points
template <typename T>
__device__ __forceinline__ void nm_restrict_tile_body(const T* __restrict__ r, T* __restrict__ fc, T* __restrict__ Pc,
                                                      const Geo& g, const Geo& gc, int bx, int by, int I0, int Iend) {
  using A = Ar<T>;
  const int K = 1 + bx * 32 + tile_x<32>(), J = 1 + by * 8 + tile_y<32>();
  if (K >= gc.NN || J >= gc.NN) return;
  for (int I = I0; I < Iend; ++I) {
    const T* q = r + (long long)(2 * I - 1) * g.S2 + (long long)(2 * J - 1) * g.S + 2 * K - 1;
    T v = T(0);
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int c = 0; c < 3; ++c)
          v = A::add(v, A::mul((T)((a == 1 ? 2 : 1) * (b == 1 ? 2 : 1) * (c == 1 ? 2 : 1)),
                               __ldg(q + a * g.S2 + b * g.S + c)));
    const long long id = (long long)I * gc.S2 + (long long)J * gc.S + K;
    fc[id] = A::mul(v, T(1.0 / 64));
    Pc[id] = T(0);
  }
}

constexpr int kNmRrTK = 32, kNmRrTJ = 8;

// Coarse planes per block of the restriction and prolongation kernels for a launch of
// `blocks_per_plane` blocks on each of n coarse planes: 8, halved while the launch would have
// fewer than 8 blocks per SM (small levels and single grids favour more blocks).
inline int nm_mg_planes(long long blocks_per_plane, int n) {
  int planes = 8;
  while (planes > 1 && blocks_per_plane * ((n + planes - 1) / planes) < 8LL * 148) planes /= 2;
  return planes;
}

// coarsest level: `sweeps` red-black sweeps in FP64 by one block; sm: 2*S^3 doubles of smem
template <typename T>
__device__ __forceinline__ void nm_coarsest_body(T* __restrict__ P, const T* __restrict__ f, const Geo& g, double h2,
                                                 int sweeps, double* sm) {
  double* sP = sm;
  double* sf = sm + g.S3;
  for (long long q = threadIdx.x; q < g.S3; q += blockDim.x) { sP[q] = (double)P[q]; sf[q] = (double)f[q]; }
  __syncthreads();
  const int n = g.NN - 1, S = g.S, S2 = (int)g.S2;  // the coarsest level is at most 29^3 points
  const int nint = n * n * n;
  for (int s = 0; s < sweeps; ++s)
    for (int color = 0; color < 2; ++color) {
      for (int q = threadIdx.x; q < nint; q += blockDim.x) {
        const int k = 1 + q % n, j = 1 + (q / n) % n, i = 1 + q / (n * n);
        if (((i + j + k) & 1) != color) continue;
        const int id = i * S2 + j * S + k;
        const double sum = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(sP[id + S2], sP[id - S2]), sP[id + S]),
                                                        sP[id - S]), sP[id + 1]), sP[id - 1]);
        sP[id] = __ddiv_rn(__dadd_rn(sum, __dmul_rn(h2, sf[id])), 6.0);
      }
      __syncthreads();
    }
  for (long long q = threadIdx.x; q < g.S3; q += blockDim.x) P[q] = (T)sP[q];
}

constexpr int kNmEnergyCap = 2;
template <class Sm>
struct EnergySmem {
  Sm sums;  // DomTable<kNmPD, 128> or BlockSums<kNmPD>
  RunList<kNmPD, kNmEnergyCap> list;
};
// Per-domain readout sums, kNmPD per domain: (norm, T, V_eK, h^3 sum P rho, h^3 sum P (A P)) on the
// march tile, A = -lap_h with Dirichlet faces (the multigrid's operator).  T counts every
// same-label edge with an interior end point once (forward edges + the edge to the Dirichlet face
// on the first layer).  The last sum is attributed to the point's domain only for bookkeeping: the
// readout uses its total in the P-stationary Hartree energy 2 h^3 sum P rho - (h^3 / 2 pi) sum P A P
// (kNmPD, rq_internal.cuh).
// With K64 (fp32 fields) the nuclear term reads the FP64 potential: the fields evolve with the f32
// rounding of K, and reading the energy with the unrounded K removes that rounding from it at first
// order (the state is stationary, so what is left is second order).
template <typename T, class Sums>
__device__ __forceinline__ void nm_energy_body(const T* __restrict__ U, const T* __restrict__ K, const T* __restrict__ P,
                                               const int* __restrict__ label, const Geo& g, double h, int nDom,
                                               const Sums& sums, RunList<kNmPD, kNmEnergyCap>& list, int bx, int by, int bz,
                                               const double* __restrict__ K64 = nullptr, const NmTile t = kNmTile) {
  RunSumL<kNmPD, kNmEnergyCap> rs;
  rs.reset();
  const int tid = (int)(threadIdx.x + blockDim.x * threadIdx.y);
  const double h3 = h * h * h;
  int k, j, i0;
  nm_tile_origin(t, bx, by, bz, k, j, i0);
  const int iend = min(i0 + t.march, g.NN);  // uniform over the block
  const bool col = k < g.NN && j < g.NN;
  const long long S = g.S, S2 = g.S2;
  for (int i = i0; i < iend; ++i) {
    double v[kNmPD] = {};
    int L = -1;
    if (col) {
      const long long id = (long long)i * S2 + j * S + k;
      L = label[id];
      if (L < 0 || L >= nDom) {
        L = -1;
      } else {
        const double u = U[id], rho = u * u;
        const double a = (label[id + S2] == L) ? (double)U[id + S2] - u : 0.0;
        const double b = (label[id + S] == L) ? (double)U[id + S] - u : 0.0;
        const double c = (label[id + 1] == L) ? (double)U[id + 1] - u : 0.0;
        double tt = a * a + b * b + c * c;
        if (i == 1 && label[id - S2] == L) tt += u * u;
        if (j == 1 && label[id - S] == L) tt += u * u;
        if (k == 1 && label[id - 1] == L) tt += u * u;
        const double pc = (double)P[id];
        const double ap = (6.0 * pc - ((double)P[id + S2] + (double)P[id - S2] + (double)P[id + S] + (double)P[id - S] +
                                       (double)P[id + 1] + (double)P[id - 1])) / (h * h);
        const double kv = K64 ? K64[id] : (double)K[id];
        v[0] = rho * h3; v[1] = 0.5 * tt * h; v[2] = -kv * rho * h3; v[3] = pc * rho * h3; v[4] = pc * ap * h3;
      }
    }
    rs.add(L, v, list, tid, sums);
  }
  rs.finish(list, tid, sums);
}

// level-set label update (molecule.js:426-540 rule) on psi of type T, march tile
template <typename T>
__device__ __forceinline__ void nm_evolve_body(const int* __restrict__ labIn, int* __restrict__ labOut,
                                               const T* __restrict__ U, float* __restrict__ W, const Geo& g, T dt_w,
                                               T curvReg, int bx, int by, int bz, const NmTile t = kNmTile) {
  using A = Ar<T>;
  int k, j, i0;
  nm_tile_origin(t, bx, by, bz, k, j, i0);
  if (k >= g.NN || j >= g.NN || i0 >= g.NN) return;
  const int iend = min(i0 + t.march, g.NN);
  const long long S = g.S, S2 = g.S2;
  for (int i = i0; i < iend; ++i) {
    const long long id = (long long)i * S2 + j * S + k;
    const int myL = labIn[id];
    const T uc = U[id];
    const T myRho = A::mul(uc, uc);
    const long long nb[6] = {id + S2, id - S2, id + S, id - S, id + 1, id - 1};
    int bestL = myL;
    T bestRho = T(0), myCnt = T(0);
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const int l = labIn[nb[q]];
      if (l == myL) {
        myCnt = A::add(myCnt, T(1));
      } else {
        const T un = U[nb[q]];
        const T r = A::mul(un, un);
        if (r > bestRho) { bestRho = r; bestL = l; }
      }
    }
    T w = (T)W[id];
    if (myCnt >= T(6)) {
      W[id] = (float)(w > T(1) ? w : T(1));
      labOut[id] = myL;
      continue;
    }
    const T denom = A::add(myRho, bestRho);
    const T vel = (denom < (T)1e-20f) ? T(0) : A::div(A::sub(myRho, bestRho), denom);
    w = A::add(w, A::mul(dt_w, vel));
    const T curv = A::div(A::sub(myCnt, T(3)), T(3));
    w = A::add(w, A::mul(curvReg, curv));
    int newL = myL;
    if (w < T(0)) { newL = bestL; w = (T)0.1f; }
    W[id] = (float)w;
    labOut[id] = newL;
  }
}

// Gaussian-nucleus force gathers.  F_a = f sum_x w(x) (dK_a/dr / Z) (x - R)/r over the interior points,
// with w = rho and f = -h^3 Z (Hellmann-Feynman, gw == nullptr) or w = dE/dK and f = Z (gw given).  The
// pairs split at the Gaussian range (nm_point_r2): beyond it the nucleus is a point charge, dK/dr = -Z/r^2,
// and nm_gather_points_body sums them point by point; within it nm_gather_core_body sums the exact terms
// around each nucleus.  Both form r^2 by the same rounded operations, so every pair is in exactly one.
//
// One thread per nucleus over staged points (the form before) let a warp take the erf/exp branch whenever
// any of its 32 nuclei was close, and left most lanes idle when a grid has few nuclei: 60 ms for the 96
// clusters (<= 36 nuclei on ~112^3 points each), 2 ms now.  Here a thread owns points and all lanes stay
// busy; the point-charge pairs are 12 FP64 operations each, which is what bounds the kernel (64 per SM and
// clock).
__device__ __forceinline__ double nm_grid_coord(int i, double h) { return __dmul_rn((double)i, h); }
__device__ __forceinline__ double nm_pair_r2(double dx, double dy, double dz) {
  return __fma_rn(dx, dx, __fma_rn(dy, dy, __dmul_rn(dz, dz)));
}
template <typename T>
__device__ __forceinline__ double nm_gather_weight(const T* __restrict__ U, const double* __restrict__ gw, long long id) {
  if (gw) return gw[id];
  const double u = (double)U[id];
  return u * u;
}

constexpr int kGaK = 32, kGaJ = 8, kGaI = 16;  // points of a block: a 32 x 8 tile of columns, 16 planes each
constexpr int kGaChunk = 64;                   // nuclei staged at a time
struct GatherSmem {
  double pos[kGaChunk][3], fac[kGaChunk];
  int out[kGaChunk];
  double x[kGaI];
  double sum[8][kGaChunk * 3];  // per warp
  int wc[2];
};

// Point-charge pairs of the points [i0, i1) x [j0, j1) x [k0, k1) (at most 16 x 8 x 32; block of 256)
// with the candidates 0 .. nCand - 1: fetch(m, x, y, z, f) gives a candidate's position and factor f and
// returns its index in F, or -1 for none.  F[3 index + d] += f sum.
template <typename T, class Fetch>
__device__ __forceinline__ void nm_gather_points_body(const T* __restrict__ U, const double* __restrict__ gw,
                                                      const Geo& g, double h, double rp2, int i0, int i1, int j0, int j1,
                                                      int k0, int k1, int nCand, Fetch fetch, double* __restrict__ F,
                                                      GatherSmem& sm) {
  const int tid = (int)(threadIdx.x + blockDim.x * threadIdx.y), lane = tid & 31, warp = tid >> 5;
  const int j = j0 + warp, k = k0 + lane;
  const bool col = j < j1 && k < k1;
  double w[kGaI];
#pragma unroll
  for (int p = 0; p < kGaI; ++p)
    w[p] = (col && i0 + p < i1) ? nm_gather_weight<T>(U, gw, (long long)(i0 + p) * g.S2 + (long long)j * g.S + k) : 0.0;
  const double y = nm_grid_coord(j, h), z = nm_grid_coord(k, h);
  if (tid < kGaI) sm.x[tid] = nm_grid_coord(i0 + tid, h);
  for (int base = 0; base < nCand; base += kGaChunk) {
    double X = 0, Y = 0, Z = 0, f = 0;
    int out = -1;
    if (tid < kGaChunk && base + tid < nCand) out = fetch(base + tid, X, Y, Z, f);
    const unsigned bal = __ballot_sync(0xffffffffu, out >= 0);
    if (lane == 0 && warp < 2) sm.wc[warp] = __popc(bal);
    __syncthreads();
    const int nf = sm.wc[0] + sm.wc[1];
    if (out >= 0) {
      const int o = (warp ? sm.wc[0] : 0) + __popc(bal & ((1u << lane) - 1u));
      sm.pos[o][0] = X; sm.pos[o][1] = Y; sm.pos[o][2] = Z;
      sm.fac[o] = f;
      sm.out[o] = out;
    }
    __syncthreads();
    for (int m = 0; m < nf; ++m) {
      const double Xm = sm.pos[m][0], dy = __dsub_rn(y, sm.pos[m][1]), dz = __dsub_rn(z, sm.pos[m][2]);
      const double c2 = __fma_rn(dy, dy, __dmul_rn(dz, dz));
      double s = 0.0, sx = 0.0;
#pragma unroll
      for (int p = 0; p < kGaI; ++p) {
        const double dx = __dsub_rn(sm.x[p], Xm);
        const double r2 = __fma_rn(dx, dx, c2);
        // r^-3 from the FP32 estimate y0 of r^-1: with e = 1 - r2 y0^2 (y0^2 is exact in FP64) it is
        // y0^3 (1 - e)^(-3/2) = y0^3 (1 + 3e/2 + 15e^2/8 + O(e^3)), |e| < 2^-20
        const double y0 = (double)rsqrtf((float)r2);
        const double y2 = y0 * y0, e = fma(-r2, y2, 1.0), y3 = y2 * y0;
        const double v = w[p] * fma(y3 * e, fma(1.875, e, 1.5), y3);
        const double q = r2 >= rp2 ? v : 0.0;
        s += q;
        sx = fma(q, dx, sx);
      }
      double sy = s * dy, sz = s * dz;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        sx += __shfl_xor_sync(0xffffffffu, sx, o);
        sy += __shfl_xor_sync(0xffffffffu, sy, o);
        sz += __shfl_xor_sync(0xffffffffu, sz, o);
      }
      if (lane == 0) {
        sm.sum[warp][3 * m] = -sx; sm.sum[warp][3 * m + 1] = -sy; sm.sum[warp][3 * m + 2] = -sz;
      }
    }
    __syncthreads();
    for (int q = tid; q < 3 * nf; q += 256) {
      double v = 0.0;
#pragma unroll
      for (int x = 0; x < 8; ++x) v += sm.sum[x][q];
      atomicAdd(&F[3 * sm.out[q / 3] + q % 3], sm.fac[q / 3] * v);
    }
    __syncthreads();
  }
}

// The exact pairs of one nucleus: the interior points within the Gaussian range of (X, Y, Z), shared by
// `parts` blocks of 256.  F[d] += f sum.
template <typename T>
__device__ __forceinline__ void nm_gather_core_body(const T* __restrict__ U, const double* __restrict__ gw, const Geo& g,
                                                    double h, double sigma, double X, double Y, double Z, double f,
                                                    double* __restrict__ F, int part, int parts) {
  __shared__ double red[8][3];
  const double rp2 = nm_point_r2(sigma), rp = sqrt(rp2);
  const double inv = 1.0 / (1.4142135623730951 * sigma), gs = 0.7978845608028654 / sigma, inv2 = inv * inv;
  int lo[3], n[3];
  const double R[3] = {X, Y, Z};
#pragma unroll
  for (int d = 0; d < 3; ++d) {  // one point of slack on either side; the test below decides
    lo[d] = (int)fmin(fmax(floor((R[d] - rp) / h) - 1.0, 1.0), (double)g.NN);
    n[d] = (int)fmin(fmax(ceil((R[d] + rp) / h) + 1.0, 0.0), (double)(g.NN - 1)) - lo[d] + 1;
  }
  double sx = 0, sy = 0, sz = 0;
  if (part == 0 && threadIdx.x == 0) sx = (X - X) + (Y - Y) + (Z - Z);  // NaN for a position that is not finite
  if (n[0] > 0 && n[1] > 0 && n[2] > 0) {
    // unsigned: a grid of more than 2^32 points does not fit the memory, one of more than 2^31 does
    const unsigned nk = (unsigned)n[2], nj = (unsigned)n[1], tot = (unsigned)n[0] * nj * nk;
    for (unsigned q = (unsigned)part * 256 + threadIdx.x; q < tot; q += 256 * parts) {
      const unsigned row = q / nk;
      const int k = lo[2] + (int)(q - row * nk), j = lo[1] + (int)(row % nj), i = lo[0] + (int)(row / nj);
      const double dx = __dsub_rn(nm_grid_coord(i, h), X), dy = __dsub_rn(nm_grid_coord(j, h), Y),
                   dz = __dsub_rn(nm_grid_coord(k, h), Z);
      const double r2 = nm_pair_r2(dx, dy, dz);
      if (r2 >= rp2 || r2 < 1e-24) continue;
      const double r = sqrt(r2);
      const double v = nm_gather_weight<T>(U, gw, (long long)i * g.S2 + (long long)j * g.S + k) *
                       (gs * exp(-r2 * inv2) / r - erf(r * inv) / r2) / r;
      sx = fma(v, dx, sx); sy = fma(v, dy, sy); sz = fma(v, dz, sz);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sx += __shfl_xor_sync(0xffffffffu, sx, o);
    sy += __shfl_xor_sync(0xffffffffu, sy, o);
    sz += __shfl_xor_sync(0xffffffffu, sz, o);
  }
  if (threadIdx.x % 32 == 0) {
    red[threadIdx.x / 32][0] = sx; red[threadIdx.x / 32][1] = sy; red[threadIdx.x / 32][2] = sz;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double v = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) v += red[w][threadIdx.x];
    atomicAdd(&F[threadIdx.x], f * v);
  }
}
constexpr int kGaCoreParts = 4;  // blocks per nucleus of the core gather (19^3 points at sigma = h)

// The two gathers over all entries of one grid (at: x, y, z, Z_nuc per entry; Z_nuc <= 0: no nucleus)
template <typename T>
__device__ __forceinline__ void nm_gather_all_body(const T* __restrict__ U, const double* __restrict__ gw,
                                                   const double* __restrict__ at, int nAt, const Geo& g, double h,
                                                   double sigma, double* __restrict__ F, int bx, int by, int bz,
                                                   GatherSmem& sm) {
  const double scale = gw ? 1.0 : -(h * h * h);
  const int i0 = 1 + bz * kGaI, j0 = 1 + by * kGaJ, k0 = 1 + bx * kGaK;
  const int i1 = min(i0 + kGaI, g.NN), j1 = min(j0 + kGaJ, g.NN), k1 = min(k0 + kGaK, g.NN);
  const double rp2 = nm_point_r2(sigma);
  nm_gather_points_body<T>(U, gw, g, h, rp2, i0, i1, j0, j1, k0, k1, nAt,
                           [&](int m, double& X, double& Y, double& Z, double& f) -> int {
                             const double q = at[m * 4 + 3];
                             X = at[m * 4]; Y = at[m * 4 + 1]; Z = at[m * 4 + 2];
                             f = scale * q;
                             // a nucleus whose range holds all points of the block has no pair here (64^3, 400
                             // nuclei, sigma = 10 h: 1.70 ms with these pairs formed and dropped, 1.19 without);
                             // no range is that wide unless sigma is
                             if (rp2 > 0.25 * h * h * (kGaK * kGaK)) {
                               auto far = [&](double r, int a, int b) {
                                 const double u = nm_grid_coord(a, h) - r, v = nm_grid_coord(b - 1, h) - r;
                                 return fmax(u * u, v * v);
                               };
                               if (far(X, i0, i1) + far(Y, j0, j1) + far(Z, k0, k1) < rp2 * (1.0 - 1e-12)) return -1;
                             }
                             return q > 0.0 ? m : -1;
                           },
                           F, sm);
}
template <typename T>
__device__ __forceinline__ void nm_gather_core_entry(const T* __restrict__ U, const double* __restrict__ gw,
                                                     const double* __restrict__ at, int a, const Geo& g, double h,
                                                     double sigma, double* __restrict__ F, int part) {
  const double q = at[a * 4 + 3];
  if (!(q > 0.0)) return;  // uniform per block
  nm_gather_core_body<T>(U, gw, g, h, sigma, at[a * 4], at[a * 4 + 1], at[a * 4 + 2], (gw ? 1.0 : -(h * h * h)) * q,
                         F + 3 * a, part, kGaCoreParts);
}
inline dim3 nm_gather_grid(const Geo& g) {
  const unsigned n = (unsigned)(g.NN - 1);
  return dim3((n + kGaK - 1) / kGaK, (n + kGaJ - 1) / kGaJ, (n + kGaI - 1) / kGaI);
}

}  // namespace rq
