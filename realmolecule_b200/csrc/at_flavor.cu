// at_flavor.cu -- the atom.js per-shell solver (rq_shells_*): one U, W (front) and P field per
// electron shell, the weighted Laplacian div(w grad u), front tracking, and either the
// simultaneous Poisson update or a multigrid Poisson solve per shell (atom.js:1-346).
//
// atom.js updates every field IN PLACE in lexicographic (i, j, k) order: a cell reads the new
// values of its i-1, j-1, k-1 neighbours and the old values of its i+1, j+1, k+1 neighbours.
// That order is kept exactly by two nested hyperplane wavefronts.  The grid is cut into B^3 blocks;
// the blocks of one diagonal bi + bj + bk depend only on the diagonals before (new values) and after
// (old values), so each diagonal is one launch; and inside its block a thread block walks the cell
// planes i + j + k = t in shared memory, one barrier per plane.  The in-place Gauss-Seidel sweeps of
// the Poisson solve are pipelined over the block diagonals: sweep q runs on diagonal tau - 2q in
// launch tau, so all sweeps of a smoothing call (and all shells, which are independent there) share
// one wavefront.  Arithmetic is that of JS numbers: f64 throughout, each Float32Array store rounded
// to f32, in the reference's operation order; only the f64 sums of the normalisation and the
// energies are summed in a different order.
//
// What bounds it: the dependent chain, ~3 N planes per sweep, not bandwidth.  One launch per cell
// plane (the form before) cost 3.7 us a plane for a sweep and 32 us for the cell update, whose
// energy sums were FP64 atomics on one shared word per quantity; a plane inside a block costs a
// barrier and the f64 chain, 220 cycles or 0.11 us (B200).  A physicsStep of two half-space shells at N = 100 with the
// multigrid solve: 12.0 ms in 1880 launches before, 1.56 ms in 131.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/rq.h"
#include "rq_internal.cuh"
#include "vec_stencil.cuh"

namespace rq {

constexpr int kAtMaxShells = 8;

struct AtGeo {
  int N, S;
  long long S2, S3;
};

inline AtGeo at_geo(int N) {
  AtGeo g;
  g.N = N; g.S = N + 1; g.S2 = (long long)g.S * g.S; g.S3 = g.S2 * g.S;
  return g;
}

// Block edge: 16 where the shared tiles of the kernel fit, else 8.  The wavefront of a block of edge B
// has 3B - 2 planes and the grid (3 ceil(n / B) - 2) diagonals, so both cost about 3n barriers; the
// larger block pays fewer launches and halo loads.
constexpr int kAtB = 16;

// Strides of a block's shared tile of (B + 2)^3 values, so that the cells of one plane i + j + k = t
// (a warp: 32 / B values of i, B of j) fall in different banks: R - 1 along j and PS - 1 along i.
template <int B, typename T> struct AtTile;
template <> struct AtTile<16, float> { static constexpr int R = 19, PS = 342; };
template <> struct AtTile<8, float> { static constexpr int R = 10, PS = 130; };
template <> struct AtTile<16, double> { static constexpr int R = 18, PS = 324; };
template <> struct AtTile<8, double> { static constexpr int R = 10, PS = 105; };

struct AtBlock {
  int i0, j0, k0;  // first interior cell
  int ni, nj, nk;  // interior cells per axis (at most B)
};

// block (blockIdx.x -> bi, bj) of diagonal d; false if the diagonal has no such block
template <int B>
__device__ __forceinline__ bool at_block(const AtGeo& g, int d, AtBlock& b) {
  const int n = g.N - 1, nb = (n + B - 1) / B;
  const int bi = (int)blockIdx.x / nb, bj = (int)blockIdx.x % nb, bk = d - bi - bj;
  if (bk < 0 || bk >= nb) return false;
  b.i0 = 1 + bi * B; b.j0 = 1 + bj * B; b.k0 = 1 + bk * B;
  b.ni = min(B, g.N - b.i0); b.nj = min(B, g.N - b.j0); b.nk = min(B, g.N - b.k0);
  return true;
}

// The block's cells and its six face layers of `src` into the tile, a B x B layer per round and thread
// (edges and corners of the halo are not read: those cells may be written by another block of the same
// launch).  All loads are issued before a value is stored.  Taken cell by cell with divisions, one load at a
// time, the tiles' loads and stores were most of a launch: 31 us for a smoothing launch of blocks of 16,
// 14 us now (83 and 34 us for the cell update).
template <int B, typename T>
__device__ __forceinline__ void at_load(T* __restrict__ tile, const float* __restrict__ src, const AtGeo& g,
                                        const AtBlock& b) {
  using L = AtTile<B, T>;
  const int x = (int)threadIdx.x % B, y = (int)threadIdx.x / B;
  const float* base = src + (long long)b.i0 * g.S2 + (long long)b.j0 * g.S + b.k0;
  float v[B + 6];
  const bool jk = y < b.nj && x < b.nk, ik = y < b.ni && x < b.nk, ij = y < b.ni && x < b.nj;
  const float* c = base + (long long)y * g.S + x;                // (i, y, x)
#pragma unroll
  for (int i = 0; i < B; ++i) v[i] = (jk && i < b.ni) ? c[i * g.S2] : 0.0f;
  v[B] = jk ? c[-g.S2] : 0.0f;
  v[B + 1] = jk ? c[b.ni * g.S2] : 0.0f;
  const float* ci = base + (long long)y * g.S2 + x;              // (y, j, x)
  v[B + 2] = ik ? ci[-g.S] : 0.0f;
  v[B + 3] = ik ? ci[(long long)b.nj * g.S] : 0.0f;
  const float* cj = base + (long long)y * g.S2 + (long long)x * g.S;  // (y, x, k)
  v[B + 4] = ij ? cj[-1] : 0.0f;
  v[B + 5] = ij ? cj[b.nk] : 0.0f;
  T* t = tile + (y + 1) * L::R + x + 1;
#pragma unroll
  for (int i = 0; i < B; ++i)
    if (jk && i < b.ni) t[(i + 1) * L::PS] = (T)v[i];
  if (jk) {
    t[0] = (T)v[B];
    t[(b.ni + 1) * L::PS] = (T)v[B + 1];
  }
  if (ik) {
    T* ti = tile + (y + 1) * L::PS + x + 1;
    ti[0] = (T)v[B + 2];
    ti[(b.nj + 1) * L::R] = (T)v[B + 3];
  }
  if (ij) {
    T* tj = tile + (y + 1) * L::PS + (x + 1) * L::R;
    tj[0] = (T)v[B + 4];
    tj[b.nk + 1] = (T)v[B + 5];
  }
}

// the block's interior cells without a halo, B^3 packed
template <int B>
__device__ __forceinline__ void at_load_centre(float* __restrict__ tile, const float* __restrict__ src, const AtGeo& g,
                                               const AtBlock& b) {
  const float* base = src + (long long)b.i0 * g.S2 + (long long)b.j0 * g.S + b.k0;
  const int k = (int)threadIdx.x % B, j = (int)threadIdx.x / B;
  const float* c = base + (long long)j * g.S + k;
  float v[B];
#pragma unroll
  for (int i = 0; i < B; ++i) v[i] = (i < b.ni && j < b.nj && k < b.nk) ? c[i * g.S2] : 0.0f;
#pragma unroll
  for (int i = 0; i < B; ++i) tile[(i * B + j) * B + k] = v[i];
}

template <int B, typename T>
__device__ __forceinline__ void at_store(const T* __restrict__ tile, float* __restrict__ dst, const AtGeo& g,
                                         const AtBlock& b) {
  using L = AtTile<B, T>;
  const int k = (int)threadIdx.x % B, j = (int)threadIdx.x / B;
  if (j >= b.nj || k >= b.nk) return;
  float* c = dst + (long long)b.i0 * g.S2 + (long long)(b.j0 + j) * g.S + (b.k0 + k);
  const T* t = tile + L::PS + (j + 1) * L::R + k + 1;
#pragma unroll
  for (int i = 0; i < B; ++i)
    if (i < b.ni) c[i * g.S2] = (float)t[i * L::PS];
}

struct AtFixed {
  int w[kAtMaxShells];  // the shell's front does not move
};

template <int B>
constexpr size_t at_gs_smem() {
  return sizeof(double) * (B + 2) * AtTile<B, double>::PS + sizeof(float) * B * B * B;
}

// bytes of dynamic shared memory of k_at_cells: U, W (and P with its neighbours, or its centre) per
// shell, K
template <int B>
constexpr size_t at_cells_smem(int nS, bool simultaneous) {
  return sizeof(float) * ((size_t)nS * (simultaneous ? 3 : 2) * (B + 2) * AtTile<B, float>::PS +
                          (size_t)(simultaneous ? 1 : 1 + nS) * B * B * B);
}

// physicsStep's cell body (atom.js:217-315) for every shell on the block diagonal d.
// acc: E_T, E_ee, E_eK (3) then per shell (ET, Eee, EeK, nrm): f64 sums per thread, one atomic per
// block and quantity.  Two half-space shells at N = 100: 297 launches, 9.6 ms, before; 19 launches, 0.65 ms.
template <int B, int NS, bool SIM>
__global__ void __launch_bounds__(B * B) k_at_cells(float* __restrict__ U, float* __restrict__ W, float* __restrict__ P,
                                                    const float* __restrict__ K, AtFixed fixed, AtGeo g, double h,
                                                    double d, int diag, double* __restrict__ acc) {
  using L = AtTile<B, float>;
  constexpr int TS = (B + 2) * L::PS, C3 = B * B * B;
  extern __shared__ float at_sm[];
  AtBlock b;
  if (!at_block<B>(g, diag, b)) return;
  float* sU = at_sm;            // [NS][TS]
  float* sW = sU + NS * TS;     // [NS][TS]
  float* sP = sW + NS * TS;     // SIM: [NS][TS], else [NS][C3]
  float* sK = sP + NS * (SIM ? TS : C3);
#pragma unroll
  for (int m = 0; m < NS; ++m) {
    at_load<B>(sU + m * TS, U + m * g.S3, g, b);
    at_load<B>(sW + m * TS, W + m * g.S3, g, b);
    if (SIM) at_load<B>(sP + m * TS, P + m * g.S3, g, b);
    else at_load_centre<B>(sP + m * C3, P + m * g.S3, g, b);
  }
  at_load_centre<B>(sK, K, g, b);
  __syncthreads();
  const int li = (int)threadIdx.x / B, lj = (int)threadIdx.x % B;
  const bool column = li < b.ni && lj < b.nj;
  const double h2 = h * h, h3 = h * h * h, dt = d * h2, PI = 3.141592653589793, hd = __dmul_rn(0.5, d);
  double eT = 0, eEE = 0, eEK = 0, em[NS][4];
#pragma unroll
  for (int m = 0; m < NS; ++m) em[m][0] = em[m][1] = em[m][2] = em[m][3] = 0.0;
  for (int t = 0; t <= b.ni + b.nj + b.nk - 3; ++t) {
    const int lk = t - li - lj;
    if (column && lk >= 0 && lk < b.nk) {
      const int id = (li + 1) * L::PS + (lj + 1) * L::R + lk + 1;
      const int ip = id + L::PS, im = id - L::PS, jp = id + L::R, jm = id - L::R, kp = id + 1, km = id - 1;
      const int ic = (li * B + lj) * B + lk;
      const double Kc = (double)sK[ic];
      float c[NS];
#pragma unroll
      for (int m = 0; m < NS; ++m) {
        c[m] = 0.0f;
#pragma unroll
        for (int n = 0; n < NS; ++n) {
          if (n != m) c[m] = (float)__dsub_rn((double)c[m], (double)sU[n * TS + id]);
          c[m] = (float)__dmul_rn(0.5, __dadd_rn((double)c[m], (double)sU[m * TS + id]));
        }
      }
#pragma unroll
      for (int m = 0; m < NS; ++m) {
        float* Um = sU + m * TS;
        float* Wm = sW + m * TS;
        const float wip = Wm[ip], wim = Wm[im], wjp = Wm[jp], wjm = Wm[jm], wkp = Wm[kp], wkm = Wm[km];
        if (!fixed.w[m]) {
          const double s6 = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn((double)wip, (double)wim), (double)wjp),
                                                          (double)wjm), (double)wkp), (double)wkm);
          const double lapW = __ddiv_rn(__dsub_rn(s6, __dmul_rn(6.0, (double)Wm[id])), h2);
          const double gwx = __ddiv_rn(__dsub_rn((double)wip, (double)wim), h);
          const double gwy = __ddiv_rn(__dsub_rn((double)wjp, (double)wjm), h);
          const double gwz = __ddiv_rn(__dsub_rn((double)wkp, (double)wkm), h);
          const double gradW = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(gwx, gwx), __dmul_rn(gwy, gwy)), __dmul_rn(gwz, gwz)));
          const double cm = (double)c[m];
          const double a = __dmul_rn(__dmul_rn(__dmul_rn(2.0, dt), fabs(cm)), lapW);
          const double q = __dmul_rn(__dmul_rn(__dmul_rn(9.0, dt), cm), gradW);
          Wm[id] = (float)__dadd_rn((double)Wm[id], __dadd_rn(a, q));
        }
        const double uid = Um[id], wid = Wm[id];
        const float uip = Um[ip], ujp = Um[jp], ukp = Um[kp];
        auto flux = [&](float up, float wp, float um, float wm) {
          const double f1 = __dmul_rn(__dmul_rn(__dsub_rn((double)up, uid), __dadd_rn((double)wp, wid)), 0.5);
          const double f2 = __dmul_rn(__dmul_rn(__dsub_rn(uid, (double)um), __dadd_rn(wid, (double)wm)), 0.5);
          return __dmul_rn(hd, __dsub_rn(f1, f2));
        };
        const double wlap = __dadd_rn(__dadd_rn(flux(uip, wip, Um[im], wim), flux(ujp, wjp, Um[jm], wjm)),
                                      flux(ukp, wkp, Um[km], wkm));
        const double Pc = (double)(SIM ? sP[m * TS + id] : sP[m * C3 + ic]);
        const double pot = __dmul_rn(__dmul_rn(__dmul_rn(dt, __dsub_rn(Kc, __dmul_rn(2.0, Pc))), uid), wid);
        const float unew = (float)__dadd_rn(uid, __dadd_rn(wlap, pot));
        Um[id] = unew;
        // energy where this shell's front dominates (atom.js:258-283)
        const double un = unew;
        const float wc = (float)wid;
        bool dominated = true;
#pragma unroll
        for (int n = 0; n < NS; ++n)
          if (n != m && sW[n * TS + id] >= wc) dominated = false;
        if (dominated && wid > 0.01) {
          bool dip = true, djp = true, dkp = true;
#pragma unroll
          for (int n = 0; n < NS; ++n)
            if (n != m) {
              if (sW[n * TS + ip] >= wip) dip = false;
              if (sW[n * TS + jp] >= wjp) djp = false;
              if (sW[n * TS + kp] >= wkp) dkp = false;
            }
          const double gx = dip ? __dsub_rn((double)uip, un) : 0.0;
          const double gy = djp ? __dsub_rn((double)ujp, un) : 0.0;
          const double gz = dkp ? __dsub_rn((double)ukp, un) : 0.0;
          const double tm = __dmul_rn(__dmul_rn(0.5, __dadd_rn(__dadd_rn(__dmul_rn(gx, gx), __dmul_rn(gy, gy)), __dmul_rn(gz, gz))), h);
          const double eem = __dmul_rn(__dmul_rn(__dmul_rn(Pc, un), un), h3);
          const double ekm = __dmul_rn(__dmul_rn(__dmul_rn(-Kc, un), un), h3);
          eT += tm; eEE += eem; eEK += ekm;
          em[m][0] += tm; em[m][1] += eem; em[m][2] += ekm;
          em[m][3] += __dmul_rn(__dmul_rn(un, un), h3);
        }
        if (SIM) {  // atom.js:286-293
          double rho = 0.0;
#pragma unroll
          for (int n = 0; n < NS; ++n)
            if (n != m) {
              const double un2 = sU[n * TS + id];
              rho = __dadd_rn(rho, __dmul_rn(__dmul_rn(un2, un2), (double)sW[n * TS + id]));
            }
          float* Pm = sP + m * TS;
          const double s6 = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn((double)Pm[ip], (double)Pm[im]), (double)Pm[jp]),
                                                          (double)Pm[jm]), (double)Pm[kp]), (double)Pm[km]);
          const double lapP = __ddiv_rn(__dsub_rn(s6, __dmul_rn(6.0, Pc)), h2);
          const double inc = __dadd_rn(__dmul_rn(dt, lapP), __dmul_rn(__dmul_rn(__dmul_rn(2.0, PI), dt), rho));
          Pm[id] = (float)__dadd_rn(Pc, inc);
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int m = 0; m < NS; ++m) {
    at_store<B>(sU + m * TS, U + m * g.S3, g, b);
    if (!fixed.w[m]) at_store<B>(sW + m * TS, W + m * g.S3, g, b);
    if (SIM) at_store<B>(sP + m * TS, P + m * g.S3, g, b);
  }
  // the block's sums: a butterfly per warp, then one word per warp in shared memory
  __shared__ double red[(B * B + 31) / 32][3 + 4 * NS];
  const int warp = (int)threadIdx.x / 32;
  auto put = [&](int q, double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x % 32 == 0) red[warp][q] = v;
  };
  put(0, eT);
  put(1, eEE);
  put(2, eEK);
#pragma unroll
  for (int m = 0; m < NS; ++m)
#pragma unroll
    for (int q = 0; q < 4; ++q) put(3 + 4 * m + q, em[m][q]);
  __syncthreads();
  for (int q = threadIdx.x; q < 3 + 4 * NS; q += B * B) {
    double v = 0.0;
#pragma unroll
    for (int w = 0; w < (B * B + 31) / 32; ++w) v += red[w][q];
    if (v != 0.0) atomicAdd(&acc[q], v);
  }
}

// rhs of the Poisson problems of shells m0, m0 + 1, .. (blockIdx.y): 2 pi sum_{n != m} U_n^2 W_n
// (atom.js:299-308), interior points
__global__ void k_at_rhs(const float* __restrict__ U, const float* __restrict__ W, float* __restrict__ rhs, int nS, int m0,
                         AtGeo g) {
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = g.N - 1;
  if (q >= n * n * n) return;
  const int m = m0 + blockIdx.y;
  const long long id = (1 + q / (n * n)) * g.S2 + (1 + (q / n) % n) * g.S + 1 + q % n;
  double rho = 0.0;
  for (int s = 0; s < nS; ++s)
    if (s != m) {
      const double u = U[s * g.S3 + id];
      rho = __dadd_rn(rho, __dmul_rn(__dmul_rn(u, u), (double)W[s * g.S3 + id]));
    }
  rhs[blockIdx.y * g.S3 + id] = (float)__dmul_rn(__dmul_rn(2.0, 3.141592653589793), rho);
}

// launch tau of pipelined in-place Gauss-Seidel sweeps (atom.js:127-138): sweep blockIdx.y works on
// the block diagonal tau - 2 blockIdx.y, shell blockIdx.z on its own P and rhs.  The tile holds the
// f32 values widened, so a cell converts once; a thread owns a column (i, j) and walks k.
// Two shells at N = 100, four sweeps: 301 launches of 3.7 us per shell before, 25 of 14 us for both now.
template <int B>
__global__ void __launch_bounds__(B * B) k_at_gs(float* __restrict__ P, const float* __restrict__ rhs, AtGeo g, double h2,
                                                 int tau) {
  using L = AtTile<B, double>;
  extern __shared__ double at_smd[];
  double* sP = at_smd;
  float* sR = reinterpret_cast<float*>(sP + (B + 2) * L::PS);
  AtBlock b;
  if (!at_block<B>(g, tau - 2 * (int)blockIdx.y, b)) return;
  P += blockIdx.z * g.S3;
  rhs += blockIdx.z * g.S3;
  at_load<B>(sP, P, g, b);
  at_load_centre<B>(sR, rhs, g, b);
  __syncthreads();
  const int li = (int)threadIdx.x / B, lj = (int)threadIdx.x % B;
  const bool column = li < b.ni && lj < b.nj;
  int id = (li + 1) * L::PS + (lj + 1) * L::R + 1;
  const float* r = sR + (li * B + lj) * B;
  double pk = column ? sP[id - 1] : 0.0;  // the cell below, as it is now
  for (int t = 0; t <= b.ni + b.nj + b.nk - 3; ++t) {
    const int lk = t - li - lj;
    if (column && lk >= 0 && lk < b.nk) {
      const double f = __dmul_rn(h2, (double)r[lk]);
      const double s6 = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(sP[id + L::PS], sP[id - L::PS]), sP[id + L::R]),
                                                      sP[id - L::R]), sP[id + 1]), pk);
      // f32 values and h^2 times one: 0, or far above 2^-900
      pk = (double)(float)sixth_in_range(__dadd_rn(s6, f));
      sP[id] = pk;
      ++id;
    }
    __syncthreads();
  }
  at_store<B>(sP, P, g, b);
}

// residual res = rhs + lap P (atom.js:173-184) at the points the injection (atom.js:140-153) takes:
// coarse interior (I, J, K) from fine (2I, 2J, 2K); blockIdx.y = shell
__global__ void k_at_restrict(const float* __restrict__ P, const float* __restrict__ rhs, float* __restrict__ coarse,
                              AtGeo g, AtGeo gc, double h2) {
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = gc.N - 1;
  if (q >= n * n * n) return;
  P += blockIdx.y * g.S3;
  rhs += blockIdx.y * g.S3;
  const long long I = 1 + q / (n * n), J = 1 + (q / n) % n, Kc = 1 + q % n;
  const long long id = (2 * I) * g.S2 + (2 * J) * g.S + 2 * Kc;
  const double s6 = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn((double)P[id + g.S2], (double)P[id - g.S2]),
                                                              (double)P[id + g.S]), (double)P[id - g.S]),
                                        (double)P[id + 1]), (double)P[id - 1]);
  const double lap = __ddiv_rn(__dsub_rn(s6, __dmul_rn(6.0, (double)P[id])), h2);
  coarse[blockIdx.y * gc.S3 + I * gc.S2 + J * gc.S + Kc] = (float)__dadd_rn((double)rhs[id], lap);
}

// injection-add prolongation (atom.js:155-171): fine interior point x gets coarse floor(x/2)
// when that is a coarse interior point; blockIdx.y = shell
__global__ void k_at_prolong(const float* __restrict__ Pc, float* __restrict__ P, AtGeo g, AtGeo gc) {
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = g.N - 1;
  if (q >= n * n * n) return;
  const int i = 1 + (int)(q / (n * n)), j = 1 + (int)((q / n) % n), k = 1 + (int)(q % n);
  const int ci = i >> 1, cj = j >> 1, ck = k >> 1;
  if (ci < 1 || ci >= gc.N || cj < 1 || cj >= gc.N || ck < 1 || ck >= gc.N) return;
  const long long id = blockIdx.y * g.S3 + (long long)i * g.S2 + (long long)j * g.S + k;
  P[id] = (float)__dadd_rn((double)P[id], (double)Pc[blockIdx.y * gc.S3 + (long long)ci * gc.S2 + (long long)cj * gc.S + ck]);
}

// sum of U^2 h^3 over the interior of shell blockIdx.y (block sums, then FP64 atomics)
__global__ void __launch_bounds__(256) k_at_norm2(const float* __restrict__ U, AtGeo g, double h3, double* __restrict__ out) {
  __shared__ double red[256];
  const long long n = g.N - 1;
  U += blockIdx.y * g.S3;
  double sum = 0.0;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n * n * n;
       q += (long long)gridDim.x * blockDim.x) {
    const long long id = (1 + q / (n * n)) * g.S2 + (1 + (q / n) % n) * g.S + 1 + q % n;
    const double u = U[id];
    sum += __dmul_rn(__dmul_rn(u, u), h3);
  }
  red[threadIdx.x] = sum;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(out + blockIdx.y, red[0]);
}

// U *= 1/sqrt(n2) on the interior of shell blockIdx.y (atom.js:318-328)
__global__ void k_at_scale(float* __restrict__ U, AtGeo g, const double* __restrict__ n2) {
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = g.N - 1;
  if (q >= n * n * n) return;
  const long long id = blockIdx.y * g.S3 + (1 + q / (n * n)) * g.S2 + (1 + (q / n) % n) * g.S + 1 + q % n;
  const double sc = __ddiv_rn(1.0, __dsqrt_rn(n2[blockIdx.y]));
  U[id] = (float)__dmul_rn((double)U[id], sc);
}

}  // namespace rq

using namespace rq;

struct rq_shells {
  rq_shells_config cfg{};
  std::vector<rq_shell> shells;
  int nS = 0;
  AtGeo g{}, gc{};
  double h = 0;
  float *U = nullptr, *W = nullptr, *P = nullptr, *K = nullptr;
  // of nP shells (1 at least) whose Poisson problems run together: right-hand side, coarse residual and correction
  int nP = 0;
  float *rhs = nullptr, *cd = nullptr, *Pc = nullptr;
  double* acc = nullptr;  // 3 + 4 nS energy sums, then nS norms
  AtFixed fixed{};
  cudaStream_t st = nullptr;
  cudaGraphExec_t graph = nullptr;
  long long launches = 0, graph_launches = 0;
  std::string last_error;
};

#define SCK(call)                                                          \
  do {                                                                     \
    cudaError_t _e = (call);                                               \
    if (_e != cudaSuccess) {                                               \
      s->last_error = std::string(#call) + ": " + cudaGetErrorString(_e);  \
      return _e == cudaErrorMemoryAllocation ? RQ_ENOMEM : RQ_ECUDA;       \
    }                                                                      \
  } while (0)
#define SLAUNCH() SCK(cudaGetLastError()); s->launches++

static unsigned blocks_for(long long n) { return (unsigned)((n + 255) / 256); }

// pipelined Gauss-Seidel: `iters` in-place sweeps of the P of n shells on grid g in one wavefront of
// blocks.  Blocks of 16 as long as a row of blocks is not shorter than the pipeline: with 20 sweeps on a
// coarse grid the launches are mostly the pipeline's 2 (iters - 1), and blocks of 8 (22 planes a launch
// instead of 46) are the shorter chain.
template <int B>
static int at_smooth_b(rq_shells* s, float* P, const float* rhs, int n, const AtGeo& g, double h2, int iters) {
  const int nb = (g.N - 1 + B - 1) / B;
  constexpr size_t smem = at_gs_smem<B>();
  SCK(cudaFuncSetAttribute(k_at_gs<B>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  for (int tau = 0; tau <= 3 * (nb - 1) + 2 * (iters - 1); ++tau) {
    k_at_gs<B><<<dim3(nb * nb, iters, n), B * B, smem, s->st>>>(P, rhs, g, h2, tau);
    SLAUNCH();
  }
  return RQ_OK;
}
static int at_smooth(rq_shells* s, float* P, const float* rhs, int n, const AtGeo& g, double h2, int iters) {
  const int nb = (g.N - 1 + kAtB - 1) / kAtB;
  return 2 * (iters - 1) <= 3 * nb ? at_smooth_b<kAtB>(s, P, rhs, n, g, h2, iters)
                                   : at_smooth_b<8>(s, P, rhs, n, g, h2, iters);
}

// the cell update of every shell, one launch per block diagonal.  Blocks of 16 where the tiles of two
// shells fit one SM's shared memory (164 KB), else blocks of 8 (at most 130 KB for eight shells)
template <int B, int NS, bool SIM>
static int at_cells_b(rq_shells* s) {
  const AtGeo& g = s->g;
  const int nb = (g.N - 1 + B - 1) / B;
  const size_t smem = at_cells_smem<B>(NS, SIM);
  SCK(cudaFuncSetAttribute(k_at_cells<B, NS, SIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  for (int d = 0; d <= 3 * (nb - 1); ++d) {
    k_at_cells<B, NS, SIM><<<nb * nb, B * B, smem, s->st>>>(s->U, s->W, s->P, s->K, s->fixed, g, s->h, s->cfg.d, d, s->acc);
    SLAUNCH();
  }
  return RQ_OK;
}
template <int NS>
static int at_cells_n(rq_shells* s) {
  constexpr int B = NS <= 2 ? kAtB : 8;
  return s->cfg.poisson ? at_cells_b<B, NS, true>(s) : at_cells_b<B, NS, false>(s);
}
static int at_cells(rq_shells* s) {
  switch (s->nS) {
    case 1: return at_cells_n<1>(s);
    case 2: return at_cells_n<2>(s);
    case 3: return at_cells_n<3>(s);
    case 4: return at_cells_n<4>(s);
    case 5: return at_cells_n<5>(s);
    case 6: return at_cells_n<6>(s);
    case 7: return at_cells_n<7>(s);
    default: return at_cells_n<8>(s);
  }
}

// one physicsStep (atom.js:212-343); the energies land in s->acc
static int at_step(rq_shells* s) {
  const AtGeo& g = s->g;
  const unsigned nS = (unsigned)s->nS;
  const long long nint = (long long)(g.N - 1) * (g.N - 1) * (g.N - 1);
  const double h = s->h, h2 = h * h, h3 = h * h * h;
  SCK(cudaMemsetAsync(s->acc, 0, sizeof(double) * (3 + 5 * nS), s->st));
  int rc = at_cells(s);
  if (rc != RQ_OK) return rc;
  // poissonVcycle per shell (atom.js:186-210, :296-310), as many shells together as there are buffers for
  for (int m = 0; !s->cfg.poisson && m < s->nS; m += s->nP) {
    const AtGeo& gc = s->gc;
    const long long ncint = (long long)(gc.N - 1) * (gc.N - 1) * (gc.N - 1);
    const double hc = h * 2, hc2 = hc * hc;
    const int n = std::min(s->nP, s->nS - m);
    float* P = s->P + m * g.S3;
    k_at_rhs<<<dim3(blocks_for(nint), n), 256, 0, s->st>>>(s->U, s->W, s->rhs, s->nS, m, g);
    SLAUNCH();
    if ((rc = at_smooth(s, P, s->rhs, n, g, h2, 4)) != RQ_OK) return rc;
    k_at_restrict<<<dim3(blocks_for(ncint), n), 256, 0, s->st>>>(P, s->rhs, s->cd, g, gc, h2);
    SLAUNCH();
    SCK(cudaMemsetAsync(s->Pc, 0, sizeof(float) * gc.S3 * n, s->st));
    if ((rc = at_smooth(s, s->Pc, s->cd, n, gc, hc2, 20)) != RQ_OK) return rc;
    k_at_prolong<<<dim3(blocks_for(nint), n), 256, 0, s->st>>>(s->Pc, P, g, gc);
    SLAUNCH();
    if ((rc = at_smooth(s, P, s->rhs, n, g, h2, 4)) != RQ_OK) return rc;
  }
  // normalise each shell over the interior
  double* n2 = s->acc + 3 + 4 * nS;
  k_at_norm2<<<dim3(148 * 2, nS), 256, 0, s->st>>>(s->U, g, h3, n2);
  SLAUNCH();
  k_at_scale<<<dim3(blocks_for(nint), nS), 256, 0, s->st>>>(s->U, g, n2);
  SLAUNCH();
  return RQ_OK;
}

// atom.js:55-125 on the host (f64, exp from libm, f32 stores), then uploaded
static void at_init_host(const rq_shells* s, std::vector<float>& U, std::vector<float>& W, std::vector<float>& P,
                         std::vector<float>& K) {
  const int NN = s->cfg.NN, nS = s->nS;
  const long long S3 = s->g.S3, S = s->g.S;
  const double scr = s->cfg.screen, h = s->h, h2 = h * h, h3 = h * h * h;
  const int N2 = NN / 2;
  std::vector<double> Rmin(nS), Rmax(nS);
  Rmin[0] = 0; Rmax[0] = s->shells[0].Rmax;
  for (int m = 1; m < nS; ++m) {
    Rmin[m] = s->shells[m - 1].Rmax;
    Rmax[m] = s->shells[m].Rmax ? s->shells[m].Rmax : scr / 2;
  }
  U.assign(S3 * nS, 0.f); W.assign(S3 * nS, 0.f); P.assign(S3 * nS, 0.f); K.assign(S3, 0.f);
  for (int i = 0; i <= NN; ++i)
    for (int j = 0; j <= NN; ++j)
      for (int k = 0; k <= NN; ++k) {
        const long long id = ((long long)i * S + j) * S + k;
        const double r2 = (double)((i - N2) * (i - N2)) * h2 + (double)((j - N2) * (j - N2)) * h2 +
                          (double)((k - N2) * (k - N2)) * h2 + 0.12 * h2;
        const double r = std::sqrt(r2);
        K[id] = (float)(s->cfg.Z_kernel / r);
        for (int m = 0; m < nS; ++m) {
          const rq_shell& c = s->shells[m];
          bool in;
          float& w = W[m * S3 + id];
          if (c.split) {
            if (i == N2) { in = true; w = 0.5f; }
            else in = c.half_index == 0 ? (i < N2) : (i > N2);
          } else if (c.outer_half) {
            in = r >= Rmin[m] && r < Rmax[m] && i > N2;
          } else {
            in = r >= Rmin[m] && r < Rmax[m];
          }
          if (in) {
            U[m * S3 + id] = (float)std::exp(-c.Zeff * r);
            double wv = 1.0;
            const double smoothW = 2 * h;
            if (!c.split) {
              if (Rmin[m] > 0) { const double din = r - Rmin[m]; if (din < smoothW) wv = std::fmin(wv, din / smoothW); }
              const double dout = Rmax[m] - r;
              if (dout < smoothW) wv = std::fmin(wv, dout / smoothW);
            }
            wv = std::fmax(0.01, wv);
            if (w == 0) w = (float)wv;
          }
        }
        for (int m = 0; m < nS; ++m) P[m * S3 + id] = (float)(0.5 / r);
      }
  for (int m = 0; m < nS; ++m) {
    double n2 = 0;
    for (long long id = 0; id < S3; ++id) n2 += (double)U[m * S3 + id] * U[m * S3 + id] * h3;
    const double sc = 1 / std::sqrt(n2);
    for (long long id = 0; id < S3; ++id) U[m * S3 + id] = (float)(U[m * S3 + id] * sc);
  }
}

extern "C" int rq_shells_create(const rq_shells_config* cfg, const rq_shell* shells, int32_t n_shells, rq_shells** out) {
  if (!cfg || !shells || !out || n_shells < 1 || n_shells > kAtMaxShells) return RQ_EINVAL;
  *out = nullptr;
  if (cfg->NN < 8 || cfg->NN % 2 || cfg->screen <= 0 || cfg->d <= 0 || cfg->poisson < 0 || cfg->poisson > 1)
    return RQ_EINVAL;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return RQ_ENODEV;
  rq_shells* s = new (std::nothrow) rq_shells();
  if (!s) return RQ_ENOMEM;
  s->cfg = *cfg;
  s->shells.assign(shells, shells + n_shells);
  s->nS = n_shells;
  s->g = at_geo(cfg->NN);
  s->gc = at_geo(cfg->NN / 2);
  s->h = cfg->screen / cfg->NN;
  auto fail = [&](int rc) {
    std::fprintf(stderr, "rq_shells_create: %s\n", s->last_error.c_str());
    rq_shells_destroy(s);
    return rc;
  };
  int rc = RQ_OK;
  auto alloc = [&](void** p, size_t bytes) -> int {
    if (cudaMalloc(p, bytes) != cudaSuccess) { *p = nullptr; s->last_error = "cudaMalloc"; return RQ_ENOMEM; }
    if (cudaMemset(*p, 0, bytes) != cudaSuccess) { s->last_error = "cudaMemset"; return RQ_ECUDA; }
    return RQ_OK;
  };
  const size_t S3 = (size_t)s->g.S3, SC3 = (size_t)s->gc.S3;
  if ((rc = alloc((void**)&s->U, sizeof(float) * S3 * n_shells)) || (rc = alloc((void**)&s->W, sizeof(float) * S3 * n_shells)) ||
      (rc = alloc((void**)&s->P, sizeof(float) * S3 * n_shells)) || (rc = alloc((void**)&s->K, sizeof(float) * S3)) ||
      (rc = alloc((void**)&s->acc, sizeof(double) * (3 + 5 * n_shells))))
    return fail(rc);
  // The Poisson buffers: of all shells, or of as many as the memory holds (one shell after the other takes n_shells
  // chains of launches instead of one).
  for (s->nP = cfg->poisson ? 0 : n_shells; s->nP > 0; --s->nP) {
    rc = RQ_OK;
    if (!(rc = alloc((void**)&s->rhs, sizeof(float) * S3 * s->nP)) && !(rc = alloc((void**)&s->cd, sizeof(float) * SC3 * s->nP)) &&
        !(rc = alloc((void**)&s->Pc, sizeof(float) * SC3 * s->nP)))
      break;
    for (float** p : {&s->rhs, &s->cd, &s->Pc}) {
      if (*p) cudaFree(*p);
      *p = nullptr;
    }
    cudaGetLastError();  // the allocation that failed
    if (rc != RQ_ENOMEM) break;
  }
  if (rc != RQ_OK) return fail(rc);
  if (cudaStreamCreateWithFlags(&s->st, cudaStreamNonBlocking) != cudaSuccess) {
    s->last_error = "cudaStreamCreate";
    return fail(RQ_ECUDA);
  }
  for (int m = 0; m < n_shells; ++m) s->fixed.w[m] = shells[m].fixed_w;
  std::vector<float> U, W, P, K;
  at_init_host(s, U, W, P, K);
  if (cudaMemcpy(s->U, U.data(), sizeof(float) * U.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(s->W, W.data(), sizeof(float) * W.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(s->P, P.data(), sizeof(float) * P.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(s->K, K.data(), sizeof(float) * K.size(), cudaMemcpyHostToDevice) != cudaSuccess) {
    s->last_error = "initial upload";
    return fail(RQ_ECUDA);
  }
  *out = s;
  return RQ_OK;
}

extern "C" void rq_shells_destroy(rq_shells* s) {
  if (!s) return;
  if (s->st) cudaStreamSynchronize(s->st);
  if (s->graph) cudaGraphExecDestroy(s->graph);
  for (void* p : {(void*)s->U, (void*)s->W, (void*)s->P, (void*)s->K, (void*)s->rhs, (void*)s->cd, (void*)s->Pc,
                  (void*)s->acc})
    if (p) cudaFree(p);
  if (s->st) cudaStreamDestroy(s->st);
  delete s;
}

extern "C" const char* rq_shells_last_error(const rq_shells* s) { return s ? s->last_error.c_str() : "null"; }

extern "C" int rq_shells_step(rq_shells* s, int32_t n, double* E, double* per_shell) {
  if (!s || n < 0) return RQ_EINVAL;
  for (int q = 0; q < n; ++q) {
    if (!s->graph) {  // one step is always the same launch sequence: captured once, replayed
      const long long l0 = s->launches;
      SCK(cudaStreamBeginCapture(s->st, cudaStreamCaptureModeThreadLocal));
      int rc = at_step(s);
      cudaGraph_t gr = nullptr;
      cudaError_t e = cudaStreamEndCapture(s->st, &gr);
      if (rc != RQ_OK) {
        if (gr) cudaGraphDestroy(gr);
        return rc;
      }
      SCK(e);
      e = cudaGraphInstantiate(&s->graph, gr, 0);
      cudaGraphDestroy(gr);
      SCK(e);
      s->graph_launches = s->launches - l0;
    } else {
      s->launches += s->graph_launches;
    }
    SCK(cudaGraphLaunch(s->graph, s->st));
  }
  const int nS = s->nS;
  std::vector<double> acc(3 + 5 * nS);
  SCK(cudaMemcpyAsync(acc.data(), s->acc, sizeof(double) * acc.size(), cudaMemcpyDeviceToHost, s->st));
  SCK(cudaStreamSynchronize(s->st));
  if (E) {
    E[1] = acc[0]; E[2] = acc[2]; E[3] = acc[1];
    E[0] = E[1] + E[2] + E[3];
  }
  if (per_shell)
    for (int m = 0; m < nS; ++m) {
      double* o = per_shell + 5 * m;
      const double* a = &acc[3 + 4 * m];
      o[0] = a[0]; o[1] = a[1]; o[2] = a[2]; o[3] = a[3];
      o[4] = (a[0] + 2 * a[1] + a[2]) / (a[3] != 0 ? a[3] : 1);  // atom.js:340
    }
  return RQ_OK;
}

extern "C" int rq_shells_download(rq_shells* s, int32_t m, float* U, float* W, float* P) {
  if (!s || m < 0 || m >= s->nS) return RQ_EINVAL;
  const size_t S3 = (size_t)s->g.S3;
  if (U) SCK(cudaMemcpyAsync(U, s->U + m * S3, sizeof(float) * S3, cudaMemcpyDeviceToHost, s->st));
  if (W) SCK(cudaMemcpyAsync(W, s->W + m * S3, sizeof(float) * S3, cudaMemcpyDeviceToHost, s->st));
  if (P) SCK(cudaMemcpyAsync(P, s->P + m * S3, sizeof(float) * S3, cudaMemcpyDeviceToHost, s->st));
  SCK(cudaStreamSynchronize(s->st));
  return RQ_OK;
}

extern "C" int rq_shells_upload(rq_shells* s, int32_t m, const float* U, const float* W, const float* P) {
  if (!s || m < 0 || m >= s->nS) return RQ_EINVAL;
  const size_t S3 = (size_t)s->g.S3;
  if (U) SCK(cudaMemcpyAsync(s->U + m * S3, U, sizeof(float) * S3, cudaMemcpyHostToDevice, s->st));
  if (W) SCK(cudaMemcpyAsync(s->W + m * S3, W, sizeof(float) * S3, cudaMemcpyHostToDevice, s->st));
  if (P) SCK(cudaMemcpyAsync(s->P + m * S3, P, sizeof(float) * S3, cudaMemcpyHostToDevice, s->st));
  SCK(cudaStreamSynchronize(s->st));
  return RQ_OK;
}

extern "C" int rq_shells_info(const rq_shells* s, int64_t* kernel_launches) {
  if (!s) return RQ_EINVAL;
  if (kernel_launches) *kernel_launches = s->launches;
  return RQ_OK;
}
