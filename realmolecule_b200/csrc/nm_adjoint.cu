// nm_adjoint.cu -- gradient of the new flavour's energy readout with respect to the nuclear
// positions and an external potential, by a reverse sweep through the last recorded steps.
//
// One forward step s of the new flavour (nm_flavor.cu) acts on the normalised state as
//   [V-cycle]    P <- M P + B f,  f = 2 pi psi^2                 (every poisson_interval steps)
//   update       psi~ = A psi,  A = I + half_dv L + dt diag(K - 2P)   (L: same-label Laplacian)
//   [normalise]  psi = c psi~,  c_d = sqrt(Z_d / (h^3 sum_d psi~^2))
// and the readout is E = sum_d w_d (T_d + V_eK,d + 2 h^3 sum_d P rho) - (h^3 / 2 pi) sum P (A_h P),
// w_d = Z_d / N_d, A_h = -lap_h (the P-stationary Hartree form), with K = K_nuclei(R) + v.
// The reverse sweep starts from dE/dpsi, dE/dP and dE/dK of the readout and applies the
// transposes step by step, newest first:
//   normalise^T  lam <- c (lam - (h^3 / Z) psi <psi, lam>_d)
//   update^T     lam <- A lam (A is symmetric: L is the same-label graph Laplacian with Dirichlet
//                faces), dE/dK += dt psi lam, dE/dP += -2 dt psi lam
//   V-cycle^T    the smoothing colours, the residual, full weighting and trilinear prolongation
//                transposed in reverse order (full weighting^T = prolongation / 8), the coarsest
//                sweeps in reverse; this gives dE/dP before the cycle and dE/df, and
//                lam += 4 pi psi dE/df.
// The labels are integers and held fixed; the state the window starts from is held fixed (a
// warm start).  F_a = -dE/dR_a is then the Hellmann-Feynman-shaped gather with the weight dE/dK
// in place of -h^3 rho (nm_gather_points_body); with no recorded step dE/dK = -h^3 rho and the force is
// the Hellmann-Feynman force, exact at a converged state.  dE/dv = dE/dK.
//
// The reference computes forces with the Hellmann-Feynman integral of its own softened nuclei
// (cloud/solver.py:282-315 computeForceAll, molecule.js:1271-1330) or the Hartree-gradient ball
// (molecule.js:1200-1269); this is the exact derivative of the discrete energy the new flavour
// actually reaches after a finite number of warm-started iterations.
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <cstring>

#include "nm_tail.cuh"
#include "rq_flavors.h"
#include "rq_kernels.h"
#include "vec_stencil.cuh"

using namespace rq;

#define CK(call)                                 \
  do {                                           \
    int _rc = rq_cuda(c, (call), #call);         \
    if (_rc != RQ_OK) return _rc;                \
  } while (0)

namespace {

unsigned nblk(long long n, long long b = 256) { return (unsigned)((n + b - 1) / b); }

// interior point number q -> (i, j, k) and its linear index
struct Pt {
  int i, j, k;
  long long id;
};
// Interior point of a 3-D launch (grid3 / kBlk3): x runs along k, y along j, z is the plane i.  No
// integer division per point, and a block's threads read contiguous rows.
constexpr int kB3x = 64, kB3y = 4;
__device__ __forceinline__ bool interior_pt3(const Geo& g, Pt& p) {
  p.k = 1 + (int)(blockIdx.x * kB3x + threadIdx.x);
  p.j = 1 + (int)(blockIdx.y * kB3y + threadIdx.y);
  p.i = 1 + (int)blockIdx.z;
  p.id = (long long)p.i * g.S2 + (long long)p.j * g.S + p.k;
  return p.k < g.NN && p.j < g.NN && p.i < g.NN;
}
inline dim3 grid3(const Geo& g) {
  const unsigned n = (unsigned)(g.NN - 1);
  return dim3((n + kB3x - 1) / kB3x, (n + kB3y - 1) / kB3y, n);
}
const dim3 kBlk3(kB3x, kB3y, 1);

// dE/dpsi, dE/dP and dE/dK of the readout at psi (nm_energy: E = sum_d w_d Q_d - (h^3 / 2 pi) <P, A P>,
// Q_d = T_d + V_eK,d + 2 h^3 sum_d P rho, w_d = Z_d / N_d).  wq: per domain (w, Q/N).  T = h/2 sum
// over same-label edges (psi_a - psi_b)^2 (edges to a Dirichlet face included), so dT/dpsi = -h L psi
// with the update's Laplacian; dE/dP = 2 w h^3 rho - (h^3 / pi) A P.
template <typename T>
__global__ void __launch_bounds__(256) k_adj_seed(const T* __restrict__ U, const T* __restrict__ K,
                                                  const T* __restrict__ P, const int* __restrict__ label, Geo g,
                                                  double h, int nDom, const double* __restrict__ wq,
                                                  T* __restrict__ lam, T* __restrict__ muP, double* __restrict__ gK,
                                                  const double* __restrict__ K64) {
  Pt p;
  if (!interior_pt3(g, p)) return;
  const long long id = p.id, S = g.S, S2 = g.S2;
  const int L = label[id];
  if (L < 0 || L >= nDom) {
    lam[id] = T(0);
    muP[id] = T(0);
    gK[id] = 0.0;
    return;
  }
  const double h3 = h * h * h, u = (double)U[id];
  const long long nb[6] = {id + S2, id - S2, id + S, id - S, id + 1, id - 1};
  double lap = 0.0;
#pragma unroll
  for (int t = 0; t < 6; ++t)
    if (label[nb[t]] == L) lap += (double)U[nb[t]] - u;
  const double w = wq[2 * L], qn = wq[2 * L + 1];
  const double pc = (double)P[id];
  const double ap = (6.0 * pc - ((double)P[id + S2] + (double)P[id - S2] + (double)P[id + S] + (double)P[id - S] +
                                 (double)P[id + 1] + (double)P[id - 1])) / (h * h);
  const double kv = K64 ? K64[id] : (double)K[id];  // the readout's K (nm_energy_body)
  lam[id] = (T)(w * (-h * lap + 2.0 * h3 * u * (2.0 * pc - kv - qn)));
  muP[id] = (T)(2.0 * w * h3 * u * u - h3 / M_PI * ap);
  gK[id] = -w * h3 * u * u;
}

// per-domain <psi, lam> in FP64 over the interior (both are 0 on the faces), by columns as nm_norms_body
template <typename T>
__global__ void __launch_bounds__(256) k_adj_dot(const T* __restrict__ psi, const T* __restrict__ lam,
                                                 const int* __restrict__ label, Geo g, int nDom,
                                                 long long* __restrict__ dots) {
  __shared__ NormSmem<BlockSums<1>> sm;
  const ExactSums<1> sums{sm.sums, dots};
  RunSumL<1, kNmNormCap> rs;
  rs.reset();
  const int tid = (int)threadIdx.x, k = 1 + (int)blockIdx.x * 32 + (tid & 31), j = 1 + (int)blockIdx.y * 8 + (tid >> 5);
  const int i0 = 1 + (int)blockIdx.z * kNmNormPlanes, iend = min(i0 + kNmNormPlanes, g.NN);
  const bool in = k < g.NN && j < g.NN;
  const long long col = in ? (long long)j * g.S + k : 0;
  constexpr int AH = 4;  // planes loaded ahead of their sums
  for (int i = i0; i < iend; i += AH) {
    T p[AH], q[AH];
    int l[AH];
#pragma unroll
    for (int t = 0; t < AH; ++t) {
      const long long id = (long long)min(i + t, g.NN) * g.S2 + col;
      p[t] = __ldg(psi + id);
      q[t] = __ldg(lam + id);
      l[t] = __ldg(label + id);
    }
#pragma unroll
    for (int t = 0; t < AH; ++t) {
      const bool on = in && i + t < iend && l[t] >= 0 && l[t] < nDom;
      const double v = on ? (double)p[t] * (double)q[t] : 0.0;
      rs.add(on ? l[t] : -1, &v, sm.list, tid, sums);
    }
  }
  rs.finish(sm.list, tid, sums);
}

// per-domain (c, beta) of a transposed normalisation: c = the forward scale, beta = c h^3 <psi, lam> / Z; a warp
// per domain
__global__ void __launch_bounds__(128) k_adj_norm_coef(const double* __restrict__ scale, const double* __restrict__ Zdom,
                                                       const long long* __restrict__ dots, int nDom, double h3,
                                                       double* __restrict__ coef) {
  const int d = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (d >= nDom) return;
  const double dot = exact_value_warp(dots + (long long)d * kExWords);
  if (threadIdx.x % 32 != 0) return;
  const double c = scale[d], Z = Zdom[d];
  coef[2 * d] = c;
  coef[2 * d + 1] = Z > 0.0 ? c * h3 * dot / Z : 0.0;
}

// the transposed normalisation lam <- c lam - beta psi_s with the domain's (c, beta), rounded to T, in place.  A
// pass of its own: folded into the update below it was redone for six neighbours per point and doubled the
// update's vectors (114 us on 192^3 for 24 + 30 us).
template <typename T>
__global__ void __launch_bounds__(256) k_adj_apply(T* __restrict__ lam, const T* __restrict__ psi_s,
                                                   const int* __restrict__ label, const double* __restrict__ coef,
                                                   long long S3, int nDom) {
  constexpr int W = Vec<T>::W;
  const long long a = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * W;
  auto value = [&](T x, T p, int l) {
    return l >= 0 && l < nDom ? (T)(coef[2 * l] * (double)x - coef[2 * l + 1] * (double)p) : x;
  };
  if (a + W <= S3) {
    Quad<T> x = *reinterpret_cast<const Quad<T>*>(lam + a);
    const Quad<T> p = ldq<T>(psi_s + a);
    int l[W];
    VGroup r;
    r.a = a;
    vlabels<T>(label, r, l);
#pragma unroll
    for (int e = 0; e < W; ++e) x.v[e] = value(x.v[e], p.v[e], l[e]);
    stq(lam + a, x);
  } else {
    for (long long id = a; id < S3; ++id) lam[id] = value(lam[id], psi_s[id], label[id]);
  }
}

// update^T on 16-byte groups: out = A(K, P) in
template <typename T, int ROW>
__global__ void __launch_bounds__(256) k_adj_update(const T* __restrict__ in, T* __restrict__ out,
                                                    const T* __restrict__ K, const T* __restrict__ P,
                                                    const unsigned char* __restrict__ mask, Geo g, double half_dv,
                                                    double dt, int planes) {
  constexpr int W = Vec<T>::W;
  const int i0 = 1 + (int)blockIdx.y * planes, iend = min(i0 + planes, g.NN);
  for (int i = i0; i < iend; ++i) {
    const VGroup r = vgroup<T>(g, i, blockIdx.x);
    const VLoad<T, ROW> l(in, r, g);
    const Quad<T> kq = ldq<T>(K + r.a), pq = ldq<T>(P + r.a);
    const unsigned mw = vbytes<T>(mask, r);
    const Star<T> u = vstar(l);
    Quad<T> o;
#pragma unroll
    for (int e = 0; e < W; ++e) {
      const unsigned m = mw >> (8 * e);
      const double lc = (double)u.c.v[e];
      double lap = 0.0;
      if (m & kNmIp) lap += (double)u.ip.v[e] - lc;
      if (m & kNmIm) lap += (double)u.im.v[e] - lc;
      if (m & kNmJp) lap += (double)u.jp.v[e] - lc;
      if (m & kNmJm) lap += (double)u.jm.v[e] - lc;
      if (m & kNmKp) lap += (double)u.kp.v[e] - lc;
      if (m & kNmKm) lap += (double)u.km.v[e] - lc;
      o.v[e] = (m & kNmIn) ? (T)(lc + half_dv * lap + dt * ((double)kq.v[e] - 2.0 * (double)pq.v[e]) * lc) : T(0);
    }
    if (r.own) stq(out + r.a, o);
  }
}

// dE/dK += dt psi lam and dE/dP += -2 dt psi lam of up to kAdjPend reverse steps in one pass, in the order of
// the steps (newest first), each muP step rounded to T: lam is the input of the step's transposed update, psi
// the state the forward update started from.  Once per step these sums were 24 of its 45 B per point (and
// in the kernel above a third of its loads); per group of steps dE/dK and dE/dP move once.
constexpr int kAdjPend = 4;
struct AdjPend {
  const void *lam[kAdjPend], *psi[kAdjPend];
  int n;
};
template <typename T>
__global__ void __launch_bounds__(256) k_adj_accum(const AdjPend p, double* __restrict__ gK, T* __restrict__ muP, double dt,
                                                   long long S3) {
  constexpr int W = Vec<T>::W;
  const long long a = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * W;
  auto sums = [&](int n, double* k, T* m, const T (*l)[W], const T (*s)[W], int w) {
    for (int e = 0; e < w; ++e)
#pragma unroll
      for (int q = 0; q < kAdjPend; ++q)
        if (q < n) {
          const double pv = (double)s[q][e], lc = (double)l[q][e];
          k[e] += dt * pv * lc;
          m[e] = (T)((double)m[e] - 2.0 * dt * pv * lc);
        }
  };
  T l[kAdjPend][W], s[kAdjPend][W], m[W];
  double k[W];
  if (a + W <= S3) {
#pragma unroll
    for (int q = 0; q < kAdjPend; ++q)
      if (q < p.n) {
        const Quad<T> x = ldq<T>((const T*)p.lam[q] + a), y = ldq<T>((const T*)p.psi[q] + a);
#pragma unroll
        for (int e = 0; e < W; ++e) { l[q][e] = x.v[e]; s[q][e] = y.v[e]; }
      }
    Quad<T> mq = *reinterpret_cast<const Quad<T>*>(muP + a);
    Quad<double> kq[W / 2];
#pragma unroll
    for (int h = 0; h < W / 2; ++h) kq[h] = *reinterpret_cast<const Quad<double>*>(gK + a + 2 * h);
#pragma unroll
    for (int e = 0; e < W; ++e) { m[e] = mq.v[e]; k[e] = kq[e / 2].v[e % 2]; }
    sums(p.n, k, m, l, s, W);
#pragma unroll
    for (int e = 0; e < W; ++e) { mq.v[e] = m[e]; kq[e / 2].v[e % 2] = k[e]; }
    stq(muP + a, mq);
#pragma unroll
    for (int h = 0; h < W / 2; ++h) stq(gK + a + 2 * h, kq[h]);
  } else if (a < S3) {
    const int w = (int)(S3 - a);
    for (int e = 0; e < w; ++e) {
      for (int q = 0; q < p.n; ++q) { l[q][e] = ((const T*)p.lam[q])[a + e]; s[q][e] = ((const T*)p.psi[q])[a + e]; }
      m[e] = muP[a + e];
      k[e] = gK[a + e];
    }
    sums(p.n, k, m, l, s, w);
    for (int e = 0; e < w; ++e) { muP[a + e] = m[e]; gK[a + e] = k[e]; }
  }
}

// A red-black sweep (colour 0, then 1) transposed is two half passes, colour 1 first.  With m the adjoint
// of P after the sweep:
//   k_adj_half   (colour 1 transposed)  m0 += (1/6) sum_6 m1, in place: the points of colour 1 are kept
//   k_adj_other  (colour 0 transposed)  m1' = (1/6) sum_6 m0, m0' = 0, into another buffer
// and the sweep's share of dE/df is (h^2 / 6) m between the two passes, at every point: the buffer of the
// half pass holds it, so nothing is accumulated on the way.  The kernels before (out of place, a running
// dE/df per colour) moved 3.5 fields per colour; values and roundings are the same.
template <typename T, int ROW>
__global__ void __launch_bounds__(256) k_adj_half(T* __restrict__ m, Geo g, int planes) {
  constexpr int W = Vec<T>::W;
  const int i0 = 1 + (int)blockIdx.y * planes, iend = min(i0 + planes, g.NN);
  for (int i = i0; i < iend; ++i) {
    const VGroup r = vgroup<T>(g, i, blockIdx.x);
    const VLoad<T, ROW, false> l(m, r, g);
    const VRow row = vrow(g, r, i);
    const Star<T> u = vstar(l);
#pragma unroll
    for (int e = 0; e < W; e += 2) {  // colour 0: even ids (S is odd)
      const double s = (double)u.ip.v[e] + (double)u.im.v[e] + (double)u.jp.v[e] + (double)u.jm.v[e] +
                       (double)u.kp.v[e] + (double)u.km.v[e];
      if (r.own && vinterior(g, row, e)) m[r.a + e] = (T)((double)u.c.v[e] + sixth(s));
    }
  }
}

// the second half pass; PRE on the finest level also takes the whole dE/df of the V-cycle -- the two
// sweeps' shares and the residual's, muf = (h^2/6) mA + mur + (h^2/6) m, each sum rounded to T as it forms --
// into lam += 4 pi psi muf (the right-hand side is f = 2 pi psi^2).  out may be mA's buffer.
template <typename T, bool PRE, int ROW>
__global__ void __launch_bounds__(256) k_adj_other(const T* __restrict__ m, T* out, const T* mA, const T* __restrict__ mur,
                                                   const T* __restrict__ psi, T* __restrict__ lam, Geo g, double c6,
                                                   int planes) {
  constexpr int W = Vec<T>::W;
  const int i0 = 1 + (int)blockIdx.y * planes, iend = min(i0 + planes, g.NN);
  for (int i = i0; i < iend; ++i) {
    const VGroup r = vgroup<T>(g, i, blockIdx.x);
    const VLoad<T, ROW> l(m, r, g);
    Quad<T> qa, qr, qs, ql;
    if (PRE) {
      qa = *reinterpret_cast<const Quad<T>*>(mA + r.a);
      qr = ldq<T>(mur + r.a);
      qs = ldq<T>(psi + r.a);
      ql = *reinterpret_cast<const Quad<T>*>(lam + r.a);
    }
    const VRow row = vrow(g, r, i);
    const Star<T> u = vstar(l);
    Quad<T> o;
#pragma unroll
    for (int e = 0; e < W; ++e) {
      const bool in = vinterior(g, row, e);
      o.v[e] = T(0);
      if (e & 1) {
        const double s = (double)u.ip.v[e] + (double)u.im.v[e] + (double)u.jp.v[e] + (double)u.jm.v[e] +
                         (double)u.kp.v[e] + (double)u.km.v[e];
        if (in) o.v[e] = (T)(0.0 + sixth(s));
      }
      if (PRE && in) {
        T f = (T)(c6 * (double)qa.v[e]);
        f = (T)((double)f + (double)qr.v[e]);
        f = (T)fma(c6, (double)u.c.v[e], (double)f);
        ql.v[e] = (T)((double)ql.v[e] + 12.566370614359172 * (double)qs.v[e] * (double)f);
      }
    }
    if (r.own) {
      stq(out + r.a, o);
      if (PRE) stq(lam + r.a, ql);
    }
  }
}

// the same dE/df on a coarser level (whose cycle starts from P = 0, so nothing else is needed there)
template <typename T>
__global__ void __launch_bounds__(256) k_adj_muf(const T* __restrict__ mA, const T* __restrict__ mur, const T* __restrict__ mB,
                                                 T* __restrict__ muf, long long S3, double c6) {
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= S3) return;
  T f = (T)(c6 * (double)mA[q]);
  f = (T)((double)f + (double)mur[q]);
  muf[q] = (T)fma(c6, (double)mB[q], (double)f);
}

// residual transposed (forward r = f + (sum_6 P - 6 P) / h^2) on the adjoint of P: m += (sum_6 mur - 6 mur) / h^2
// (its share of dE/df, mur itself, is added where dE/df is used)
template <typename T, int ROW>
__global__ void __launch_bounds__(256) k_adj_res(const T* __restrict__ mur, T* __restrict__ m, Geo g, double inv_h2,
                                                 int planes) {
  constexpr int W = Vec<T>::W;
  const int i0 = 1 + (int)blockIdx.y * planes, iend = min(i0 + planes, g.NN);
  for (int i = i0; i < iend; ++i) {
    const VGroup r = vgroup<T>(g, i, blockIdx.x);
    const VLoad<T, ROW> l(mur, r, g);
    Quad<T> q = *reinterpret_cast<const Quad<T>*>(m + r.a);
    const VRow row = vrow(g, r, i);
    const Star<T> u = vstar(l);
#pragma unroll
    for (int e = 0; e < W; ++e) {
      const double c = (double)u.c.v[e];
      const double s = (double)u.ip.v[e] + (double)u.im.v[e] + (double)u.jp.v[e] + (double)u.jm.v[e] +
                       (double)u.kp.v[e] + (double)u.km.v[e];
      if (vinterior(g, row, e)) q.v[e] = (T)((double)q.v[e] + (s - 6.0 * c) * inv_h2);
    }
    if (r.own) stq(m + r.a, q);
  }
}

// one colour of a red-black sweep, transposed.  Forward: P <- (sum_6 P + h^2 f) / 6 at the points
// of colour `color` ((i+j+k) % 2 == color).  Transposed: at those points out = 0 and
// muf += h^2/6 in; at the others out = in + (1/6) sum_6 in (every neighbour has colour `color`).
// Boundary entries of the adjoint arrays hold 0 and are never written.
template <typename T>
__global__ void __launch_bounds__(256) k_adj_rbgs(const T* __restrict__ in, T* __restrict__ out, T* __restrict__ muf,
                                                  Geo g, double h2, int color) {
  Pt p;
  if (!interior_pt3(g, p)) return;
  const long long id = p.id, S = g.S, S2 = g.S2;
  const double v = (double)in[id];
  if (((p.i + p.j + p.k) & 1) == color) {
    out[id] = T(0);
    muf[id] = (T)((double)muf[id] + h2 / 6.0 * v);
  } else {
    const double s = (double)in[id + S2] + (double)in[id - S2] + (double)in[id + S] + (double)in[id - S] +
                     (double)in[id + 1] + (double)in[id - 1];
    out[id] = (T)(v + s / 6.0);
  }
}

// residual transposed (forward r = f + (sum_6 P - 6 P) / h^2): muf += mur, muP += (sum_6 mur - 6 mur) / h^2
template <typename T>
__global__ void __launch_bounds__(256) k_adj_residual(const T* __restrict__ mur, T* __restrict__ muP,
                                                      T* __restrict__ muf, Geo g, double inv_h2) {
  Pt p;
  if (!interior_pt3(g, p)) return;
  const long long id = p.id, S = g.S, S2 = g.S2;
  const double r = (double)mur[id];
  const double s = (double)mur[id + S2] + (double)mur[id - S2] + (double)mur[id + S] + (double)mur[id - S] +
                   (double)mur[id + 1] + (double)mur[id - 1];
  muf[id] = (T)((double)muf[id] + r);
  muP[id] = (T)((double)muP[id] + (s - 6.0 * r) * inv_h2);
}

// full weighting transposed: mur = (1/8) trilinear(mufc) at the fine interior points, by coarse cells (the
// walk of nm_prolong_cells_body: every load unconditional, a coarse plane loaded once)
template <typename T>
__global__ void __launch_bounds__(256) k_adj_restrict(const T* __restrict__ mufc, T* __restrict__ mur, Geo g, Geo gc,
                                                      int planes) {
  const int nc = gc.NN;
  const int K = blockIdx.x * kNmPrTK + tile_x<32>(), J = blockIdx.y * kNmPrTJ + tile_y<32>();
  if (K >= nc || J >= nc) return;
  const int I0 = blockIdx.z * planes, Iend = min(I0 + planes, nc);
  const long long S = g.S, S2 = g.S2, Sc = gc.S, Sc2 = gc.S2;
  double c0[2][2], c1[2][2];
#pragma unroll
  for (int b = 0; b < 2; ++b)
#pragma unroll
    for (int c = 0; c < 2; ++c) c0[b][c] = (double)mufc[(long long)I0 * Sc2 + (long long)(J + b) * Sc + K + c];
  for (int I = I0; I < Iend; ++I) {
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int c = 0; c < 2; ++c) c1[b][c] = (double)mufc[(long long)(I + 1) * Sc2 + (long long)(J + b) * Sc + K + c];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int i = 2 * I + a, j = 2 * J + b, k = 2 * K + c;
          if (i < 1 || j < 1 || k < 1) continue;
          double v = 0.0;
          v += c0[0][0];
          if (c) v += c0[0][1];
          if (b) {
            v += c0[1][0];
            if (c) v += c0[1][1];
          }
          if (a) {
            v += c1[0][0];
            if (c) v += c1[0][1];
            if (b) {
              v += c1[1][0];
              if (c) v += c1[1][1];
            }
          }
          mur[(long long)i * S2 + (long long)j * S + k] = (T)(v * (1.0 / (8.0 * (1 + a) * (1 + b) * (1 + c))));
        }
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int c = 0; c < 2; ++c) c0[b][c] = c1[b][c];
  }
}

// trilinear prolongation transposed: muPc = (1/8) sum (8,4,2,1 weights) muP at the coarse interior points
template <typename T>
__global__ void __launch_bounds__(256) k_adj_prolong(const T* __restrict__ muP, T* __restrict__ muPc, Geo g, Geo gc) {
  Pt p;
  if (!interior_pt3(gc, p)) return;
  double v = 0.0;
  for (int a = -1; a <= 1; ++a)
    for (int b = -1; b <= 1; ++b)
      for (int cc = -1; cc <= 1; ++cc) {
        const double w = (a == 0 ? 2 : 1) * (b == 0 ? 2 : 1) * (cc == 0 ? 2 : 1);
        v += w * (double)muP[(long long)(2 * p.i + a) * g.S2 + (long long)(2 * p.j + b) * g.S + (2 * p.k + cc)];
      }
  muPc[p.id] = (T)(v / 8.0);
}

// the coarsest level's red-black sweeps transposed, in reverse order, by one block in FP64 shared
// memory: given dE/dP after the solve (which started from P = 0), writes dE/df
template <typename T>
__global__ void __launch_bounds__(1024) k_adj_coarsest(const T* __restrict__ muP, T* __restrict__ muf, Geo g, double h2,
                                                       int sweeps) {
  extern __shared__ double sm[];
  double* sP = sm;
  double* sf = sm + g.S3;
  for (long long q = threadIdx.x; q < g.S3; q += blockDim.x) {
    sP[q] = (double)muP[q];
    sf[q] = 0.0;
  }
  __syncthreads();
  const int n = g.NN - 1, S = g.S, S2 = (int)g.S2;
  const int nint = n * n * n;
  for (int s = sweeps - 1; s >= 0; --s)
    for (int color = 1; color >= 0; --color) {
      for (int q = threadIdx.x; q < nint; q += blockDim.x) {  // the other colour gathers
        const int k = 1 + q % n, j = 1 + (q / n) % n, i = 1 + q / (n * n);
        if (((i + j + k) & 1) == color) continue;
        const int id = i * S2 + j * S + k;
        sP[id] += (sP[id + S2] + sP[id - S2] + sP[id + S] + sP[id - S] + sP[id + 1] + sP[id - 1]) / 6.0;
      }
      __syncthreads();
      for (int q = threadIdx.x; q < nint; q += blockDim.x) {  // this colour: into f, then 0
        const int k = 1 + q % n, j = 1 + (q / n) % n, i = 1 + q / (n * n);
        if (((i + j + k) & 1) != color) continue;
        const int id = i * S2 + j * S + k;
        sf[id] += h2 / 6.0 * sP[id];
        sP[id] = 0.0;
      }
      __syncthreads();
    }
  for (long long q = threadIdx.x; q < g.S3; q += blockDim.x) muf[q] = (T)sf[q];
}

// lam += 4 pi psi muf (the fine right-hand side f = 2 pi psi^2)
template <typename T>
__global__ void __launch_bounds__(256) k_adj_rhs(T* __restrict__ lam, const T* __restrict__ psi, const T* __restrict__ muf,
                                                 Geo g) {
  Pt p;
  if (!interior_pt3(g, p)) return;
  const long long id = p.id;
  lam[id] = (T)((double)lam[id] + 12.566370614359172 * (double)psi[id] * (double)muf[id]);
}

// checkpoint of the state a step starts from: psi with a pending per-domain scale applied
// (FP64 product rounded once, as the update applies it) or a plain copy
template <typename T>
__global__ void __launch_bounds__(256) k_adj_ckpt(const T* __restrict__ U, const int* __restrict__ label,
                                                  const double* __restrict__ scale, T* __restrict__ out, long long S3,
                                                  int nDom) {
  for (long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x; id < S3;
       id += (long long)gridDim.x * blockDim.x) {
    const T u = U[id];
    if (!scale) {
      out[id] = u;
      continue;
    }
    const int l = label[id];
    out[id] = (l < 0 || l >= nDom) ? u : (T)((double)u * scale[l]);
  }
}

size_t esize(const rq_ctx* c) { return c->fp64 ? sizeof(double) : sizeof(float); }

// a recorded field: the slots are padded to 16 bytes, as the vector kernels read them
long long slot_stride(long long S3) { return (S3 + 3) & ~3LL; }
template <typename T>
T* slot(void* base, long long k, long long S3) {
  return (T*)base + k * slot_stride(S3);
}

// a new P snapshot slot holding the P in effect now.  A window reaches back at most cap steps,
// i.e. over fewer than np - 1 V-cycles, so no step still in the window refers to the slot that
// is overwritten.
int snapshot_p(rq_ctx* c) {
  rq_adj& A = c->adj;
  const size_t bytes = (size_t)c->g.S3 * esize(c);
  const int s = A.next_p % A.np;
  A.next_p++;
  CK(cudaMemcpyAsync((char*)A.psum + (size_t)s * slot_stride(c->g.S3) * esize(c), c->P[c->cp], bytes,
                     cudaMemcpyDeviceToDevice, c->st));
  A.cur_p = s;
  return RQ_OK;
}

}  // namespace

// ----------------------------------------------------------------------------------------
// window management
// ----------------------------------------------------------------------------------------
void nm_adj_free(rq_ctx* c) {
  rq_adj& A = c->adj;
  void* p[] = {A.psi, A.psum, A.scales, A.lam[0], A.lam[1], A.muP[0], A.muP[1], A.muf, A.gK, A.coef, A.wq};
  for (void* q : p)
    if (q) cudaFree(q);
  for (auto& L : A.lv)
    for (void* q : {L.mu[0], L.mu[1], L.muf, L.mur})
      if (q) cudaFree(q);
  A = rq_adj();
}

void nm_adj_reset(rq_ctx* c) {
  c->adj.rec.clear();
  c->adj.cur_p = -1;
}

int nm_adj_set_window(rq_ctx* c, int steps) {
  if (steps < 0) return rq_fail(c, RQ_EINVAL, "negative adjoint window");
  nm_adj_free(c);
  if (steps == 0) return RQ_OK;
  rq_adj& A = c->adj;
  const size_t S3 = (size_t)c->g.S3, es = esize(c);
  const int n = c->n_atoms;
  const int pi = std::max(1, c->cfg.poisson_interval);
  const int np = (steps + pi - 1) / pi + 2;
  auto alloc = [&](void** p, size_t bytes) -> bool {
    if (cudaMalloc(p, bytes) != cudaSuccess) return false;
    return cudaMemsetAsync(*p, 0, bytes, c->st) == cudaSuccess;
  };
  const size_t slot_bytes = (size_t)slot_stride((long long)S3) * es;
  bool ok = alloc(&A.psi, steps * slot_bytes) && alloc(&A.psum, np * slot_bytes) &&
            alloc((void**)&A.scales, sizeof(double) * (size_t)steps * n) && alloc(&A.lam[0], S3 * es) &&
            alloc(&A.lam[1], S3 * es) && alloc(&A.muP[0], S3 * es) && alloc(&A.muP[1], S3 * es) &&
            alloc(&A.muf, S3 * es) && alloc((void**)&A.gK, S3 * sizeof(double)) &&
            alloc((void**)&A.coef, sizeof(double) * 2 * n) &&
            alloc((void**)&A.wq, sizeof(double) * 2 * n);
  const int levels = (int)c->mg.size();
  A.lv.assign(levels, rq_adj::Level());
  for (int l = 0; ok && l < levels; ++l) {
    const size_t s3 = (size_t)c->mg[l].g.S3;
    if (l > 0) ok = alloc(&A.lv[l].mu[0], s3 * es) && alloc(&A.lv[l].mu[1], s3 * es) && alloc(&A.lv[l].muf, s3 * es);
    if (ok && l < levels - 1) ok = alloc(&A.lv[l].mur, s3 * es);
  }
  if (!ok) {
    nm_adj_free(c);
    return rq_cuda(c, cudaErrorMemoryAllocation, "adjoint window");
  }
  A.cap = steps;
  A.np = np;
  nm_adj_reset(c);
  return cudaStreamSynchronize(c->st) == cudaSuccess ? RQ_OK : rq_cuda(c, cudaGetLastError(), "adjoint window");
}

int nm_adj_record_step(rq_ctx* c, bool vcycle, bool norm) {
  rq_adj& A = c->adj;
  if (vcycle || A.cur_p < 0) {
    int rc = snapshot_p(c);
    if (rc != RQ_OK) return rc;
  }
  if ((int)A.rec.size() == A.cap) A.rec.erase(A.rec.begin());
  rq_adj::Rec r;
  r.psi_slot = (int)(A.next_psi % A.cap);
  A.next_psi++;
  r.p_slot = A.cur_p;
  r.vcycle = vcycle;
  r.norm = norm;
  r.label = false;
  const long long S3 = c->g.S3;
  const double* sc = c->nm_pending ? (const double*)c->scale64 : nullptr;
  if (c->fp64)
    LAUNCH(RQ_KC_OTHER, 20.0 * S3,
           (k_adj_ckpt<double><<<148 * 8, 256, 0, c->st>>>((const double*)c->U[c->cu], c->lab[c->cl], sc,
                                                           slot<double>(A.psi, r.psi_slot, S3), S3, c->n_atoms),
            cudaGetLastError()));
  else
    LAUNCH(RQ_KC_OTHER, 12.0 * S3,
           (k_adj_ckpt<float><<<148 * 8, 256, 0, c->st>>>((const float*)c->U[c->cu], c->lab[c->cl], sc,
                                                          slot<float>(A.psi, r.psi_slot, S3), S3, c->n_atoms),
            cudaGetLastError()));
  A.rec.push_back(r);
  return RQ_OK;
}

int nm_adj_record_scale(rq_ctx* c) {
  rq_adj& A = c->adj;
  if (A.rec.empty()) return RQ_OK;
  const int n = c->n_atoms;
  CK(cudaMemcpyAsync(A.scales + (size_t)A.rec.back().psi_slot * n, c->scale64, sizeof(double) * n,
                     cudaMemcpyDeviceToDevice, c->st));
  return RQ_OK;
}

void nm_adj_record_label(rq_ctx* c) {
  if (!c->adj.rec.empty()) c->adj.rec.back().label = true;
}

// ----------------------------------------------------------------------------------------
// the reverse sweep
// ----------------------------------------------------------------------------------------
namespace {

// the per-domain coefficients of a transposed normalisation of lam, with the forward scales `scale` at the
// normalised state psi (applied by k_adj_apply)
template <typename T>
int adj_norm(rq_ctx* c, const T* psi, const T* lam, const double* scale) {
  rq_adj& A = c->adj;
  const int n = c->n_atoms;
  CK(cudaMemsetAsync(c->acc, 0, sizeof(long long) * kExWords * n, c->st));
  LAUNCH(RQ_KC_FORCES, (2.0 * sizeof(T) + 4.0) * c->g.S3,
         (k_adj_dot<T><<<nm_norms_grid(c->g), 256, 0, c->st>>>(psi, lam, c->lab[c->cl], c->g, n, c->acc), cudaGetLastError()));
  LAUNCH(RQ_KC_FORCES, (8.0 * kExWords + 32.0) * n,
         (k_adj_norm_coef<<<nblk(n, 4), 128, 0, c->st>>>(scale, c->Zdom64, c->acc, n, c->h3, A.coef),
          cudaGetLastError()));
  return RQ_OK;
}

// f(row form of the grid) for the vector kernels
template <class F>
void with_row(const Geo& g, F&& f) {
  if (g.S % 4 == 1) f(std::integral_constant<int, kRowP>{});
  else f(std::integral_constant<int, kRowM>{});
}

template <typename T>
cudaError_t adj_half(const Geo& g, T* m, cudaStream_t st) {
  const int planes = vplanes<T>(g, false);
  with_row(g, [&](auto row) { k_adj_half<T, decltype(row)::value><<<vgrid<T>(g, planes), 256, 0, st>>>(m, g, planes); });
  return cudaGetLastError();
}

// restriction^T of the coarse dE/df onto level l's mur
template <typename T>
int adj_restrict(rq_ctx* c, int l) {
  rq_adj& A = c->adj;
  const Geo &g = c->mg[l].g, &gc = c->mg[l + 1].g;
  const int nc = gc.NN;
  const dim3 t((nc + kNmPrTK - 1) / kNmPrTK, (nc + kNmPrTJ - 1) / kNmPrTJ);
  const int planes = nm_mg_planes((long long)t.x * t.y, nc);
  LAUNCH(RQ_KC_MG, sizeof(T) * 1.125 * g.S3,
         (k_adj_restrict<T><<<dim3(t.x, t.y, (nc + planes - 1) / planes), 256, 0, c->st>>>(
              (const T*)A.lv[l + 1].muf, (T*)A.lv[l].mur, g, gc, planes),
          cudaGetLastError()));
  return RQ_OK;
}

template <typename T>
int adj_coarsest(rq_ctx* c, int l) {
  rq_adj& A = c->adj;
  const rq_mg_level& L = c->mg[l];
  const size_t smem = sizeof(double) * 2 * (size_t)L.g.S3;
  CK(cudaFuncSetAttribute(k_adj_coarsest<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  LAUNCH(RQ_KC_MG, 2.0 * sizeof(T) * L.g.S3,
         (k_adj_coarsest<T><<<1, kCoarsestThreads, smem, c->st>>>((const T*)A.lv[l].mu[0], (T*)A.lv[l].muf, L.g, L.h * L.h,
                                                                 c->cfg.mg_coarse_sweeps),
          cudaGetLastError()));
  return RQ_OK;
}

// Transposed V(1,1) cycle on level l.  mA holds dE/dP of the level after the cycle.  On level 0 it holds
// dE/dP before it on return, and lam has taken the right-hand side's share; on coarser levels (whose
// cycle starts from P = 0) dE/df of the level is left in its muf.
template <typename T>
int adj_vcycle11(rq_ctx* c, int l, T* mA, T* m2, const T* psi, T* lam) {
  rq_adj& A = c->adj;
  const rq_mg_level &L = c->mg[l], &C = c->mg[l + 1];
  const Geo& g = L.g;
  const double h2 = L.h * L.h, c6 = h2 / 6.0;
  const long long ni = (long long)(g.NN - 1) * (g.NN - 1) * (g.NN - 1);
  const int planes = vplanes<T>(g, false);
  const dim3 grd = vgrid<T>(g, planes);
  T* mur = (T*)A.lv[l].mur;
  LAUNCH(RQ_KC_MG, 1.5 * sizeof(T) * ni, adj_half<T>(g, mA, c->st));
  LAUNCH(RQ_KC_MG, 2.0 * sizeof(T) * ni,
         (with_row(g, [&](auto row) {
    k_adj_other<T, false, decltype(row)::value><<<grd, 256, 0, c->st>>>(mA, m2, nullptr, nullptr, nullptr, nullptr, g, c6,
                                                                      planes);
          }),
          cudaGetLastError()));
  LAUNCH(RQ_KC_MG, sizeof(T) * 1.125 * ni,
         (k_adj_prolong<T><<<grid3(C.g), kBlk3, 0, c->st>>>(m2, (T*)A.lv[l + 1].mu[0], g, C.g), cudaGetLastError()));
  T* mc = (T*)A.lv[l + 1].mu[0];
  NmTail t;
  size_t smem = 0;
  int rc = RQ_OK;
  if (l + 1 == nm_tail_plan<T>((int)c->mg.size(), [&](int q) { return c->mg[q].g; }, [&](int q) { return c->mg[q].h; },
                               c->cfg.mg_coarse_sweeps, t, smem))
    LAUNCH(RQ_KC_MG, 2.0 * sizeof(T) * C.g.S3, nm_adj_tail<T>(t, smem, mc, (T*)A.lv[l + 1].muf, c->st));
  else if (l + 1 == (int)c->mg.size() - 1)
    rc = adj_coarsest<T>(c, l + 1);
  else
    rc = adj_vcycle11<T>(c, l + 1, mc, (T*)A.lv[l + 1].mu[1], nullptr, nullptr);
  if (rc != RQ_OK || (rc = adj_restrict<T>(c, l)) != RQ_OK) return rc;
  LAUNCH(RQ_KC_MG, 3.0 * sizeof(T) * ni,
         (with_row(g, [&](auto row) {
    k_adj_res<T, decltype(row)::value><<<grd, 256, 0, c->st>>>(mur, m2, g, 1.0 / h2, planes);
          }),
          cudaGetLastError()));
  LAUNCH(RQ_KC_MG, 1.5 * sizeof(T) * ni, adj_half<T>(g, m2, c->st));
  if (l > 0) {
    LAUNCH(RQ_KC_MG, 4.0 * sizeof(T) * g.S3,
           (k_adj_muf<T><<<nblk(g.S3), 256, 0, c->st>>>(mA, mur, m2, (T*)A.lv[l].muf, g.S3, c6), cudaGetLastError()));
    return RQ_OK;
  }
  LAUNCH(RQ_KC_MG, 7.0 * sizeof(T) * ni,
         (with_row(g, [&](auto row) {
    k_adj_other<T, true, decltype(row)::value><<<grd, 256, 0, c->st>>>(m2, mA, mA, mur, psi, lam, g, c6, planes);
          }),
          cudaGetLastError()));
  return RQ_OK;
}

// The same for any number of sweeps (mg_pre, mg_post), colour by colour out of place with a running dE/df:
// mu[*cur] holds dE/dP of level l after the cycle and becomes dE/dP before it; dE/df of the level is
// accumulated into its muf
template <typename T>
int adj_vcycle(rq_ctx* c, int l, int* cur) {
  rq_adj& A = c->adj;
  const rq_mg_level& L = c->mg[l];
  T* mu[2] = {l == 0 ? (T*)A.muP[0] : (T*)A.lv[l].mu[0], l == 0 ? (T*)A.muP[1] : (T*)A.lv[l].mu[1]};
  T* muf = l == 0 ? (T*)A.muf : (T*)A.lv[l].muf;
  const double h2 = L.h * L.h;
  const long long ni = (long long)(L.g.NN - 1) * (L.g.NN - 1) * (L.g.NN - 1);
  const int last = (int)c->mg.size() - 1;
  if (l == last) return adj_coarsest<T>(c, l);
  auto smooth = [&](int sweeps) -> int {
    for (int s = 0; s < sweeps; ++s)
      for (int color = 1; color >= 0; --color) {
        LAUNCH(RQ_KC_MG, 3.5 * sizeof(T) * ni,
               (k_adj_rbgs<T><<<grid3(L.g), kBlk3, 0, c->st>>>(mu[*cur], mu[1 - *cur], muf, L.g, h2, color),
                cudaGetLastError()));
        *cur ^= 1;
      }
    return RQ_OK;
  };
  int rc = smooth(c->cfg.mg_post);
  if (rc != RQ_OK) return rc;
  const rq_mg_level& C = c->mg[l + 1];
  const long long nc = (long long)(C.g.NN - 1) * (C.g.NN - 1) * (C.g.NN - 1);
  int ccur = 0;
  LAUNCH(RQ_KC_MG, sizeof(T) * (ni + nc),
         (k_adj_prolong<T><<<grid3(C.g), kBlk3, 0, c->st>>>(mu[*cur], (T*)A.lv[l + 1].mu[0], L.g, C.g), cudaGetLastError()));
  CK(cudaMemsetAsync(A.lv[l + 1].muf, 0, sizeof(T) * C.g.S3, c->st));
  if ((rc = adj_vcycle<T>(c, l + 1, &ccur)) != RQ_OK) return rc;
  if ((rc = adj_restrict<T>(c, l)) != RQ_OK) return rc;
  LAUNCH(RQ_KC_MG, 5.0 * sizeof(T) * ni,
         (k_adj_residual<T><<<grid3(L.g), kBlk3, 0, c->st>>>((const T*)A.lv[l].mur, mu[*cur], muf, L.g, 1.0 / h2),
          cudaGetLastError()));
  return smooth(c->cfg.mg_pre);
}

template <typename T>
int adjoint_t(rq_ctx* c, double* F, double* dEdv) {
  rq_adj& A = c->adj;
  const int n = c->n_atoms;
  const Geo& g = c->g;
  const long long S3 = g.S3, ni = (long long)(g.NN - 1) * (g.NN - 1) * (g.NN - 1);
  for (const rq_adj::Rec& r : A.rec)
    if (r.label)
      return rq_fail(c, RQ_ENOTSUP,
                     "a label pass ran inside the recorded window: the adjoint holds the labels fixed (set label_until)");
  int rc = nm_ready(c);  // a normalisation it performs is recorded as the last step's
  if (rc != RQ_OK) return rc;
  const T* psi = (const T*)c->U[c->cu];
  const T* K = (const T*)c->K;
  const int* lab = c->lab[c->cl];
  // the readout's per-domain partials -> (Z/N, Q/N)
  LAUNCH(RQ_KC_ENERGY, (4.0 * sizeof(T) + 4.0) * ni,
         nm_energy<T>(psi, K, (const T*)c->P[c->cp], lab, g, c->h, n, c->acc, c->dpd, c->st, c->K64));
  std::vector<double> pd((size_t)kNmPD * n), wq((size_t)2 * n);
  CK(cudaMemcpyAsync(pd.data(), c->dpd, sizeof(double) * pd.size(), cudaMemcpyDeviceToHost, c->st));
  CK(cudaStreamSynchronize(c->st));
  for (int d = 0; d < n; ++d) {
    const double* x = &pd[(size_t)kNmPD * d];
    wq[2 * d] = domain_norm_weight(c->atoms[d].Z, x[0]);
    wq[2 * d + 1] = x[0] > 0.0 ? (x[1] + x[2] + 2.0 * x[3]) / x[0] : 0.0;
  }
  CK(cudaMemcpyAsync(A.wq, wq.data(), sizeof(double) * wq.size(), cudaMemcpyHostToDevice, c->st));
  int mi = 0;
  T* muP[2] = {(T*)A.muP[0], (T*)A.muP[1]};
  T* lam = (T*)A.lam[0];
  AdjPend pend{};
  // Buffers for lambda: the sweep's and those of the steps whose sums are pending.  Besides the window's two, the
  // state's idle buffers (the other psi, whose faces are 0 and whose interior the next update writes; the other
  // P, which holds nothing between V-cycles) and, where dE/df is not kept on the finest level, its buffer.
  const bool v11 = c->cfg.mg_pre == 1 && c->cfg.mg_post == 1;
  T* const bufs[kAdjPend + 1] = {(T*)A.lam[0], (T*)A.lam[1], (T*)c->U[1 - c->cu], (T*)c->P[1 - c->cp], (T*)A.muf};
  const int nbufs = v11 ? kAdjPend + 1 : kAdjPend;
  CK(launch_zero_faces(bufs[3], g, c->st));
  auto spare = [&]() -> T* {
    for (int b = 0; b < nbufs; ++b) {
      bool held = bufs[b] == lam;
      for (int q = 0; q < pend.n; ++q) held = held || bufs[b] == pend.lam[q];
      if (!held) return bufs[b];
    }
    return nullptr;  // not reached: at most nbufs - 2 are pending here
  };
  auto accumulate = [&]() -> int {
    if (!pend.n) return RQ_OK;
    LAUNCH(RQ_KC_FORCES, (2.0 * sizeof(T) * pend.n + 16.0 + 2.0 * sizeof(T)) * S3,
           (k_adj_accum<T><<<nblk(S3, 256 * Vec<T>::W), 256, 0, c->st>>>(pend, A.gK, muP[mi], c->dt, S3), cudaGetLastError()));
    pend.n = 0;
    return RQ_OK;
  };
  LAUNCH(RQ_KC_FORCES, (4.0 * sizeof(T) + 4.0 + 2.0 * sizeof(T) + 8.0) * ni,
         (k_adj_seed<T><<<grid3(g), kBlk3, 0, c->st>>>(psi, K, (const T*)c->P[c->cp], lab, g, c->h, n, A.wq, lam, muP[mi],
                                                     A.gK, c->K64),
          cudaGetLastError()));
  const int planes = vplanes<T>(g, false);
  for (int r = (int)A.rec.size() - 1; r >= 0; --r) {
    const rq_adj::Rec& R = A.rec[r];
    const T* psi_prev = slot<T>(A.psi, R.psi_slot, S3);
    const T* P_s = slot<T>(A.psum, R.p_slot, S3);
    T* out = spare();
    if (R.norm) {
      const T* psi_s = r + 1 < (int)A.rec.size() ? slot<T>(A.psi, A.rec[r + 1].psi_slot, S3) : psi;
      if ((rc = adj_norm<T>(c, psi_s, lam, A.scales + (size_t)R.psi_slot * n)) != RQ_OK) return rc;
      LAUNCH(RQ_KC_FORCES, (3.0 * sizeof(T) + 4.0) * S3,
             (k_adj_apply<T><<<nblk(S3, 256 * Vec<T>::W), 256, 0, c->st>>>(lam, psi_s, lab, A.coef, S3, n),
              cudaGetLastError()));
    }
    LAUNCH(RQ_KC_FORCES, (4.0 * sizeof(T) + 1.0) * ni,
           (with_row(g, [&](auto row) {
      k_adj_update<T, decltype(row)::value><<<vgrid<T>(g, planes), 256, 0, c->st>>>(lam, out, K, P_s, c->nbm, g, c->half_dv,
                                                                                    c->dt, planes);
            }),
            cudaGetLastError()));
    pend.lam[pend.n] = lam;
    pend.psi[pend.n++] = psi_prev;
    lam = out;
    if ((R.vcycle || pend.n == nbufs - 1) && (rc = accumulate()) != RQ_OK) return rc;
    if (R.vcycle && v11) {
      if ((rc = adj_vcycle11<T>(c, 0, muP[mi], muP[1 - mi], psi_prev, lam)) != RQ_OK) return rc;
    } else if (R.vcycle) {
      CK(cudaMemsetAsync(A.muf, 0, sizeof(T) * S3, c->st));
      if ((rc = adj_vcycle<T>(c, 0, &mi)) != RQ_OK) return rc;
      LAUNCH(RQ_KC_FORCES, 4.0 * sizeof(T) * ni,
             (k_adj_rhs<T><<<grid3(g), kBlk3, 0, c->st>>>(lam, psi_prev, (const T*)A.muf, g), cudaGetLastError()));
    }
  }
  if ((rc = accumulate()) != RQ_OK) return rc;
  if (F) {
    CK(cudaMemsetAsync(c->dF, 0, sizeof(double) * 3 * n, c->st));
    if ((rc = nm_gather(c, psi, A.gK)) != RQ_OK) return rc;
    CK(cudaMemcpyAsync(F, c->dF, sizeof(double) * 3 * n, cudaMemcpyDeviceToHost, c->st));
  }
  if (dEdv) CK(cudaMemcpyAsync(dEdv, A.gK, sizeof(double) * S3, cudaMemcpyDefault, c->st));  // host or device
  CK(cudaStreamSynchronize(c->st));
  return RQ_OK;
}

}  // namespace

int nm_adjoint(rq_ctx* c, double* F, double* dEdv) {
  if (c->adj.cap > 0) return c->fp64 ? adjoint_t<double>(c, F, dEdv) : adjoint_t<float>(c, F, dEdv);
  // no recording window: the gradient of the readout alone (the Hellmann-Feynman terms); the
  // forces alone are the HF gather, dE/dv needs the reverse-sweep buffers for this call
  if (!dEdv) return F ? nm_forces(c, RQ_FORCE_HF, F) : RQ_OK;
  int rc = nm_adj_set_window(c, 1);
  if (rc == RQ_OK) rc = c->fp64 ? adjoint_t<double>(c, F, dEdv) : adjoint_t<float>(c, F, dEdv);
  nm_adj_free(c);
  return rc;
}
