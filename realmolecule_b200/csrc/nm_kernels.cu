// nm_kernels.cu -- single-grid kernels of the new flavour: Gaussian-smoothed nuclei, red-black
// Gauss-Seidel multigrid for the Hartree half-potential, FP64 per-domain sums, and the
// stationary-point gradient with respect to the nuclear centres.  The point-wise code lives
// in nm_bodies.cuh (shared with the batched kernels); here each body gets its block
// coordinates from blockIdx.  T = float (mixed path) or double (FP64 path).
#include <type_traits>

#include "nm_bodies.cuh"
#include "nm_tail.cuh"
#include "rq_kernels.h"
#include "vec_stencil.cuh"

namespace rq {

template <typename T>
__global__ void __launch_bounds__(256) k_nm_potential(T* K, const double* at, int nAt, Geo g, double h, double sigma,
                                                      double* K64) {
  __shared__ double sa[128 * 4];
  nm_potential_body<T>(K, at, nAt, g, h, sigma, blockIdx.x, sa, K64);
}

template <typename T>
__global__ void __launch_bounds__(256) k_nm_init(T* U, int* label, const float4* seeds, int nSeed, Geo g, float h) {
  __shared__ float4 ss[256];
  nm_init_body<T>(U, label, seeds, nSeed, g, h, blockIdx.x, ss);
}

template <int ROW>
__global__ void __launch_bounds__(256) k_nm_mask(const int* __restrict__ label, unsigned char* __restrict__ mask, Geo g) {
  nm_mask_body<ROW>(label, mask, g, blockIdx.x, 1 + (int)blockIdx.y);
}

// mask: the same-label neighbour mask of `label`.  seed[0]: the step seed of the unbiased fp32 rounding
// (null: round to nearest); the next step's seed, seed[0] + 1, goes to seed_next (read and written in
// different words, so every block reads the same value)
template <typename T, bool SR, int ROW>
__global__ void __launch_bounds__(256) k_nm_update(const T* U, T* Unew, const T* K, const T* P, const int* label, Geo g,
                                                   T half_dv, T dt, int nDom, const double* scale, const unsigned* seed,
                                                   unsigned* seed_next, const unsigned char* __restrict__ mask, int planes) {
  if (SR && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *seed_next = *seed + 1u;
  const int i0 = 1 + (int)blockIdx.y * planes;
  nm_vupdate_body<T, SR, ROW>(U, Unew, K, P, label, mask, g, half_dv, dt, nDom, blockIdx.x, i0, min(i0 + planes, g.NN),
                              scale, seed);
}

// scale[l] = sqrt(Zdom_l / n_l) (FP64) for every domain; a norm that is NaN or Inf sets bit 0 of *err
// and leaves its domain unscaled.  The norms of a batch's concatenated domains are plain sums, those of a single
// grid accumulators (exact_sum.h), a warp each.
__global__ void k_nm_norm_scale(const double* __restrict__ norms, const double* __restrict__ Zdom, int nDom,
                                double* __restrict__ scale, int* __restrict__ err) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l < nDom) scale[l] = nm_domain_scale(norms[l], Zdom[l], err);
}
__global__ void __launch_bounds__(128) k_nm_norm_scale_acc(const long long* __restrict__ acc, const double* __restrict__ Zdom,
                                                           int nDom, double* __restrict__ scale, int* __restrict__ err) {
  const int l = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (l >= nDom) return;
  const double n = exact_value_warp(acc + (long long)l * kExWords);
  if (threadIdx.x % 32 == 0) scale[l] = nm_domain_scale(n, Zdom[l], err);
}

// out[q] = the double next to accumulator q
__global__ void __launch_bounds__(256) k_nm_acc_value(const long long* __restrict__ acc, int n, double* __restrict__ out) {
  const int q = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (q >= n) return;
  const double v = exact_value_warp(acc + (long long)q * kExWords);
  if (threadIdx.x % 32 == 0) out[q] = v;
}

template <typename T>
__global__ void __launch_bounds__(256) k_nm_apply_scale(T* U, const int* label, const double* scale, long long S3, int nDom) {
  nm_apply_scale_body<T>(U, label, scale, S3, nDom, blockIdx.x);
}

template <typename T>
__global__ void __launch_bounds__(256) k_nm_norms(const T* U, const int* label, Geo g, double h3, int nDom, long long* acc) {
  __shared__ NormSmem<BlockSums<1>> sm;
  const int i0 = 1 + (int)blockIdx.z * kNmNormPlanes;
  nm_norms_body<T>(U, label, g, h3, nDom, ExactSums<1>{sm.sums, acc}, sm.list, blockIdx.x, blockIdx.y, i0,
                   min(i0 + kNmNormPlanes, g.NN));
}

template <typename T, bool FINE, int ROW, int COLOR>
__global__ void __launch_bounds__(256) k_nm_rbgs(T* P, const T* f, Geo g, T h2, int planes) {
  const int i0 = 1 + (int)blockIdx.y * planes;
  nm_vrbgs_body<T, FINE, ROW, COLOR>(P, f, g, h2, blockIdx.x, i0, min(i0 + planes, g.NN));
}

template <typename T, bool FINE, int ROW>
__global__ void __launch_bounds__(256) k_nm_residual(const T* P, const T* f, T* r, Geo g, T inv_h2, int planes) {
  const int i0 = 1 + (int)blockIdx.y * planes;
  nm_vresidual_body<T, FINE, ROW>(P, f, r, g, inv_h2, blockIdx.x, i0, min(i0 + planes, g.NN));
}

template <typename T>
__global__ void __launch_bounds__(256) k_nm_restrict(const T* r, T* fc, T* Pc, Geo g, Geo gc) {
  nm_restrict_tile_body<T>(r, fc, Pc, g, gc, blockIdx.x, blockIdx.y, 1 + (int)blockIdx.z, 2 + (int)blockIdx.z);
}

template <typename T>
__global__ void __launch_bounds__(256) k_nm_prolong(const T* Ec, T* P, Geo g, Geo gc, int planes) {
  nm_prolong_cells_body<T>(Ec, P, g, gc, blockIdx.x, blockIdx.y, blockIdx.z, planes);
}

template <typename T>
__global__ void __launch_bounds__(1024) k_nm_coarsest(T* P, const T* f, Geo g, double h2, int sweeps) {
  extern __shared__ double sm[];
  nm_coarsest_body<T>(P, f, g, h2, sweeps, sm);
}

template <typename T>
__global__ void __launch_bounds__(256) k_nm_energy(const T* U, const T* K, const T* P, const int* label, Geo g, double h,
                                                   int nDom, long long* acc, const double* K64) {
  __shared__ EnergySmem<BlockSums<kNmPD>> sm;
  nm_energy_body<T>(U, K, P, label, g, h, nDom, ExactSums<kNmPD>{sm.sums, acc}, sm.list, blockIdx.x, blockIdx.y, blockIdx.z,
                    K64);
}

template <typename T>
__global__ void __launch_bounds__(256) k_nm_evolve(const int* labIn, int* labOut, const T* U, float* W, Geo g, T dt_w,
                                                   T curvReg) {
  nm_evolve_body<T>(labIn, labOut, U, W, g, dt_w, curvReg, blockIdx.x, blockIdx.y, blockIdx.z);
}

template <typename T>
__global__ void __launch_bounds__(256, 3) k_nm_gather(const T* U, const double* at, int nAt, Geo g, double h, double sigma,
                                                   double* F, const double* gw) {
  __shared__ GatherSmem sm;
  nm_gather_all_body<T>(U, gw, at, nAt, g, h, sigma, F, blockIdx.x, blockIdx.y, blockIdx.z, sm);
}

template <typename T>
__global__ void __launch_bounds__(256) k_nm_gather_core(const T* U, const double* at, Geo g, double h, double sigma,
                                                        double* F, const double* gw) {
  nm_gather_core_entry<T>(U, gw, at, blockIdx.x, g, h, sigma, F, blockIdx.y);
}

template <typename T>
__global__ void k_nm_add(T* __restrict__ K, const T* __restrict__ v, long long n) {
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
    K[q] = Ar<T>::add(K[q], v[q]);
}

// ======================================================================================
// host launchers (T = float or double)
// ======================================================================================
using RowP = std::integral_constant<int, kRowP>;
using RowM = std::integral_constant<int, kRowM>;
static unsigned nblk(long long n, long long b = 256) { return (unsigned)((n + b - 1) / b); }

template <typename T>
cudaError_t nm_potential(T* K, const double* at, int nAt, const Geo& g, double h, double sigma, cudaStream_t st,
                         double* K64) {
  k_nm_potential<T><<<nblk(g.S3), 256, 0, st>>>(K, at, nAt, g, h, sigma, K64);
  return cudaGetLastError();
}
template <typename T>
cudaError_t nm_init(T* U, int* label, const float4* seeds, int nSeed, const Geo& g, float h, cudaStream_t st) {
  k_nm_init<T><<<nblk(g.S3), 256, 0, st>>>(U, label, seeds, nSeed, g, h);
  return cudaGetLastError();
}
template <typename T>
cudaError_t nm_update(const T* U, T* Unew, const T* K, const T* P, const int* label, const Geo& g, T half_dv, T dt,
                      double h3, int nDom, long long* norms, cudaStream_t st, const double* scale, const unsigned* seed,
                      unsigned* seed_next, const unsigned char* mask) {
  if (g.NN < 2) return cudaSuccess;
  const int planes = vplanes<T>(g, false);
  auto go = [&](auto sr, auto row) {
    k_nm_update<T, decltype(sr)::value, decltype(row)::value><<<vgrid<T>(g, planes), 256, 0, st>>>(
        U, Unew, K, P, label, g, half_dv, dt, nDom, scale, seed, seed_next, mask, planes);
  };
  using Y = std::true_type;
  using N = std::false_type;
  if (g.S % 4 == 1) { if (seed) go(Y{}, RowP{}); else go(N{}, RowP{}); }
  else              { if (seed) go(Y{}, RowM{}); else go(N{}, RowM{}); }
  if (norms) k_nm_norms<T><<<nm_norms_grid(g), 256, 0, st>>>(Unew, label, g, h3, nDom, norms);
  return cudaGetLastError();
}
cudaError_t nm_mask(const int* label, unsigned char* mask, const Geo& g, cudaStream_t st) {
  if (g.S % 4 == 1)
    k_nm_mask<kRowP><<<vgrid<int>(g, 1), 256, 0, st>>>(label, mask, g);
  else
    k_nm_mask<kRowM><<<vgrid<int>(g, 1), 256, 0, st>>>(label, mask, g);
  return cudaGetLastError();
}
template <typename T>
cudaError_t nm_apply(T* U, const int* label, const double* scale, int nDom, const Geo& g, cudaStream_t st) {
  k_nm_apply_scale<T><<<nblk(g.S3, 256 * kNmFlatChunk), 256, 0, st>>>(U, label, scale, g.S3, nDom);
  return cudaGetLastError();
}
template <typename T>
cudaError_t nm_normalize(T* U, const int* label, const long long* norms, const double* Zdom, int nDom, double* scale,
                         int* err, const Geo& g, cudaStream_t st) {
  k_nm_norm_scale_acc<<<nblk(nDom, 4), 128, 0, st>>>(norms, Zdom, nDom, scale, err);
  k_nm_apply_scale<T><<<nblk(g.S3, 256 * kNmFlatChunk), 256, 0, st>>>(U, label, scale, g.S3, nDom);
  return cudaGetLastError();
}
cudaError_t nm_norm_scale(const double* norms, const double* Zdom, int nDom, double* scale, int* err, cudaStream_t st) {
  k_nm_norm_scale<<<nblk(nDom, 128), 128, 0, st>>>(norms, Zdom, nDom, scale, err);
  return cudaGetLastError();
}
cudaError_t nm_norm_scale(const long long* norms, const double* Zdom, int nDom, double* scale, int* err, cudaStream_t st) {
  k_nm_norm_scale_acc<<<nblk(nDom, 4), 128, 0, st>>>(norms, Zdom, nDom, scale, err);
  return cudaGetLastError();
}
template <typename T>
cudaError_t nm_norms(const T* U, const int* label, const Geo& g, double h3, int nDom, long long* norms, cudaStream_t st) {
  k_nm_norms<T><<<nm_norms_grid(g), 256, 0, st>>>(U, label, g, h3, nDom, norms);
  return cudaGetLastError();
}
template <typename T>
cudaError_t nm_rbgs(T* P, const T* f, bool fine, const Geo& g, double h2, int color, cudaStream_t st) {
  const int planes = vplanes<T>(g, false);
  const dim3 grd = vgrid<T>(g, planes);
  auto go = [&](auto fn, auto row) {
    if (color)
      k_nm_rbgs<T, decltype(fn)::value, decltype(row)::value, 1><<<grd, 256, 0, st>>>(P, f, g, (T)h2, planes);
    else
      k_nm_rbgs<T, decltype(fn)::value, decltype(row)::value, 0><<<grd, 256, 0, st>>>(P, f, g, (T)h2, planes);
  };
  using Y = std::true_type;
  using N = std::false_type;
  if (g.S % 4 == 1) { if (fine) go(Y{}, RowP{}); else go(N{}, RowP{}); }
  else              { if (fine) go(Y{}, RowM{}); else go(N{}, RowM{}); }
  return cudaGetLastError();
}
template <typename T>
cudaError_t nm_residual(const T* P, const T* f, bool fine, T* r, const Geo& g, double inv_h2, cudaStream_t st) {
  const int planes = vplanes<T>(g, false);
  const dim3 grd = vgrid<T>(g, planes);
  auto go = [&](auto fn, auto row) {
    k_nm_residual<T, decltype(fn)::value, decltype(row)::value><<<grd, 256, 0, st>>>(P, f, r, g, (T)inv_h2, planes);
  };
  using Y = std::true_type;
  using N = std::false_type;
  if (g.S % 4 == 1) { if (fine) go(Y{}, RowP{}); else go(N{}, RowP{}); }
  else              { if (fine) go(Y{}, RowM{}); else go(N{}, RowM{}); }
  return cudaGetLastError();
}
template <typename T>
cudaError_t nm_restrict(const T* r, T* fc, T* Pc, const Geo& g, const Geo& gc, cudaStream_t st) {
  const unsigned n = (unsigned)(gc.NN - 1);
  if (n < 1) return cudaSuccess;
  k_nm_restrict<T><<<dim3((n + 31) / 32, (n + 7) / 8, n), 256, 0, st>>>(r, fc, Pc, g, gc);
  return cudaGetLastError();
}
template <typename T>
cudaError_t nm_prolong(const T* Ec, T* P, const Geo& g, const Geo& gc, cudaStream_t st) {
  const int nc = gc.NN;  // coarse cells per axis
  const long long tiles = (long long)((nc + kNmPrTK - 1) / kNmPrTK) * ((nc + kNmPrTJ - 1) / kNmPrTJ);
  const int planes = nm_mg_planes(tiles, nc);
  const dim3 blk(32, 8), grd((nc + kNmPrTK - 1) / kNmPrTK, (nc + kNmPrTJ - 1) / kNmPrTJ, (nc + planes - 1) / planes);
  k_nm_prolong<T><<<grd, blk, 0, st>>>(Ec, P, g, gc, planes);
  return cudaGetLastError();
}
template <typename T>
cudaError_t nm_coarsest(T* P, const T* f, const Geo& g, double h2, int sweeps, cudaStream_t st) {
  const size_t smem = sizeof(double) * 2 * (size_t)g.S3;
  if (smem > 200 * 1024) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(k_nm_coarsest<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_nm_coarsest<T><<<1, kCoarsestThreads, smem, st>>>(P, f, g, h2, sweeps);
  return cudaGetLastError();
}
template <typename T>
cudaError_t nm_tail(const NmTail& t, size_t smem, const T* f, T* P, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(k_nm_tail<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_nm_tail<T><<<1, kTailThreads, smem, st>>>(t, f, P);
  return cudaGetLastError();
}
template <typename T>
cudaError_t nm_adj_tail(const NmTail& t, size_t smem, const T* mA, T* muf, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(k_adj_tail<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_adj_tail<T><<<1, kTailThreads, smem, st>>>(t, mA, muf);
  return cudaGetLastError();
}
template <typename T>
cudaError_t nm_energy(const T* U, const T* K, const T* P, const int* label, const Geo& g, double h, int nDom,
                      long long* acc, double* pd, cudaStream_t st, const double* K64) {
  const cudaError_t e = cudaMemsetAsync(acc, 0, sizeof(long long) * kExWords * kNmPD * (size_t)nDom, st);
  if (e != cudaSuccess) return e;
  k_nm_energy<T><<<nm_march_grid(g), nm_march_block(), 0, st>>>(U, K, P, label, g, h, nDom, acc, K64);
  k_nm_acc_value<<<nblk((long long)nDom * kNmPD, 8), 256, 0, st>>>(acc, nDom * kNmPD, pd);
  return cudaGetLastError();
}
template <typename T>
cudaError_t nm_evolve(const int* labIn, int* labOut, const T* U, float* W, const Geo& g, double dt_w, double curvReg,
                      cudaStream_t st) {
  if (g.NN < 2) return cudaSuccess;
  k_nm_evolve<T><<<nm_march_grid(g), nm_march_block(), 0, st>>>(labIn, labOut, U, W, g, (T)(float)dt_w, (T)(float)curvReg);
  return cudaGetLastError();
}
template <typename T>
cudaError_t nm_force(const T* U, const double* at, int nAt, const Geo& g, double h, double sigma, double* F,
                     cudaStream_t st, const double* gw) {
  if (g.NN < 2 || nAt <= 0) return cudaSuccess;
  k_nm_gather<T><<<nm_gather_grid(g), 256, 0, st>>>(U, at, nAt, g, h, sigma, F, gw);
  k_nm_gather_core<T><<<dim3((unsigned)nAt, kGaCoreParts), 256, 0, st>>>(U, at, g, h, sigma, F, gw);
  return cudaGetLastError();
}
template <typename T>
cudaError_t nm_add(T* K, const T* v, long long n, cudaStream_t st) {
  k_nm_add<T><<<148 * 8, 256, 0, st>>>(K, v, n);
  return cudaGetLastError();
}

#define RQ_NM_INSTANTIATE(T)                                                                                          \
  template cudaError_t nm_add<T>(T*, const T*, long long, cudaStream_t);                                           \
  template cudaError_t nm_potential<T>(T*, const double*, int, const Geo&, double, double, cudaStream_t, double*);  \
  template cudaError_t nm_init<T>(T*, int*, const float4*, int, const Geo&, float, cudaStream_t);                   \
  template cudaError_t nm_update<T>(const T*, T*, const T*, const T*, const int*, const Geo&, T, T, double, int,     \
                                    long long*, cudaStream_t, const double*, const unsigned*, unsigned*,             \
                                    const unsigned char*);                                                           \
  template cudaError_t nm_apply<T>(T*, const int*, const double*, int, const Geo&, cudaStream_t);                   \
  template cudaError_t nm_normalize<T>(T*, const int*, const long long*, const double*, int, double*, int*,          \
                                       const Geo&, cudaStream_t);                                                    \
  template cudaError_t nm_norms<T>(const T*, const int*, const Geo&, double, int, long long*, cudaStream_t);        \
  template cudaError_t nm_rbgs<T>(T*, const T*, bool, const Geo&, double, int, cudaStream_t);                       \
  template cudaError_t nm_residual<T>(const T*, const T*, bool, T*, const Geo&, double, cudaStream_t);               \
  template cudaError_t nm_restrict<T>(const T*, T*, T*, const Geo&, const Geo&, cudaStream_t);                       \
  template cudaError_t nm_prolong<T>(const T*, T*, const Geo&, const Geo&, cudaStream_t);                           \
  template cudaError_t nm_coarsest<T>(T*, const T*, const Geo&, double, int, cudaStream_t);                         \
  template cudaError_t nm_tail<T>(const NmTail&, size_t, const T*, T*, cudaStream_t);                                \
  template cudaError_t nm_adj_tail<T>(const NmTail&, size_t, const T*, T*, cudaStream_t);                            \
  template cudaError_t nm_energy<T>(const T*, const T*, const T*, const int*, const Geo&, double, int, long long*,  \
                                    double*, cudaStream_t, const double*);                                           \
  template cudaError_t nm_evolve<T>(const int*, int*, const T*, float*, const Geo&, double, double, cudaStream_t);  \
  template cudaError_t nm_force<T>(const T*, const double*, int, const Geo&, double, double, double*, cudaStream_t,  \
                                   const double*);
RQ_NM_INSTANTIATE(float)
RQ_NM_INSTANTIATE(double)

}  // namespace rq
