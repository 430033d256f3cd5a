// Weights of the evaluation without design rows.
//
// The quadratic energy of atom a is w0 + w_lin . B_a + B_a^T W B_a with W the K x K block of the
// weights in the reference's full layout (index K*(id1-1)+id2, mld_energy.F90:170-266).  Its
// gradient with respect to B_a is beta_a = w_lin + (W + W^T) B_a, and the quadratic force and
// stress rows dotted with the weights reduce to the linear contraction of dB with beta
// (mld_forces.F90:410-500: the centre's beta; mld_stress.F90:580-603: the neighbour's beta).
// dE/dc is a sum over the distinct Z blocks, with gamma_b = sum of scale * beta_k over the triples k
// that use block b: the evaluation kernel takes gamma instead of beta.
#include <cuda_runtime.h>

#include <type_traits>

#include "ds.cuh"
#include "mld_internal.h"

namespace mld {

namespace {

constexpr int kGammaThreads = 128;
constexpr int kGammaAtoms = 4;  // atoms per CTA: each reads Wsym once for all of them

__global__ void k_split_pairs(const double* __restrict__ in, float2* __restrict__ out, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float h, l;
  ds_split(in[i], h, l);
  out[i] = make_float2(h, l);
}

// beta[k] = w_lin[k] + sum_j Wsym[j][k] B[j] (Wsym symmetric, read by rows j so that consecutive threads
// read consecutive k), the atom's energy w0 + B . (beta + w_lin) / 2 and gamma of every channel and
// block.  The sums over j run in double-FP32 for FP32 descriptors (2^-44 relative; FP64 issues at 1/64
// of the FP32 rate and took 182 us of a 4,001-atom step with K = 110, 2 channels), in FP64 for FP64
// ones.  B null: beta = w_lin, no energy, and G holds every weight in full (a pair for T = float).
__device__ __forceinline__ void put_weight(float* g, double v) { *g = (float)v; }
__device__ __forceinline__ void put_weight(double* g, double v) { *g = v; }
__device__ __forceinline__ void put_weight(float2* g, double v) {
  float h, l;
  ds_split(v, h, l);
  *g = make_float2(h, l);
}

template <typename T, typename G>
__global__ void __launch_bounds__(kGammaThreads) k_eval_gamma(const int* __restrict__ gam_off,
                                                              const GammaItem* __restrict__ gam, int nblk, int nch,
                                                              int K, int A, const T* __restrict__ B,
                                                              const double* __restrict__ wlin,
                                                              const double* __restrict__ wsym,
                                                              const float2* __restrict__ wsym32, double w0,
                                                              G* __restrict__ gamma, double* __restrict__ Eatom) {
  extern __shared__ double beta[];  // [kGammaAtoms][nchK], then B as T
  __shared__ double red[kGammaAtoms][kGammaThreads / 32];
  const int tid = threadIdx.x, nchK = nch * K, a0 = blockIdx.x * kGammaAtoms;
  const int na = B ? min(kGammaAtoms, A - a0) : 1;
  T* bsh = reinterpret_cast<T*>(beta + kGammaAtoms * nchK);
  if (B) {
    for (int j = tid; j < kGammaAtoms * nchK; j += kGammaThreads)
      bsh[j] = j < na * nchK ? B[(size_t)a0 * nchK + j] : T(0);
    __syncthreads();
  }
  double e[kGammaAtoms];
#pragma unroll
  for (int a = 0; a < kGammaAtoms; ++a) e[a] = 0.0;
  for (int k = tid; k < nchK; k += kGammaThreads) {
    double v[kGammaAtoms];
#pragma unroll
    for (int a = 0; a < kGammaAtoms; ++a) v[a] = wlin[k];
    if (B) {
      if constexpr (sizeof(T) == 4) {
        float h[kGammaAtoms], l[kGammaAtoms];
#pragma unroll
        for (int a = 0; a < kGammaAtoms; ++a) h[a] = l[a] = 0.f;
#pragma unroll 2
        for (int j = 0; j < nchK; ++j) {
          const float2 w = wsym32[(size_t)j * nchK + k];
#pragma unroll
          for (int a = 0; a < kGammaAtoms; ++a) ds_fma(h[a], l[a], bsh[a * nchK + j], w.x, w.y);
        }
#pragma unroll
        for (int a = 0; a < kGammaAtoms; ++a) v[a] += (double)h[a] + (double)l[a];
      } else {
        for (int j = 0; j < nchK; ++j) {
          const double w = wsym[(size_t)j * nchK + k];
#pragma unroll
          for (int a = 0; a < kGammaAtoms; ++a) v[a] = fma(w, (double)bsh[a * nchK + j], v[a]);
        }
      }
#pragma unroll
      for (int a = 0; a < kGammaAtoms; ++a) e[a] = fma(0.5 * (double)bsh[a * nchK + k], v[a] + wlin[k], e[a]);
    }
#pragma unroll
    for (int a = 0; a < kGammaAtoms; ++a) beta[a * nchK + k] = B ? (double)(T)v[a] : v[a];  // B: in the method's precision
  }
  __syncthreads();
  for (int b = tid; b < nch * nblk; b += kGammaThreads) {
    const int ch = b / nblk, i = b - ch * nblk;
    const int t0 = gam_off[i], t1 = gam_off[i + 1];
    double g[kGammaAtoms];
#pragma unroll
    for (int a = 0; a < kGammaAtoms; ++a) g[a] = 0.0;
    for (int t = t0; t < t1; ++t) {
      const GammaItem it = gam[t];
      const double sc = it.snum == it.sden ? 1.0 : (double)it.snum / (double)it.sden;
#pragma unroll
      for (int a = 0; a < kGammaAtoms; ++a) g[a] = fma(sc, beta[a * nchK + ch * K + it.k], g[a]);
    }
#pragma unroll
    for (int a = 0; a < kGammaAtoms; ++a)
      if (a < na) put_weight(gamma + (size_t)(a0 + a) * nch * nblk + b, g[a]);
  }
  if (!B) return;
#pragma unroll
  for (int a = 0; a < kGammaAtoms; ++a) {
    for (int o = 16; o > 0; o >>= 1) e[a] += __shfl_xor_sync(0xffffffffu, e[a], o);
    if ((tid & 31) == 0) red[a][tid >> 5] = e[a];
  }
  __syncthreads();
  if (tid < na) Eatom[a0 + tid] = w0 + red[tid][0] + red[tid][1] + red[tid][2] + red[tid][3];
}

}  // namespace

cudaError_t launch_split_pairs(const double* in, float2* out, size_t n, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  k_split_pairs<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(in, out, n);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_eval_gamma(const DevTables& tb, const T* B, int A, int nch, const double* wlin, const double* wsym,
                              const float2* wsym32, double w0, T* gamma, double* Eatom, cudaStream_t st) {
  if (A <= 0) return cudaSuccess;
  const size_t smem = (sizeof(double) + sizeof(T)) * kGammaAtoms * nch * tb.K;
  k_eval_gamma<T, T><<<(A + kGammaAtoms - 1) / kGammaAtoms, kGammaThreads, smem, st>>>(
      tb.gamp_off, tb.gamp, tb.NBLKP, nch, tb.K, A, B, wlin, wsym, wsym32, w0, gamma, Eatom);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_block_weights(const DevTables& tb, int nch, const double* wlin, void* gamma, cudaStream_t st) {
  using G = typename std::conditional<sizeof(T) == 4, float2, double>::type;
  const size_t smem = (sizeof(double) + sizeof(T)) * kGammaAtoms * nch * tb.K;
  k_eval_gamma<T, G><<<1, kGammaThreads, smem, st>>>(tb.gamp_off, tb.gamp, tb.NBLKP, nch, tb.K, 1, nullptr, wlin,
                                                     nullptr, nullptr, 0.0, static_cast<G*>(gamma), nullptr);
  return cudaGetLastError();
}

template cudaError_t launch_block_weights<double>(const DevTables&, int, const double*, void*, cudaStream_t);
template cudaError_t launch_block_weights<float>(const DevTables&, int, const double*, void*, cudaStream_t);

template cudaError_t launch_eval_gamma<double>(const DevTables&, const double*, int, int, const double*, const double*,
                                               const float2*, double, double*, double*, cudaStream_t);
template cudaError_t launch_eval_gamma<float>(const DevTables&, const float*, int, int, const double*, const double*,
                                              const float2*, double, float*, double*, cudaStream_t);

}  // namespace mld
