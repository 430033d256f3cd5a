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

#include "mld_internal.h"

namespace mld {

namespace {

constexpr int kGammaThreads = 128;

// One CTA per atom: beta[k] = w_lin[k] + sum_j Wsym[j][k] B[j] (Wsym symmetric, read by rows j
// so that consecutive threads read consecutive k), the atom's energy w0 + B . (beta + w_lin) / 2 and
// gamma of every channel and block.  B null: beta = w_lin, no energy.
template <typename T>
__global__ void __launch_bounds__(kGammaThreads) k_eval_gamma(const int* __restrict__ gam_off,
                                                              const GammaItem* __restrict__ gam, int nblk, int nch,
                                                              int K, const T* __restrict__ B,
                                                              const double* __restrict__ wlin,
                                                              const double* __restrict__ wsym, double w0,
                                                              T* __restrict__ gamma, double* __restrict__ Eatom) {
  extern __shared__ double bsh[];  // B, then beta: 2 * nch * K
  __shared__ double red[4];
  const int a = blockIdx.x, tid = threadIdx.x, nchK = nch * K;
  double* beta = bsh + nchK;
  if (B) {
    for (int j = tid; j < nchK; j += kGammaThreads) bsh[j] = (double)B[(size_t)a * nchK + j];
    __syncthreads();
  }
  double e = 0.0;
  for (int k = tid; k < nchK; k += kGammaThreads) {
    double v = wlin[k];
    if (B) {
      for (int j = 0; j < nchK; ++j) v = fma(wsym[(size_t)j * nchK + k], bsh[j], v);
      e = fma(0.5 * bsh[k], v + wlin[k], e);
    }
    beta[k] = (double)(T)v;  // the weights in the method's precision
  }
  __syncthreads();
  for (int b = tid; b < nch * nblk; b += kGammaThreads) {
    const int ch = b / nblk, i = b - ch * nblk;
    double g = 0.0;
    for (int t = gam_off[i]; t < gam_off[i + 1]; ++t)
      g = fma((double)gam[t].snum / (double)gam[t].sden, beta[ch * K + gam[t].k], g);
    gamma[(size_t)a * nch * nblk + b] = (T)g;
  }
  if (!B) return;
  for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  if ((tid & 31) == 0) red[tid >> 5] = e;
  __syncthreads();
  if (tid == 0) Eatom[a] = w0 + red[0] + red[1] + red[2] + red[3];
}

}  // namespace

template <typename T>
cudaError_t launch_eval_gamma(const DevTables& tb, const T* B, int A, int nch, const double* wlin, const double* wsym,
                              double w0, T* gamma, double* Eatom, cudaStream_t st) {
  if (A <= 0) return cudaSuccess;
  const size_t smem = sizeof(double) * 2 * nch * tb.K;
  if (B)
    k_eval_gamma<T><<<A, kGammaThreads, smem, st>>>(tb.gam_off, tb.gam, tb.NBLK, nch, tb.K, B, wlin, wsym, w0, gamma, Eatom);
  else
    k_eval_gamma<T><<<1, kGammaThreads, smem, st>>>(tb.gamp_off, tb.gamp, tb.NBLKP, nch, tb.K, nullptr, wlin, nullptr, w0,
                                                    gamma, nullptr);
  return cudaGetLastError();
}

template cudaError_t launch_eval_gamma<double>(const DevTables&, const double*, int, int, const double*, const double*,
                                               double, double*, double*, cudaStream_t);
template cudaError_t launch_eval_gamma<float>(const DevTables&, const float*, int, int, const double*, const double*,
                                              double, float*, double*, cudaStream_t);

}  // namespace mld
