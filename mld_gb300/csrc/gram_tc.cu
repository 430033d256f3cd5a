// Weighted Gram matrix G = X^T W X on the 5th-generation tensor cores (tcgen05) in BF16 split
// precision with FP32 accumulation: the mixed method's normal matrix (parameters.F90:1018-1099
// for the linear block, :404-421,476-1015 for the quadratic block of the QNML fit).
//
//   x' = sqrt(w_r) x_r,  x' = hi + lo  (hi = bf16(x'), lo = bf16(x' - hi)),
//   x'_i x'_j ~= hi_i hi_j + hi_i lo_j + lo_i hi_j      (three bf16 MMAs per K step)
//
// A row chunk of X is first transposed into K-major bf16 planes Xt_hi / Xt_lo (D x Mp, the design
// row index contiguous), so both MMA operands of an output tile (features i, features j) are
// 128 x 64 K-major slices of the same planes, fetched by TMA with 128-byte swizzle.  Feature rows
// beyond D and design rows beyond the chunk are zero-filled by TMA.
//
// Grid: (upper-triangle tile pairs) x (row splits), split-major so that the CTAs resident at one
// time read the same rows (L2 reuse).  Per CTA: warp 0 issues TMA loads into a 3-stage ring,
// warp 1 allocates four 128-column TMEM accumulators and issues tcgen05.mma from one thread,
// warps 2-17 drain the accumulators with tcgen05.ld into compensated FP32 sums.
//
// 60,000 rows x 1541 columns: k_gram_tc 705 -> 495 us (1.1 PFLOP/s of the three products), k_split_bf16
// 336 -> 165 us.  Of the first, 125 us were the last of three rounds of CTAs (gram_tc_splits); with
// two accumulators the MMAs waited for the epilogue's chain of load, wait and add.  What bounds it
// now is the operand traffic, 64 KB per 64-row slice of a tile: 11 TB/s from L2.  With several
// row splits each split writes its tile to a partial buffer and k_gram_tc_reduce adds the splits
// into the FP64 Gram in split order (without that buffer: FP64 atomics, order not fixed); with
// one split the CTA adds its tile directly.  Every mbarrier wait
// is bounded: on expiry the CTA sets *err, waits (bounded) for its copies in flight and still
// frees its TMEM.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "mld_internal.h"
#include "ptx.cuh"
#include "tc.cuh"

namespace mld {

namespace {

using tc::kTK;
using tc::kTM;
using tc::kTileBytes;
constexpr int kStages = 3;
constexpr int kStageBytes = 4 * kTileBytes;    // A_hi, A_lo, B_hi, B_lo
constexpr int kFlush = 1;                      // K slices per TMEM accumulation (64 design rows)
constexpr int kAcc = 4;                        // TMEM accumulators: the MMAs run ahead of the epilogue
constexpr int kEpiWarps = 16;                  // four per TMEM lane quarter, 32 columns each
constexpr int kGramThreads = 32 * (2 + kEpiWarps);
constexpr size_t kGramSmem = (size_t)kStages * kStageBytes + 1024 + 256;

using ptx::mbar_expect_tx;
using ptx::mbar_init;
using ptx::mbar_wait;
using ptx::smem_u32;
using ptx::tma_load_2d;
using tc::mma_bf16;
using tc::mma_commit;
using tc::sw128_desc;

// two FP32 values in one 64-bit register
__device__ __forceinline__ uint64_t pack2(uint32_t a, uint32_t b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ float part2(uint64_t v, int i) {
  uint32_t a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(v));
  return __uint_as_float(i ? b : a);
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// eight TMEM columns of the warp's lanes; the registers are valid after tmem_wait8
__device__ __forceinline__ void tmem_ld8(uint32_t (&v)[8], uint32_t taddr) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait8(uint32_t (&v)[8]) {
  // the registers are operands so that nothing that reads them moves above the wait
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7])::"memory");
}

}  // namespace

// Transpose rows [r0, r0 + rows) of X (row stride ldx, columns [c0, c0 + D)) into the K-major
// bf16 planes hi/lo (D x Mp), scaling row r by sqrt(w[r]); design rows [rows, Mp) are zeroed.
// grid.x: kSplitRows-row blocks of the chunk, grid.y: blocks of kSplitTiles tiles of 64 columns.
//
// A thread carries two rows of a column through shared memory as one float2 (row pair p at
// [p][column], odd stride: no bank conflicts either way), so a warp reads 128 bytes of a row of X
// and writes 128 bytes of a plane row; the next tile's loads are issued before this one's stores.
constexpr int kSplitTiles = 4, kSplitRows = 128, kSplitWarps = 16;

template <typename T>
__global__ void __launch_bounds__(32 * kSplitWarps) k_split_bf16(const T* __restrict__ X, int ldx, int c0, int D,
                                                    const double* __restrict__ w, long long r0, long long rows,
                                                    long long Mp, __nv_bfloat16* __restrict__ hi,
                                                    __nv_bfloat16* __restrict__ lo) {
  __shared__ float2 tile[kSplitRows / 2][65];
  __shared__ float sw[kSplitRows];
  const long long rb = (long long)blockIdx.x * kSplitRows;
  const int lane = threadIdx.x, wy = threadIdx.y;  // block (32, kSplitWarps)
  const int tid = wy * 32 + lane;
  const int nrow = (int)min((long long)kSplitRows, rows - rb);  // may be <= 0 in the zeroed rows
  // sqrt(w) and x' in FP32: the split keeps about 17 bits of x', and FP64 runs at 1/64 rate
  if (tid < kSplitRows) sw[tid] = tid < nrow ? (float)sqrt(w[r0 + rb + tid]) : 0.f;
  __syncthreads();
  const T* Xb = X + (r0 + rb) * ldx + c0;
  // warp wy holds row pairs wy, wy + 16, ... and column halves 0, 1 of a tile
  float2 v[4][2];
  auto load = [&](int cb) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = 2 * (wy + kSplitWarps * i), c = cb + 32 * h + lane;
        v[i][h].x = r < nrow && c < D ? (float)Xb[(long long)r * ldx + c] * sw[r] : 0.f;
        v[i][h].y = r + 1 < nrow && c < D ? (float)Xb[(long long)(r + 1) * ldx + c] * sw[r + 1] : 0.f;
      }
  };
  const int cbeg = blockIdx.y * (64 * kSplitTiles), cend = min(D, cbeg + 64 * kSplitTiles);
  load(cbeg);
  for (int cb = cbeg; cb < cend; cb += 64) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) tile[wy + kSplitWarps * i][32 * h + lane] = v[i][h];
    __syncthreads();
    if (cb + 64 < cend) load(cb + 64);
#pragma unroll
    for (int i = 0; i < 64 / kSplitWarps; ++i) {
      const int cl = wy + kSplitWarps * i, c = cb + cl;
#pragma unroll
      for (int g = 0; g < kSplitRows / 64; ++g) {
        const long long r = rb + 64 * g + 2 * lane;
        if (c < cend && r < Mp) {  // (Mp is even)
          const float2 x = tile[32 * g + lane][cl];
          const __nv_bfloat162 h = __floats2bfloat162_rn(x.x, x.y);
          const size_t o = (size_t)c * Mp + r;
          *reinterpret_cast<__nv_bfloat162*>(hi + o) = h;
          *reinterpret_cast<__nv_bfloat162*>(lo + o) =
              __floats2bfloat162_rn(x.x - __low2float(h), x.y - __high2float(h));
        }
      }
    }
    __syncthreads();
  }
}

// blockIdx.x = tile + ntile * split; tile enumerates the upper-triangle pairs ti <= tj.
// Row split s covers K slices [s * kps, min(nk, (s + 1) * kps)) of 64 design rows.
//
// The FP32 accumulator lives in TMEM for `flush` K slices only (kFlush = 1: 64 design rows), because
// the tensor core rounds its FP32 accumulation toward zero (a bias that grows with the chain): the MMA issuer
// cycles through kAcc 128-column TMEM buffers, and the epilogue warps drain the full ones
// into compensated (Kahan) FP32 register sums, so the error of the whole split stays at the
// level of one short FP32 accumulation.  Epilogue warp w reads TMEM lane quarter w % 4 and one
// quarter (32 columns) of the tile.
__global__ void __launch_bounds__(kGramThreads, 1)
    k_gram_tc(const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo, int nt,
              int ntile, int nk, int kps, int flush, int D, double* __restrict__ G, double* __restrict__ part,
              int* __restrict__ err, int skip_loads, long long wait_limit) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(tiles + kStages * kStageBytes);
  uint64_t* empty = full + kStages;
  uint64_t* tfull = empty + kStages;  // [kAcc] accumulator buffer ready for the epilogue
  uint64_t* tempty = tfull + kAcc;    // [kAcc] accumulator buffer drained
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + kAcc);

  int t = blockIdx.x % ntile, ti = 0;
  const int split = blockIdx.x / ntile;
  while (t >= nt - ti) {
    t -= nt - ti;
    ++ti;
  }
  const int tj = ti + t;
  const int kb = split * kps;
  const int nkl = min(nk, kb + kps) - kb;  // >= 1 by construction of the grid
  const int ngrp = (nkl + flush - 1) / flush;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < kAcc; ++b) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], kEpiWarps);
    }
    ptx::mbar_init_fence();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kAcc * kTM));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;
  bool ok = true;

  if (warp == 0 && lane == 0) {
    // producer: A = features of tile ti, B = features of tile tj
    int issued = 0;
    for (int k = 0; k < (skip_loads ? 0 : nkl); ++k) {
      const int s = k % kStages;
      if (k >= kStages && !mbar_wait(&empty[s], ((k / kStages) - 1) & 1, wait_limit)) {
        ok = false;
        break;
      }
      unsigned char* st = tiles + s * kStageBytes;
      const int x = (kb + k) * kTK;
      mbar_expect_tx(&full[s], kStageBytes);
      tma_load_2d(st, &map_hi, x, ti * kTM, &full[s]);
      tma_load_2d(st + kTileBytes, &map_lo, x, ti * kTM, &full[s]);
      tma_load_2d(st + 2 * kTileBytes, &map_hi, x, tj * kTM, &full[s]);
      tma_load_2d(st + 3 * kTileBytes, &map_lo, x, tj * kTM, &full[s]);
      issued = k + 1;
    }
    // the copies issued last may still be in flight: wait for them (bounded) before leaving
    for (int k = max(0, issued - kStages); k < issued; ++k) mbar_wait(&full[k % kStages], (k / kStages) & 1, wait_limit);
  } else if (warp == 1 && lane == 0) {
    // MMA issuer: K-slice group g accumulates into TMEM buffer g % kAcc
    for (int g = 0; g < ngrp && ok; ++g) {
      const int b = g % kAcc;
      if (g >= kAcc && !mbar_wait(&tempty[b], ((g / kAcc) - 1) & 1, wait_limit)) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t acc = tmem + (uint32_t)(b * kTM);
      const int k1 = min(nkl, (g + 1) * flush);
      for (int k = g * flush; k < k1; ++k) {
        const int s = k % kStages;
        if (!mbar_wait(&full[s], (k / kStages) & 1, wait_limit)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t st = smem_u32(tiles + s * kStageBytes);
#pragma unroll
        for (int kk = 0; kk < kTK / 16; ++kk) {
          const uint32_t off = kk * 32;  // 16 bf16 along K inside the 128-byte swizzle row
          const uint64_t ahi = sw128_desc(st + off), alo = sw128_desc(st + kTileBytes + off);
          const uint64_t bhi = sw128_desc(st + 2 * kTileBytes + off), blo = sw128_desc(st + 3 * kTileBytes + off);
          mma_bf16(acc, ahi, bhi, (k > g * flush || kk > 0) ? 1u : 0u);
          mma_bf16(acc, ahi, blo, 1u);
          mma_bf16(acc, alo, bhi, 1u);
        }
        mma_commit(&empty[s]);  // frees the stage once these MMAs have read it
      }
      mma_commit(&tfull[b]);
    }
  } else if (warp >= 2) {
    // epilogue: Kahan sums of 32 columns of one TMEM lane quarter
    const int q = warp & 3, cq = (warp - 2) >> 2;
    uint64_t sum[16], cmp[16];  // column pairs
#pragma unroll
    for (int c = 0; c < 16; ++c) sum[c] = cmp[c] = 0;
    // Eight columns at a time, the next eight (of this or the next accumulator) on their way while
    // these are added; an accumulator is given back as soon as its last columns are in registers.
    const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(cq * 32);
    uint32_t v[2][8];
    bool got = mbar_wait(&tfull[0], 0, wait_limit);
    if (got) {
      asm volatile("tcgen05.fence::after_thread_sync;");
      tmem_ld8(v[0], tbase);
    }
    for (int g = 0; g < ngrp && got; ++g) {
      const uint32_t tb = tbase + (uint32_t)(g % kAcc * kTM);
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        tmem_wait8(v[h & 1]);
        if (h < 3) {
          tmem_ld8(v[(h + 1) & 1], tb + (h + 1) * 8);
        } else {
          asm volatile("tcgen05.fence::before_thread_sync;");
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&tempty[g % kAcc]);
          if (g + 1 < ngrp) {
            got = mbar_wait(&tfull[(g + 1) % kAcc], ((g + 1) / kAcc) & 1, wait_limit);
            asm volatile("tcgen05.fence::after_thread_sync;");
            if (got) tmem_ld8(v[0], tbase + (uint32_t)((g + 1) % kAcc * kTM));
          }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int e = h * 4 + c;
          const uint64_t y = sub2(pack2(v[h & 1][2 * c], v[h & 1][2 * c + 1]), cmp[e]);
          const uint64_t tt = add2(sum[e], y);
          cmp[e] = sub2(sub2(tt, sum[e]), y);
          sum[e] = tt;
        }
      }
    }
    if (got && part) {
      // this split's tile, added to G in split order by k_gram_tc_reduce
      double* pt = part + ((size_t)split * ntile + blockIdx.x % ntile) * (kTM * kTM) + (size_t)(q * 32 + lane) * kTM +
                   cq * 32;
#pragma unroll
      for (int c = 0; c < 16; ++c)
        *reinterpret_cast<double2*>(pt + 2 * c) =
            make_double2((double)part2(sum[c], 0) - (double)part2(cmp[c], 0),
                         (double)part2(sum[c], 1) - (double)part2(cmp[c], 1));
    } else if (got) {
      // straight into G: with a single split the CTA is the only writer of these elements
      const int i = ti * kTM + q * 32 + lane;
      if (i < D) {
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          const int j = tj * kTM + cq * 32 + c;
          if (j < D && j >= i)
            atomicAdd(&G[(size_t)i * D + j], (double)part2(sum[c >> 1], c & 1) - (double)part2(cmp[c >> 1], c & 1));
        }
      }
    } else if (lane == 0) {
      atomicExch(err, 1);
    }
  }
  if (!ok) atomicExch(err, 1);
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kAcc * kTM));
  }
}

// ---------------------------------------------------------------------------------------
// Test hook of the timeout path: with skip_loads the producer issues no TMA loads, so the MMA
// and epilogue warps' bounded waits expire (after wait_limit clocks), the CTA reports *err = 1
// and frees its TMEM.  (0, 0) restores normal operation.
namespace {
int g_skip_loads = 0;
long long g_wait_limit = ptx::kWaitLimit;
}  // namespace
void gram_tc_test_timeout(int skip_loads, long long wait_limit) {
  g_skip_loads = skip_loads ? 1 : 0;
  g_wait_limit = wait_limit > 0 ? wait_limit : ptx::kWaitLimit;
}

size_t gram_tc_min_workspace(int D) { return (size_t)4 * D * kTK + 256; }

namespace {
// Row splits of one chunk of nk 64-row slices.  One CTA runs per SM, so the chunk takes
// rounds(ns) = ceil(ntile ns / nsm) times the slices of a split plus a CTA's own cost (ring fill,
// partial tile), about kSplitCost slices; ns makes that least among those whose partials fit
// (gram_tc_max_splits).  1541 columns x 60,000 rows: 91 tiles, 5 splits fill 2.99 rounds; the 4 that
// "two waves of CTAs" asks for filled 2.39 of 3.
constexpr int kSplitCost = 8;
int gram_tc_max_splits(int ntile, int nsm) { return std::max(1, (3 * nsm + ntile / 2) / ntile); }
int gram_tc_splits(int nk, int ntile, int nsm, int* kps) {
  const int most = std::min(nk, gram_tc_max_splits(ntile, nsm));
  long long best = 0;
  int ns = 1;
  for (int s = 1; s <= most; ++s) {
    const long long per = (nk + s - 1) / s, n = (nk + per - 1) / per;  // n splits, none empty
    const long long t = ((long long)ntile * n + nsm - 1) / nsm * (per + kSplitCost);
    if (s == 1 || t < best) {
      best = t;
      ns = (int)n;
      *kps = (int)per;
    }
  }
  return ns;
}

// G[i][j] += sum over the splits of their tile partials, in split order (upper triangle).
__global__ void k_gram_tc_reduce(const double* __restrict__ part, int nt, int ntile, int nsplit, int D,
                                 double* __restrict__ G) {
  const int tile = blockIdx.y;
  int t = tile, ti = 0;
  while (t >= nt - ti) {
    t -= nt - ti;
    ++ti;
  }
  const int tj = ti + t;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;  // element of the kTM x kTM tile
  if (e >= kTM * kTM) return;
  const int i = ti * kTM + e / kTM, j = tj * kTM + e % kTM;
  if (i >= D || j >= D || j < i) return;
  double s = 0.0;
#pragma unroll 16
  for (int sp = 0; sp < nsplit; ++sp) s += part[((size_t)sp * ntile + tile) * (kTM * kTM) + e];
  G[(size_t)i * D + j] += s;
}
}  // namespace

size_t gram_tc_part_doubles(int D, int nsm) {
  const int nt = (D + kTM - 1) / kTM, ntile = nt * (nt + 1) / 2;
  const int ns = gram_tc_max_splits(ntile, nsm);
  return ns > 1 ? (size_t)ns * ntile * kTM * kTM : 0;  // one split per chunk: no partials
}

bool gram_tc_available() { return tc::encode_fn() != nullptr; }

// G (FP64, D x D, upper triangle) += sum over rows r of w_r x_r x_r^T for columns [c0, c0 + D)
// of X (M rows, stride ldx).  `ws` holds ws_bytes >= gram_tc_min_workspace(D) bytes; the rows
// are processed in chunks that fit it.  The caller zeroes G and *err and symmetrises G.
template <typename T>
cudaError_t launch_gram_tc(const T* X, int ldx, int c0, int D, const double* w, long long M, double* G, void* ws,
                           size_t ws_bytes, int* err, int nsm, cudaStream_t st, double* part, size_t part_doubles) {
  if (M <= 0 || D <= 0) return cudaSuccess;
  if (ws_bytes < gram_tc_min_workspace(D) || ((uintptr_t)ws & 15)) return cudaErrorInvalidValue;
  // chunk rows: a multiple of 64 whose two planes fit the workspace
  long long chunk = (long long)((ws_bytes - 256) / (4 * (size_t)D)) / kTK * kTK;
  chunk = std::min(chunk, (M + kTK - 1) / kTK * kTK);
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(k_gram_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGramSmem);
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  const int nt = (D + kTM - 1) / kTM;
  const int ntile = nt * (nt + 1) / 2;
  __nv_bfloat16* hi = reinterpret_cast<__nv_bfloat16*>(ws);
  for (long long r0 = 0; r0 < M; r0 += chunk) {
    const long long rows = std::min(chunk, M - r0);
    const long long Mp = (rows + 7) / 8 * 8;  // 16-byte plane row stride
    __nv_bfloat16* lo = hi + (size_t)D * Mp;
    dim3 g1((unsigned)((Mp + kSplitRows - 1) / kSplitRows), (unsigned)((D + 64 * kSplitTiles - 1) / (64 * kSplitTiles)));
    k_split_bf16<T><<<g1, dim3(32, kSplitWarps), 0, st>>>(X, ldx, c0, D, w, r0, rows, Mp, hi, lo);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    CUtensorMap mh, ml;
    if (!tc::make_plane_map(&mh, hi, Mp, D, Mp) || !tc::make_plane_map(&ml, lo, Mp, D, Mp)) return cudaErrorInvalidValue;
    const int nk = (int)((rows + kTK - 1) / kTK);
    int kps = 1;
    const int nsplit = gram_tc_splits(nk, ntile, nsm, &kps);
    // several splits of a tile: per-split partials reduced in split order when the workspace
    // holds them (deterministic); otherwise FP64 atomics (order of the splits not fixed)
    const bool use_part = nsplit > 1 && part && part_doubles >= (size_t)nsplit * ntile * kTM * kTM;
    double* pt = use_part ? part : nullptr;
    k_gram_tc<<<(unsigned)(ntile * nsplit), kGramThreads, kGramSmem, st>>>(mh, ml, nt, ntile, nk, kps, kFlush, D, G,
                                                                           pt, err, g_skip_loads, g_wait_limit);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (use_part) {
      k_gram_tc_reduce<<<dim3((kTM * kTM + 255) / 256, (unsigned)ntile), 256, 0, st>>>(part, nt, ntile, nsplit, D, G);
      e = cudaGetLastError();
      if (e != cudaSuccess) return e;
    }
  }
  return cudaSuccess;
}

template cudaError_t launch_gram_tc<float>(const float*, int, int, int, const double*, long long, double*, void*,
                                           size_t, int*, int, cudaStream_t, double*, size_t);
template cudaError_t launch_gram_tc<double>(const double*, int, int, int, const double*, long long, double*, void*,
                                            size_t, int*, int, cudaStream_t, double*, size_t);

}  // namespace mld
