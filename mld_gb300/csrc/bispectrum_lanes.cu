// Sums over the Clebsch-Gordan (Z) terms with a lane per atom: the descriptors B, and y = dE/dc for
// the evaluation.
//
// Inside a CTA that works on one atom, the Z terms are lanes: their index lists, extents and
// coefficients differ, so operands are gathered with bank conflicts, lanes idle where extents
// differ, and every term forms its own products of c.  Here the 32 lanes of a warp hold 32 atoms
// and run the same term: control flow is uniform, coefficients are broadcast, c (entry, atom) is
// read without conflicts, and the products of an operand pair (jA, jB) are formed once for all its
// output layers jO,
//   Z_jO(m1,m2) = sum_a CG_jO(a; m1) sum_b CG_jO(b; m2) c^jA[a, b] c^jB[m1 - a, m2 - b]
// (17.3k products and 163k FMAs per channel at j_max 4, against 42.6k and 255k of the term lists).
// The sums that the terms feed stay in registers: no term is stored.
//   B  a job is an operand pair: B_k = sum_m w Re(conj(c^l(m)) Z_l(m)) of its triples (l >= jA)
//   y  a job is an output position (m1, m2): y_jO(m1,m2) = sum over the pairs of gamma Z_jO(m1,m2)
// Four warps share a job (its records in four fixed parts of equal work, added in order), so the
// sums do not depend on the number of atoms or on how the jobs fall on the CTAs.
//
// Bound: shared-memory reads in FP32 (two 8-byte operands per product), the FP64 pipe in FP64.
#include <cuda_runtime.h>

#include <algorithm>

#include "bispectrum.cuh"

namespace mld {

namespace {

constexpr int kGroups = kNW / 4;  // four warps share a job

template <typename T>
struct LaneArgs {
  DevTables tb;
  const LaneRec* recs;
  const LaneJob* jobs;
  int njobs;
  const T* cg;
  const cx<T>* c;       // A x nch x HU
  const int* nbr_off;   // of the first atom
  const T* gamma;       // y: nch * NBLKP
  int A, nch;
  T* B;                 // A x nch*K
  cx<T>* y;             // A x nch x HU
};

// lanes that hold atoms: 32, or 16 where the c of 32 atoms does not fit in shared memory
struct LanePlan {
  int width, stride;
  size_t c, cg, gamma, part, total;
};

__host__ __device__ inline size_t upl(size_t x) { return (x + 15) & ~(size_t)15; }

__host__ __device__ inline LanePlan lane_plan(const DevTables& tb, int eb, int width) {
  LanePlan s;
  s.width = width;
  s.stride = width + 1;
  size_t o = 0;
  s.c = o;     o = upl(o + (size_t)2 * eb * tb.NU * s.stride);
  s.cg = o;    o = upl(o + (eb == 4 ? (size_t)eb * tb.NCGV : 0));  // FP64 reads them through the cache
  s.gamma = o; o = upl(o + (size_t)eb * tb.NBLKP);
  s.part = o;  o = upl(o + (size_t)kGroups * 4 * (tb.J / 2 + 1) * 32 * 2 * eb);
  s.total = o;
  return s;
}

// C consecutive b of a record, all its a: zs[o] += sum_a c1[a][o] sum_{b<C} c2[b][o] c c, o < NJ
template <int NJ, int C, typename T>
__device__ __forceinline__ void lane_chunk(const cx<T>* __restrict__ pa, const cx<T>* __restrict__ pb, int ST, int da,
                                           int db, int na, const T* __restrict__ c1p, int st1,
                                           const T* __restrict__ c2p, int st2, cx<T>* zs) {
  T c2[C][NJ];
#pragma unroll
  for (int b = 0; b < C; ++b)
#pragma unroll
    for (int o = 0; o < NJ; ++o) c2[b][o] = c2p[b * st2 + o];
  for (int a = 0; a < na; ++a) {
    cx<T> part[NJ];
#pragma unroll
    for (int b = 0; b < C; ++b) {
      const cx<T> u = pa[b * ST], v = pb[-b * ST];
      const cx<T> pr = {fma(u.x, v.x, -(u.y * v.y)), fma(u.x, v.y, u.y * v.x)};
#pragma unroll
      for (int o = 0; o < NJ; ++o) {
        if (b == 0) {
          part[o] = {c2[b][o] * pr.x, c2[b][o] * pr.y};
        } else {
          part[o].x = fma(c2[b][o], pr.x, part[o].x);
          part[o].y = fma(c2[b][o], pr.y, part[o].y);
        }
      }
    }
#pragma unroll
    for (int o = 0; o < NJ; ++o) {
      const T c1 = c1p[o];
      zs[o].x = fma(c1, part[o].x, zs[o].x);
      zs[o].y = fma(c1, part[o].y, zs[o].y);
    }
    c1p += st1;
    pa += da;
    pb -= db;
  }
}

// Z of the NJ output layers of a record
template <int NJ, typename T>
__device__ __forceinline__ void lane_terms(uint4 z0, const cx<T>* __restrict__ cl, int ST, const T* __restrict__ cg,
                                           cx<T>* zs) {
  // x = i1 | i2 << 16, y = cg1 | cg2 << 16, z = na | nb << 8 | s1 << 16 | s2 << 24, w = st1 | st2 << 8 | ..
  const cx<T>* pa = cl + (size_t)(z0.x & 0xFFFF) * ST;
  const cx<T>* pb = cl + (size_t)(z0.x >> 16) * ST;
  const int na = z0.z & 0xFF, da = ((z0.z >> 16) & 0xFF) * ST, db = (z0.z >> 24) * ST;
  const int st1 = z0.w & 0xFF, st2 = (z0.w >> 8) & 0xFF;
  const T* c1p = cg + (z0.y & 0xFFFF);
  const T* c2p = cg + (z0.y >> 16);
  int nb = (z0.z >> 8) & 0xFF;
#pragma unroll
  for (int o = 0; o < NJ; ++o) zs[o] = {T(0), T(0)};
  for (; nb >= 4; nb -= 4) {
    lane_chunk<NJ, 4>(pa, pb, ST, da, db, na, c1p, st1, c2p, st2, zs);
    pa += 4 * ST;
    pb -= 4 * ST;
    c2p += 4 * st2;
  }
  if (nb == 1) lane_chunk<NJ, 1>(pa, pb, ST, da, db, na, c1p, st1, c2p, st2, zs);
  else if (nb == 2) lane_chunk<NJ, 2>(pa, pb, ST, da, db, na, c1p, st1, c2p, st2, zs);
  else if (nb == 3) lane_chunk<NJ, 3>(pa, pb, ST, da, db, na, c1p, st1, c2p, st2, zs);
}

__device__ __forceinline__ int out_of(uint4 z1, int o) {
  const unsigned w = o < 2 ? z1.x : (o < 4 ? z1.y : z1.z);
  return (w >> (16 * (o & 1))) & 0xFFFF;
}

// A record into the job's sums.  y: acc[off + o] += gamma[out_o] Z_o; B: acc[o].x += w Re(conj(c[out_o]) Z_o)
template <int NJ, bool kY, typename T>
__device__ __forceinline__ void lane_record(uint4 z0, uint4 z1, const cx<T>* __restrict__ cl, int ST,
                                            const T* __restrict__ cg, const T* __restrict__ gam, cx<T>* acc) {
  cx<T> zs[NJ];
  lane_terms<NJ, T>(z0, cl, ST, cg, zs);
  if constexpr (kY) {
    const int off = z0.w >> 24;
#pragma unroll
    for (int o = 0; o < NJ; ++o) {
      const T g = gam[out_of(z1, o)];
#pragma unroll
      for (int k = 0; k + o < kMaxZOut; ++k)
        if (k == off) {
          acc[k + o].x = fma(g, zs[o].x, acc[k + o].x);
          acc[k + o].y = fma(g, zs[o].y, acc[k + o].y);
        }
    }
  } else {
    const T w = (T)(z1.w & 0xFFFF);
#pragma unroll
    for (int o = 0; o < NJ; ++o) {
      const cx<T> c = cl[(size_t)out_of(z1, o) * ST];
      acc[o].x = fma(w, fma(c.x, zs[o].x, c.y * zs[o].y), acc[o].x);
    }
  }
}

template <typename T, bool kY>
__global__ void __launch_bounds__(kNW * 32, sizeof(T) == 4 ? 2 : 1) k_lanes(LaneArgs<T> args, int width) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const DevTables& tb = args.tb;
  const LanePlan sp = lane_plan(tb, (int)sizeof(T), width);
  const int ST = sp.stride, HU = tb.HU, K = tb.K;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ch = blockIdx.z, a0 = blockIdx.x * width;
  const int na = min(width, args.A - a0);
  cx<T>* sc = reinterpret_cast<cx<T>*>(smem_raw + sp.c);
  T* sg = reinterpret_cast<T*>(smem_raw + sp.gamma);
  cx<T>* part = reinterpret_cast<cx<T>*>(smem_raw + sp.part);
  const T* cg = args.cg;
  // c of the atoms, expanded to full layers; a warp per atom
  for (int a = warp; a < width; a += kNW) {
    const cx<T>* src = args.c + ((size_t)(a0 + min(a, na - 1)) * args.nch + ch) * HU;
    for (int f = lane; f < tb.NU; f += 32) sc[(size_t)f * ST + a] = fetch(src, tb.expand[f]);
  }
  if constexpr (sizeof(T) == 4) {
    T* scg = reinterpret_cast<T*>(smem_raw + sp.cg);
    for (int e = tid; e < tb.NCGV; e += kNW * 32) scg[e] = args.cg[e];
    cg = scg;
  }
  if constexpr (kY) {
    for (int b = tid; b < tb.NBLKP; b += kNW * 32) sg[b] = args.gamma[ch * tb.NBLKP + b];
  }
  __syncthreads();
  const int al = lane < width ? lane : lane - width;  // (16 atoms: both halves of the warp hold them)
  const int atom = a0 + al;
  const bool mine = lane < width && al < na;
  const cx<T>* cl = sc + al;
  const int group = warp >> 2, q = warp & 3, no = tb.J / 2 + 1;
  const bool alone = !kY && (mine ? args.nbr_off[atom + 1] == args.nbr_off[atom] : false);
  cx<T>* mypart = part + (size_t)group * 4 * no * 32;
  for (int job = blockIdx.y * kGroups + group; job < args.njobs; job += gridDim.y * kGroups) {
    const LaneJob& jb = args.jobs[job];
    cx<T> acc[kMaxZOut];
#pragma unroll
    for (int o = 0; o < kMaxZOut; ++o) acc[o] = {T(0), T(0)};
    const int r0 = jb.rec[q], r1 = jb.rec[q + 1];
    const uint4* rp = reinterpret_cast<const uint4*>(args.recs);
    uint4 n0 = make_uint4(0, 0, 0, 0), n1 = n0;
    if (r0 < r1) {
      n0 = __ldg(rp + 2 * (size_t)r0);
      n1 = __ldg(rp + 2 * (size_t)r0 + 1);
    }
    for (int r = r0; r < r1; ++r) {
      const uint4 z0 = n0, z1 = n1;
      if (r + 1 < r1) {
        n0 = __ldg(rp + 2 * (size_t)(r + 1));
        n1 = __ldg(rp + 2 * (size_t)(r + 1) + 1);
      }
      switch ((z0.w >> 16) & 0xFF) {
        case 1: lane_record<1, kY, T>(z0, z1, cl, ST, cg, sg, acc); break;
        case 2: lane_record<2, kY, T>(z0, z1, cl, ST, cg, sg, acc); break;
        case 3: lane_record<3, kY, T>(z0, z1, cl, ST, cg, sg, acc); break;
        case 4: lane_record<4, kY, T>(z0, z1, cl, ST, cg, sg, acc); break;
        case 5: lane_record<5, kY, T>(z0, z1, cl, ST, cg, sg, acc); break;
        default: lane_record<6, kY, T>(z0, z1, cl, ST, cg, sg, acc); break;
      }
    }
#pragma unroll
    for (int o = 0; o < kMaxZOut; ++o)
      if (o < no) mypart[(q * no + o) * 32 + lane] = acc[o];
    asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");
    for (int o = q; o < jb.nout; o += 4) {
      cx<T> v = mypart[o * 32 + lane];
#pragma unroll
      for (int p = 1; p < 4; ++p) {
        const cx<T> w = mypart[(p * no + o) * 32 + lane];
        v = {v.x + w.x, v.y + w.y};
      }
      if (mine) {
        if constexpr (kY) args.y[((size_t)atom * args.nch + ch) * HU + jb.out[o]] = v;
        else args.B[((size_t)atom * args.nch + ch) * K + jb.out[o]] = alone ? T(0) : v.x;
      }
    }
    asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");
  }
}

// ---- c of every atom ---------------------------------------------------------------------------
template <typename T>
struct CArgs {
  DevTables tb;
  PairSource<T> src;
  const int* nbr_off;
  T chw[kMaxCh * kMaxTypes];
  T rin[kMaxTypes * kMaxTypes];
  int nch;
  const int* order;
  int first;
  int* counter;
  unsigned long long chains;
  int slots;
  cx<T>* c;
};

struct CPlan {
  size_t hd, zx, fcw, next, c, U, total;
};

__host__ __device__ inline CPlan c_plan(const DevTables& tb, int nch, int eb, int slots) {
  CPlan s;
  size_t o = 0;
  s.hd = o;   o = upl(o + tb.HU);
  s.zx = o;   o = upl(o + (size_t)eb * 4 * slots);
  s.fcw = o;  o = upl(o + (size_t)eb * nch * slots);
  s.next = o; o = upl(o + 16);
  s.c = o;    o = upl(o + (size_t)2 * eb * nch * tb.HU);
  s.U = o;    o = upl(o + (size_t)2 * eb * u_stride(tb.HU) * slots);
  s.total = o;
  return s;
}

// c on half layers, one atom per CTA turn (bispectrum.cuh: geometry, column chains, ordered sum)
template <typename T>
__global__ void __launch_bounds__(kNW * 32, sizeof(T) == 4 ? 2 : 1) k_c_half(CArgs<T> args, int A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const DevTables& tb = args.tb;
  const int HU = tb.HU, nch = args.nch, HS = u_stride(HU);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int nth = kNW * 32;
  const CPlan sp = c_plan(tb, nch, (int)sizeof(T), args.slots);
  int8_t* shd = reinterpret_cast<int8_t*>(smem_raw + sp.hd);
  T* zx = reinterpret_cast<T*>(smem_raw + sp.zx);
  T* fcw = reinterpret_cast<T*>(smem_raw + sp.fcw);
  int* snext = reinterpret_cast<int*>(smem_raw + sp.next);
  cx<T>* chalf = reinterpret_cast<cx<T>*>(smem_raw + sp.c);
  cx<T>* Us = reinterpret_cast<cx<T>*>(smem_raw + sp.U);
  for (int e = tid; e < HU; e += nth) shd[e] = tb.half_diag[e];
  int nxt = 0;
  if (tid == 0) nxt = atomicAdd(args.counter, 1);
  for (;;) {
    if (tid == 0) snext[0] = nxt;
    __syncthreads();
    const int qi = snext[0];
    if (qi >= A) break;
    if (tid == 0) nxt = atomicAdd(args.counter, 1);
    const int atom = args.order ? args.order[qi] : args.first + qi;
    const int ti = args.src.types[atom];
    const int p0 = args.nbr_off[atom];
    const int nn = args.nbr_off[atom + 1] - p0;
    for (int base = 0; base < nn; base += args.slots) {
      const int count = min(args.slots, nn - base);
      for (int n = tid; n < count; n += nth) {
        T g[kGeo];
        int nb, tn;
        pair_geometry<T>(args.src, args.rin, (size_t)(p0 + base + n), ti, g, &nb, &tn);
        for (int ch = 0; ch < nch; ++ch) fcw[n * nch + ch] = g[kGeoFc] * args.chw[ch * args.src.ntypes + tn];
#pragma unroll
        for (int k = 0; k < 4; ++k) zx[n * 4 + k] = g[kGeoZx + k];
        Us[(size_t)n * HS] = {T(1), T(0)};
      }
      __syncthreads();
      u_store<T>(Us, HS, count, tb.J, args.chains, warp, lane, [&](int n) { return zx + n * 4; });
      __syncthreads();
      c_sum<T>(chalf, Us, HS, fcw, shd, count, nch, HU, base == 0, base + args.slots >= nn, tid);
      if (base + args.slots < nn) __syncthreads();
    }
    cx<T>* out = args.c + (size_t)(atom - args.first) * nch * HU;
    // a thread writes the entries it has summed itself
    for (int e = tid; e < nch * HU; e += nth)
      out[e] = nn > 0 ? chalf[e] : cx<T>{shd[e % HU] ? T(1) : T(0), T(0)};
  }
}

int optin() {
  static int v = 0;
  if (!v) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  }
  return v;
}

cudaError_t sm_count(int* nsm) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(nsm, cudaDevAttrMultiProcessorCount, dev);
  return e;
}

template <typename T, bool kY>
cudaError_t launch_lanes(LaneArgs<T>& a, cudaStream_t st) {
  if (a.A <= 0 || a.njobs <= 0) return cudaSuccess;
  int width = 32;
  size_t smem = lane_plan(a.tb, (int)sizeof(T), width).total;
  if (smem > (size_t)optin()) {
    width = 16;
    smem = lane_plan(a.tb, (int)sizeof(T), width).total;
  }
  if (smem > (size_t)optin()) return cudaErrorInvalidConfiguration;
  cudaError_t e = cudaFuncSetAttribute(k_lanes<T, kY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int nsm = 0;
  if ((e = sm_count(&nsm)) != cudaSuccess) return e;
  // the jobs of a tile of atoms are spread over CTAs until about four rounds of CTAs fill the GPU; a
  // CTA keeps at least two jobs per group, or its load of c would outweigh them
  const int tiles = (a.A + width - 1) / width;
  const int most = std::max(1, a.njobs / (2 * kGroups));
  const int slices = std::min(most, std::max(1, 8 * nsm / (tiles * a.nch)));
  k_lanes<T, kY><<<dim3(tiles, slices, a.nch), kNW * 32, smem, st>>>(a, width);
  return cudaGetLastError();
}

}  // namespace

template <typename T>
cudaError_t launch_c_half(const DevTables& tb, const DevBatch& b, const BsoParams& p, int first, int count,
                          const int* order, int* counter, void* c, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  CArgs<T> a{};
  a.tb = tb;
  a.src = {b.types, b.nbr_idx, b.nbr_u, sizeof(T) == 4 ? b.nbr_u32 : nullptr, (T)p.rcut, (T)p.inv_r0,
           (T)p.rin_width, p.ntypes, p.has_rin};
  a.nbr_off = b.nbr_off;
  for (int e = 0; e < kMaxCh * kMaxTypes; ++e) a.chw[e] = (T)p.chw[e];
  for (int e = 0; e < kMaxTypes * kMaxTypes; ++e) a.rin[e] = (T)p.rin[e];
  a.nch = p.nch;
  a.order = order;
  a.first = first;
  a.counter = counter;
  a.chains = chain_order(tb.J);
  a.c = static_cast<cx<T>*>(c);
  const size_t per_sm = 228 * 1024;
  const size_t ctas = sizeof(T) == 4 ? 2 : 1;
  a.slots = 8;
  for (int s = 64; s > 8; s -= 8)
    if (per_sm / (c_plan(tb, p.nch, (int)sizeof(T), s).total + 1024) >= ctas &&
        c_plan(tb, p.nch, (int)sizeof(T), s).total <= (size_t)optin()) {
      a.slots = s;
      break;
    }
  const size_t smem = c_plan(tb, p.nch, (int)sizeof(T), a.slots).total;
  if (smem > (size_t)optin()) return cudaErrorInvalidConfiguration;
  cudaError_t e = cudaFuncSetAttribute(k_c_half<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int nsm = 0, occ = 0;
  if ((e = sm_count(&nsm)) != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_c_half<T>, kNW * 32, smem);
  if (e != cudaSuccess) return e;
  if (occ < 1) return cudaErrorInvalidConfiguration;
  e = cudaMemsetAsync(counter, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  k_c_half<T><<<(unsigned)std::min<long long>(count, (long long)nsm * occ), kNW * 32, smem, st>>>(a, count);
  return cudaGetLastError();
}

template <typename T>
static LaneArgs<T> lane_args(const DevTables& tb, const DevBatch& b, const BsoParams& p, int first, int count,
                             const void* c) {
  LaneArgs<T> a{};
  a.tb = tb;
  if constexpr (sizeof(T) == 8) a.cg = tb.cgv64;
  else a.cg = tb.cgv32;
  a.c = static_cast<const cx<T>*>(c);
  a.nbr_off = b.nbr_off + first;
  a.A = count;
  a.nch = p.nch;
  return a;
}

template <typename T>
cudaError_t launch_lane_descriptors(const DevTables& tb, const DevBatch& b, const BsoParams& p, int first, int count,
                                    const void* c, T* B, cudaStream_t st) {
  LaneArgs<T> a = lane_args<T>(tb, b, p, first, count, c);
  a.recs = tb.brecs;
  a.jobs = tb.bjobs;
  a.njobs = tb.NBJ;
  a.B = B + (size_t)first * p.nch * tb.K;
  return launch_lanes<T, false>(a, st);
}

template <typename T>
cudaError_t launch_lane_y(const DevTables& tb, const DevBatch& b, const BsoParams& p, int first, int count,
                          const void* c, const T* gamma, void* y, cudaStream_t st) {
  LaneArgs<T> a = lane_args<T>(tb, b, p, first, count, c);
  a.recs = tb.yrecs;
  a.jobs = tb.yjobs;
  a.njobs = tb.NYJ;
  a.gamma = gamma;
  a.y = static_cast<cx<T>*>(y);
  return launch_lanes<T, true>(a, st);
}

template cudaError_t launch_c_half<double>(const DevTables&, const DevBatch&, const BsoParams&, int, int, const int*,
                                           int*, void*, cudaStream_t);
template cudaError_t launch_c_half<float>(const DevTables&, const DevBatch&, const BsoParams&, int, int, const int*,
                                          int*, void*, cudaStream_t);
template cudaError_t launch_lane_descriptors<double>(const DevTables&, const DevBatch&, const BsoParams&, int, int,
                                                     const void*, double*, cudaStream_t);
template cudaError_t launch_lane_descriptors<float>(const DevTables&, const DevBatch&, const BsoParams&, int, int,
                                                    const void*, float*, cudaStream_t);
template cudaError_t launch_lane_y<double>(const DevTables&, const DevBatch&, const BsoParams&, int, int, const void*,
                                           const double*, void*, cudaStream_t);
template cudaError_t launch_lane_y<float>(const DevTables&, const DevBatch&, const BsoParams&, int, int, const void*,
                                          const float*, void*, cudaStream_t);

}  // namespace mld
