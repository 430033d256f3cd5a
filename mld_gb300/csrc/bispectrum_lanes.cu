// Sums over the Clebsch-Gordan (Z) terms with atoms on lanes: the descriptors B, and y = dE/dc for
// the evaluation.
//
// Inside a CTA that works on one atom, the Z terms are lanes: their index lists, extents and
// coefficients differ, so operands are gathered with bank conflicts, lanes idle where extents
// differ, and every term forms its own products of c.  Here the lanes of a warp hold atoms and run
// the same term: control flow is uniform, coefficients are broadcast, c (entry, atom) is read
// without conflicts, and the products of an operand pair (jA, jB) are formed once for all its
// output layers jO,
//   Z_jO(m1,m2) = sum_a CG_jO(a; m1) sum_b CG_jO(b; m2) c^jA[a, b] c^jB[m1 - a, m2 - b]
// (17.3k products and 163k FMAs per channel at j_max 4, against 42.6k and 255k of the term lists).
// In FP32 a lane holds two atoms, whose values are packed for the two-wide FP32 instructions: half
// the instructions per atom for the products, and half the loads of coefficients and records.
// For B and y the sums that the terms feed stay in registers: no term is stored.
//   B  a job is an operand pair: B_k = sum_m w Re(conj(c^l(m)) Z_l(m)) of its triples (l >= jA)
//   y  a job is an output position (m1, m2): y_jO(m1,m2) = sum over the pairs of gamma Z_jO(m1,m2)
//   z  the terms themselves, [tile of atoms][channel][term][atom], for the derivative kernel
// Four warps share a job (its records in four fixed parts of equal work, added in order), so the
// sums do not depend on the number of atoms or on how the jobs fall on the CTAs.
//
// Bound: instruction issue and shared-memory reads in FP32, the FP64 pipe in FP64.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <type_traits>

#include "bispectrum.cuh"

namespace mld {

namespace {

// The values of a lane's atoms: two FP32 packed in a register pair, or one FP64.
struct F2 {
  unsigned long long v;
};
template <typename T>
struct LaneVec;
template <>
struct LaneVec<float> {
  using type = F2;
  static constexpr int atoms = 2, warps = 16;
};
template <>
struct LaneVec<double> {
  using type = double;
  static constexpr int atoms = 1, warps = 8;  // (the FP64 pipe needs fewer warps, the terms more registers)
};
__device__ __forceinline__ F2 pack(float a, float b) {
  F2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d.v) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ void unpack(F2 a, float* v) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v[0]), "=f"(v[1]) : "l"(a.v));
}
__device__ __forceinline__ void unpack(double a, double* v) { v[0] = a; }
__device__ __forceinline__ F2 vmul(F2 a, F2 b) {
  F2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
__device__ __forceinline__ F2 vadd(F2 a, F2 b) {
  F2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
__device__ __forceinline__ F2 vfma(F2 a, F2 b, F2 c) {
  F2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return d;
}
__device__ __forceinline__ F2 vneg(F2 a) { return vmul(a, F2{0xBF800000BF800000ull}); }  // one instruction
__device__ __forceinline__ double vmul(double a, double b) { return a * b; }
__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ double vneg(double a) { return -a; }
__device__ __forceinline__ double vadd(double a, double b) { return a + b; }

// complex value of a lane's atoms (16 bytes)
template <typename V>
struct alignas(16) vcx {
  V x, y;
};

// acc += weight * z.  In FP32 a weight is a double-FP32 pair: rounded to 32 bits, it would shift the energies
// of all atoms alike.  The low part joins the product, whose rounding keeps it on average; next to the sum
// it would be below the last bit.
__device__ __forceinline__ void add_weighted(F2 weight, vcx<F2> z, vcx<F2>& acc) {
  float g[2];
  unpack(weight, g);
  const F2 h = pack(g[0], g[0]), l = pack(g[1], g[1]);
  acc.x = vadd(acc.x, vfma(h, z.x, vmul(l, z.x)));
  acc.y = vadd(acc.y, vfma(h, z.y, vmul(l, z.y)));
}
__device__ __forceinline__ void add_weighted(double weight, vcx<double> z, vcx<double>& acc) {
  acc.x = vfma(weight, z.x, acc.x);
  acc.y = vfma(weight, z.y, acc.y);
}

// the atoms' values one after the other, (re, im) each
__device__ __forceinline__ vcx<F2> interleave(vcx<F2> v) {
  float re[2], im[2];
  unpack(v.x, re);
  unpack(v.y, im);
  return {pack(re[0], im[0]), pack(re[1], im[1])};
}
__device__ __forceinline__ vcx<double> interleave(vcx<double> v) { return v; }

template <typename T>
struct LaneArgs {
  DevTables tb;
  const LaneRec* recs;
  const LaneJob* jobs;
  int njobs;
  const void* cg;       // FP32: every coefficient twice (for the packed instructions)
  const cx<T>* c;       // A x nch x HU
  const int* nbr_off;   // of the first atom
  const void* gamma;    // y: nch * NBLKP weights (FP32: double-FP32 pairs)
  int A, nch;
  T* B;                 // A x nch*K
  cx<T>* y;             // A x nch x HU
  cx<T>* z;             // tiles x nch x NZTP x atoms of a tile
};

enum { kLaneB = 0, kLaneY = 1, kLaneZ = 2 };

// lanes that hold atoms: 32, or 16 where their c does not fit in shared memory; a padded row per entry
// (16-byte values) so that the transposing stores spread over the banks
// The coefficients go to shared memory in FP32 where there is room, else they are read through the cache.
struct LanePlan {
  int stride;
  size_t c, cg, gamma, part, total;
};

__host__ __device__ inline size_t upl(size_t x) { return (x + 15) & ~(size_t)15; }

__host__ __device__ inline LanePlan lane_plan(const DevTables& tb, int eb, int lanes, bool cg_shared) {
  LanePlan s;
  s.stride = lanes + 1;
  size_t o = 0;
  s.c = o;     o = upl(o + (size_t)16 * tb.NU * s.stride);
  s.cg = o;    o = upl(o + (cg_shared ? (size_t)8 * tb.NCGV : 0));
  s.gamma = o; o = upl(o + (size_t)8 * tb.NBLKP);
  s.part = o;  o = upl(o + (size_t)16 * (eb == 4 ? LaneVec<float>::warps : LaneVec<double>::warps) * (tb.J / 2 + 1) * 32);
  s.total = o;
  return s;
}

// C consecutive b of a record, all its a: zs[o] += sum_a c1[a][o] sum_{b<C} c2[b][o] c c, o < NJ
template <int NJ, int C, typename V>
__device__ __forceinline__ void lane_chunk(const vcx<V>* __restrict__ pa, const vcx<V>* __restrict__ pb, int ST, int da,
                                           int db, int na, const V* __restrict__ c1p, int st1,
                                           const V* __restrict__ c2p, int st2, vcx<V>* zs) {
  V c2[C][NJ];
#pragma unroll
  for (int b = 0; b < C; ++b)
#pragma unroll
    for (int o = 0; o < NJ; ++o) c2[b][o] = c2p[b * st2 + o];
  for (int a = 0; a < na; ++a) {
    vcx<V> part[NJ];
#pragma unroll
    for (int b = 0; b < C; ++b) {
      const vcx<V> u = pa[b * ST], v = pb[-b * ST];
      const vcx<V> pr = {vfma(vneg(u.y), v.y, vmul(u.x, v.x)), vfma(u.x, v.y, vmul(u.y, v.x))};
#pragma unroll
      for (int o = 0; o < NJ; ++o) {
        if (b == 0) {
          part[o] = {vmul(c2[b][o], pr.x), vmul(c2[b][o], pr.y)};
        } else {
          part[o].x = vfma(c2[b][o], pr.x, part[o].x);
          part[o].y = vfma(c2[b][o], pr.y, part[o].y);
        }
      }
    }
#pragma unroll
    for (int o = 0; o < NJ; ++o) {
      const V c1 = c1p[o];
      zs[o].x = vfma(c1, part[o].x, zs[o].x);
      zs[o].y = vfma(c1, part[o].y, zs[o].y);
    }
    c1p += st1;
    pa += da;
    pb -= db;
  }
}

// Z of the NJ output layers of a record
template <int NJ, typename V>
__device__ __forceinline__ void lane_terms(uint4 z0, const vcx<V>* __restrict__ cl, int ST, const V* __restrict__ cg,
                                           vcx<V>* zs) {
  constexpr int C = NJ <= 3 || std::is_same<V, double>::value ? 4 : 2;  // C * NJ coefficients in registers
  // x = i1 | i2 << 16, y = cg1 | cg2 << 16, z = na | nb << 8 | s1 << 16 | s2 << 24, w = st1 | st2 << 8 | ..
  const vcx<V>* pa = cl + (z0.x & 0xFFFF) * ST;
  const vcx<V>* pb = cl + (z0.x >> 16) * ST;
  const int na = z0.z & 0xFF, da = ((z0.z >> 16) & 0xFF) * ST, db = (z0.z >> 24) * ST;
  const int st1 = z0.w & 0xFF, st2 = (z0.w >> 8) & 0xFF;
  const V* c1p = cg + (z0.y & 0xFFFF);
  const V* c2p = cg + (z0.y >> 16);
  int nb = (z0.z >> 8) & 0xFF;
#pragma unroll
  for (int o = 0; o < NJ; ++o) zs[o] = {V{}, V{}};
  for (; nb >= C; nb -= C) {
    lane_chunk<NJ, C, V>(pa, pb, ST, da, db, na, c1p, st1, c2p, st2, zs);
    pa += C * ST;
    pb -= C * ST;
    c2p += C * st2;
  }
  if (nb == 1) lane_chunk<NJ, 1, V>(pa, pb, ST, da, db, na, c1p, st1, c2p, st2, zs);
  if constexpr (C > 2) {
    if (nb == 2) lane_chunk<NJ, 2, V>(pa, pb, ST, da, db, na, c1p, st1, c2p, st2, zs);
    else if (nb == 3) lane_chunk<NJ, 3, V>(pa, pb, ST, da, db, na, c1p, st1, c2p, st2, zs);
  }
}

__device__ __forceinline__ int out_of(uint4 z1, int o) {
  const unsigned w = o < 2 ? z1.x : (o < 4 ? z1.y : z1.z);
  return (w >> (16 * (o & 1))) & 0xFFFF;
}

// A record into the job's sums.  y: acc[off + o] += gamma[out_o] Z_o; B: acc[o].x += w Re(conj(c[out_o]) Z_o)
// z: the terms to zo[out_o][atoms of the tile]
template <int NJ, int kMode, typename V>
__device__ __forceinline__ void lane_record(uint4 z0, uint4 z1, const vcx<V>* __restrict__ cl, int ST,
                                            const V* __restrict__ cg, const V* __restrict__ gam, vcx<V>* acc,
                                            vcx<V>* zo, int zst, bool store) {
  vcx<V> zs[NJ];
  lane_terms<NJ, V>(z0, cl, ST, cg, zs);
  if constexpr (kMode == kLaneZ) {
    if (store)
#pragma unroll
      for (int o = 0; o < NJ; ++o) zo[(size_t)out_of(z1, o) * zst] = interleave(zs[o]);
  } else if constexpr (kMode == kLaneY) {
    const int off = z0.w >> 24;
    if (off == 0) {  // pairs that reach the highest layers: most of the work
#pragma unroll
      for (int o = 0; o < NJ; ++o) add_weighted(gam[out_of(z1, o)], zs[o], acc[o]);
    } else {
#pragma unroll
      for (int o = 0; o < NJ; ++o) {
        const V g = gam[out_of(z1, o)];
#pragma unroll
        for (int k = 1; k + o < kMaxZOut; ++k)
          if (k == off) add_weighted(g, zs[o], acc[k + o]);
      }
    }
  } else {
    const int wi = z1.w & 0xFFFF;
#pragma unroll
    for (int o = 0; o < NJ; ++o) {
      const vcx<V> c = cl[out_of(z1, o) * ST];
      const V t = vfma(c.x, zs[o].x, vmul(c.y, zs[o].y));
      acc[o].x = vadd(acc[o].x, wi == 2 ? vadd(t, t) : t);
    }
  }
}

template <typename T, int kMode>
__global__ void __launch_bounds__(LaneVec<T>::warps * 32, 1) k_lanes(LaneArgs<T> args, int lanes, bool cg_shared) {
  using V = typename LaneVec<T>::type;
  constexpr int kPer = LaneVec<T>::atoms, kLaneWarps = LaneVec<T>::warps;
  constexpr int kGroups = kLaneWarps / 4;  // four warps share a job
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const DevTables& tb = args.tb;
  const LanePlan sp = lane_plan(tb, (int)sizeof(T), lanes, cg_shared);
  const int ST = sp.stride, HU = tb.HU, K = tb.K;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int nth = kLaneWarps * 32;
  const int ch = blockIdx.z, a0 = blockIdx.x * lanes * kPer;
  const int na = min(lanes * kPer, args.A - a0);
  vcx<V>* sc = reinterpret_cast<vcx<V>*>(smem_raw + sp.c);
  V* sg = reinterpret_cast<V*>(smem_raw + sp.gamma);
  vcx<V>* part = reinterpret_cast<vcx<V>*>(smem_raw + sp.part);
  // c of the atoms, expanded to full layers; a warp per atom
  for (int a = warp; a < lanes * kPer; a += kLaneWarps) {
    const cx<T>* src = args.c + ((size_t)(a0 + min(a, na - 1)) * args.nch + ch) * HU;
    T* dst = reinterpret_cast<T*>(sc + a / kPer) + a % kPer;  // re, im of atom a: kPer values apart
    for (int f = lane; f < tb.NU; f += 32) {
      const cx<T> v = fetch(src, tb.expand[f]);
      T* d = dst + (size_t)f * ST * 2 * kPer;
      d[0] = v.x;
      d[kPer] = v.y;
    }
  }
  const V* cg = static_cast<const V*>(args.cg);
  if (cg_shared) {
    V* scg = reinterpret_cast<V*>(smem_raw + sp.cg);
    for (int e = tid; e < tb.NCGV; e += nth) scg[e] = cg[e];
    cg = scg;
  }
  if constexpr (kMode == kLaneY) {
    for (int b = tid; b < tb.NBLKP; b += nth) sg[b] = static_cast<const V*>(args.gamma)[ch * tb.NBLKP + b];
  }
  __syncthreads();
  const int al = lane < lanes ? lane : lane - lanes;  // (16 lanes: both halves of the warp hold the same atoms)
  const vcx<V>* cl = sc + al;
  const int group = warp >> 2, q = warp & 3, no = tb.J / 2 + 1;
  vcx<V>* zo = nullptr;
  if constexpr (kMode == kLaneZ)
    zo = reinterpret_cast<vcx<V>*>(args.z) + ((size_t)blockIdx.x * args.nch + ch) * tb.NZTP * lanes + al;
  vcx<V>* mypart = part + (size_t)group * 4 * no * 32;
  for (int job = blockIdx.y * kGroups + group; job < args.njobs; job += gridDim.y * kGroups) {
    const LaneJob& jb = args.jobs[job];
    vcx<V> acc[kMaxZOut];
#pragma unroll
    for (int o = 0; o < kMaxZOut; ++o) acc[o] = {V{}, V{}};
    const int r0 = jb.rec[q], r1 = jb.rec[q + 1];
    constexpr int kAhead = 6;
    const uint4* rp = reinterpret_cast<const uint4*>(args.recs);
    uint4 n0 = make_uint4(0, 0, 0, 0), n1 = n0;
    if (r0 < r1) {
      n0 = __ldg(rp + 2 * (size_t)r0);
      n1 = __ldg(rp + 2 * (size_t)r0 + 1);
    }
    for (int r = r0; r < r1; ++r) {
      const uint4 z0 = n0, z1 = n1;
      // every record is read once per CTA: fetch ahead of the register prefetch
      if (r + kAhead < r1) asm volatile("prefetch.global.L1 [%0];" ::"l"(rp + 2 * (size_t)(r + kAhead)));
      if (r + 1 < r1) {
        n0 = __ldg(rp + 2 * (size_t)(r + 1));
        n1 = __ldg(rp + 2 * (size_t)(r + 1) + 1);
      }
      switch ((z0.w >> 16) & 0xFF) {
        case 1: lane_record<1, kMode, V>(z0, z1, cl, ST, cg, sg, acc, zo, lanes, lane < lanes); break;
        case 2: lane_record<2, kMode, V>(z0, z1, cl, ST, cg, sg, acc, zo, lanes, lane < lanes); break;
        case 3: lane_record<3, kMode, V>(z0, z1, cl, ST, cg, sg, acc, zo, lanes, lane < lanes); break;
        case 4: lane_record<4, kMode, V>(z0, z1, cl, ST, cg, sg, acc, zo, lanes, lane < lanes); break;
        case 5: lane_record<5, kMode, V>(z0, z1, cl, ST, cg, sg, acc, zo, lanes, lane < lanes); break;
        default: lane_record<6, kMode, V>(z0, z1, cl, ST, cg, sg, acc, zo, lanes, lane < lanes); break;
      }
    }
    if constexpr (kMode == kLaneZ) continue;
#pragma unroll
    for (int o = 0; o < kMaxZOut; ++o)
      if (o < no) mypart[(q * no + o) * 32 + lane] = acc[o];
    asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");
    for (int o = q; o < jb.nout; o += 4) {
      vcx<V> v = mypart[o * 32 + lane];
#pragma unroll
      for (int p = 1; p < 4; ++p) {
        const vcx<V> w = mypart[(p * no + o) * 32 + lane];
        v = {vadd(v.x, w.x), vadd(v.y, w.y)};
      }
      T re[kPer], im[kPer];
      unpack(v.x, re);
      unpack(v.y, im);
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const int a = al * kPer + k;
        if (lane < lanes && a < na) {
          const size_t row = (size_t)(a0 + a) * args.nch + ch;
          if constexpr (kMode == kLaneY) args.y[row * HU + jb.out[o]] = {re[k], im[k]};
          else args.B[row * K + jb.out[o]] = args.nbr_off[a0 + a + 1] == args.nbr_off[a0 + a] ? T(0) : re[k];
        }
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
  int first, by_position;
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
  // two places for the queue position in turn: an atom without neighbours passes no other barrier, and
  // thread 0 publishes the next position while other warps may still read this one
  int nxt = first_ticket();
  for (int turn = 0;; turn ^= 1) {
    if (tid == 0) snext[turn] = ticket_position(nxt);
    __syncthreads();
    const int qi = snext[turn];
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
    cx<T>* out = args.c + (size_t)(args.by_position ? qi : atom - args.first) * nch * HU;
    // a thread writes the entries it has summed itself
    for (int e = tid; e < nch * HU; e += nth)
      out[e] = nn > 0 ? chalf[e] : cx<T>{shd[e % HU] ? T(1) : T(0), T(0)};
  }
}

// ---- B from stored terms -----------------------------------------------------------------------
// A CTA per tile of atoms and channel, c of the tile turned around in shared memory, a warp per triple
// with lanes on atoms: B_k = sum w Re(conj(c^l) Z_A).  Bound: reading a third of the terms once.
constexpr int kZBWarps = 16;

template <typename T>
struct ZBArgs {
  DevTables tb;
  const cx<T>* c;
  const cx<T>* z;
  const int* order;
  const int* nbr_off;
  T* B;
  int count, nch, tile;
};

template <typename T>
__global__ void __launch_bounds__(kZBWarps * 32) k_z_descriptors(ZBArgs<T> a) {
  constexpr int kPer = 16 / (2 * (int)sizeof(T));  // atoms of a lane
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const DevTables& tb = a.tb;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, HU = tb.HU, K = tb.K;
  const int CS = a.tile + kPer;  // row of an entry, 16 bytes longer: fewer bank conflicts while turning
  cx<T>* sc = reinterpret_cast<cx<T>*>(smem_raw);
  T* sb = reinterpret_cast<T*>(sc + (size_t)HU * CS);  // [atom][K + 1]
  const int t0 = blockIdx.x / a.nch, ch = blockIdx.x - t0 * a.nch;
  const int na = min(a.tile, a.count - t0 * a.tile), lanes = a.tile / kPer;
  for (int i = warp; i < a.tile; i += kZBWarps) {
    const cx<T>* src = a.c + ((size_t)(t0 * a.tile + min(i, na - 1)) * a.nch + ch) * HU;
    for (int e = lane; e < HU; e += 32) copy_async(sc + (size_t)e * CS + i, src + e);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const cx<T>* z = a.z + ((size_t)t0 * a.nch + ch) * tb.NZTP * a.tile + kPer * lane;
  for (int k = warp; k < K; k += kZBWarps) {
    if (lane >= lanes) break;
    const TripleZ t = tb.trzp[k];
    const int l = t.l, h0 = tb.hoff[l], H = tb.hoff[l + 1] - h0;
    const int centre = (l & 1) ? -1 : H - 1;
    T b[kPer];
#pragma unroll
    for (int p = 0; p < kPer; ++p) b[p] = T(0);
#pragma unroll 8
    for (int e = 0; e < H; ++e) {
      const uint4 zr = *reinterpret_cast<const uint4*>(z + (size_t)(t.za + e) * a.tile);
      const uint4 cr = *reinterpret_cast<const uint4*>(sc + (size_t)(h0 + e) * CS + kPer * lane);
      cx<T> zv[kPer], cv[kPer];
      memcpy(zv, &zr, 16);
      memcpy(cv, &cr, 16);
      const T w = e == centre ? T(1) : T(2);
#pragma unroll
      for (int p = 0; p < kPer; ++p) b[p] = fma(w, fma(cv[p].x, zv[p].x, cv[p].y * zv[p].y), b[p]);
    }
#pragma unroll
    for (int p = 0; p < kPer; ++p) sb[(kPer * lane + p) * (K + 1) + k] = b[p];
  }
  __syncthreads();
  for (int i = warp; i < na; i += kZBWarps) {
    const int pos = t0 * a.tile + i, atom = a.order ? a.order[pos] : pos;
    const bool alone = a.nbr_off[atom + 1] == a.nbr_off[atom];
    for (int k = lane; k < K; k += 32)
      a.B[((size_t)atom * a.nch + ch) * K + k] = alone ? T(0) : sb[i * (K + 1) + k];
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

// lanes per tile and where the coefficients go; the shared memory of a CTA (0: does not fit)
size_t lane_shape(const DevTables& tb, int eb, int* lanes, bool* cg_shared) {
  *lanes = 32;
  *cg_shared = eb == 4;
  auto bytes = [&]() { return lane_plan(tb, eb, *lanes, *cg_shared).total; };
  if (bytes() > (size_t)optin()) *lanes = 16;
  if (bytes() > (size_t)optin()) *cg_shared = false;
  return bytes() <= (size_t)optin() ? bytes() : 0;
}

template <typename T, int kMode>
cudaError_t launch_lanes(LaneArgs<T>& a, cudaStream_t st) {
  if (a.A <= 0 || a.njobs <= 0) return cudaSuccess;
  int lanes;
  bool cg_shared;
  const size_t smem = lane_shape(a.tb, (int)sizeof(T), &lanes, &cg_shared);
  if (!smem) return cudaErrorInvalidConfiguration;
  cudaError_t e = cudaFuncSetAttribute(k_lanes<T, kMode>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int nsm = 0;
  if ((e = sm_count(&nsm)) != cudaSuccess) return e;
  // The jobs of a tile of atoms may be spread over several CTAs (slices), each of which loads the
  // tile's c: worth it where the tiles do not fill the GPU or leave its last round of CTAs nearly
  // empty.  Loading c costs about 1/20 of a tile's jobs in FP32, a tenth of that share in FP64.
  constexpr int kGroups = LaneVec<T>::warps / 4;
  const int per = lanes * LaneVec<T>::atoms, tiles = (a.A + per - 1) / per;
  const int most = std::max(1, (a.njobs + kGroups - 1) / kGroups);
  int slices = 1;
  double best = 0.0;
  for (int s = 1; s <= most; ++s) {
    const long long rounds = ((long long)tiles * a.nch * s + nsm - 1) / nsm;
    const double jobs = (double)((a.njobs + kGroups * s - 1) / (kGroups * s)) * kGroups / a.njobs;
    const double t = (double)rounds * (jobs + (sizeof(T) == 4 ? 0.05 : 0.005));
    if (s == 1 || t < best) {
      best = t;
      slices = s;
    }
  }
  k_lanes<T, kMode><<<dim3(tiles, slices, a.nch), LaneVec<T>::warps * 32, smem, st>>>(a, lanes, cg_shared);
  return cudaGetLastError();
}

}  // namespace

template <typename T>
cudaError_t launch_c_half(const DevTables& tb, const DevBatch& b, const BsoParams& p, int first, int count,
                          const int* order, bool by_position, int* counter, void* c, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  CArgs<T> a{};
  a.tb = tb;
  a.src = {b.types, b.nbr_idx, b.nbr_u, sizeof(T) == 4 ? b.nbr_u32 : nullptr, (T)p.rcut, (T)p.inv_r0,
           (T)p.rin_width, p.ntypes, p.has_rin, {}};
  a.src.rates.set(p.rcut, p.inv_r0);
  a.nbr_off = b.nbr_off;
  for (int e = 0; e < kMaxCh * kMaxTypes; ++e) a.chw[e] = (T)p.chw[e];
  for (int e = 0; e < kMaxTypes * kMaxTypes; ++e) a.rin[e] = (T)p.rin[e];
  a.nch = p.nch;
  a.order = order;
  a.first = first;
  a.by_position = by_position ? 1 : 0;
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
  else a.cg = tb.cgv32x2;
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
  return launch_lanes<T, kLaneB>(a, st);
}

template <typename T>
cudaError_t launch_lane_y(const DevTables& tb, const DevBatch& b, const BsoParams& p, int first, int count,
                          const void* c, const void* gamma, void* y, cudaStream_t st) {
  LaneArgs<T> a = lane_args<T>(tb, b, p, first, count, c);
  a.recs = tb.yrecs;
  a.jobs = tb.yjobs;
  a.njobs = tb.NYJ;
  a.gamma = gamma;
  a.y = static_cast<cx<T>*>(y);
  return launch_lanes<T, kLaneY>(a, st);
}

int lane_tile(const DevTables& tb, int eb) {
  int lanes;
  bool cg_shared;
  if (!lane_shape(tb, eb, &lanes, &cg_shared)) return 0;
  return lanes * (eb == 4 ? LaneVec<float>::atoms : LaneVec<double>::atoms);
}

template <typename T>
cudaError_t launch_lane_z(const DevTables& tb, int nch, int count, const void* c, void* z, cudaStream_t st) {
  LaneArgs<T> a{};
  a.tb = tb;
  if constexpr (sizeof(T) == 8) a.cg = tb.cgv64;
  else a.cg = tb.cgv32x2;
  a.c = static_cast<const cx<T>*>(c);
  a.A = count;
  a.nch = nch;
  a.recs = tb.zrecs;
  a.jobs = tb.yjobs;
  a.njobs = tb.NYJ;
  a.z = static_cast<cx<T>*>(z);
  return launch_lanes<T, kLaneZ>(a, st);
}

template <typename T>
cudaError_t launch_z_descriptors(const DevTables& tb, const DevBatch& b, const BsoParams& p, const int* order, int count,
                                 const void* c, const void* z, T* B, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  ZBArgs<T> a{};
  a.tb = tb;
  a.c = static_cast<const cx<T>*>(c);
  a.z = static_cast<const cx<T>*>(z);
  a.order = order;
  a.nbr_off = b.nbr_off;
  a.B = B;
  a.count = count;
  a.nch = p.nch;
  a.tile = lane_tile(tb, (int)sizeof(T));
  constexpr int kPer = 16 / (2 * (int)sizeof(T));
  const size_t smem = 2 * sizeof(T) * tb.HU * (a.tile + kPer) + sizeof(T) * a.tile * (tb.K + 1);
  if (!a.tile || smem > (size_t)optin()) return cudaErrorInvalidConfiguration;
  cudaError_t e = cudaFuncSetAttribute(k_z_descriptors<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const unsigned grid = (unsigned)((count + a.tile - 1) / a.tile * p.nch);
  k_z_descriptors<T><<<grid, kZBWarps * 32, smem, st>>>(a);
  return cudaGetLastError();
}

template cudaError_t launch_z_descriptors<double>(const DevTables&, const DevBatch&, const BsoParams&, const int*, int,
                                                  const void*, const void*, double*, cudaStream_t);
template cudaError_t launch_z_descriptors<float>(const DevTables&, const DevBatch&, const BsoParams&, const int*, int,
                                                 const void*, const void*, float*, cudaStream_t);
template cudaError_t launch_lane_z<double>(const DevTables&, int, int, const void*, void*, cudaStream_t);
template cudaError_t launch_lane_z<float>(const DevTables&, int, int, const void*, void*, cudaStream_t);
template cudaError_t launch_c_half<double>(const DevTables&, const DevBatch&, const BsoParams&, int, int, const int*,
                                           bool, int*, void*, cudaStream_t);
template cudaError_t launch_c_half<float>(const DevTables&, const DevBatch&, const BsoParams&, int, int, const int*,
                                          bool, int*, void*, cudaStream_t);
template cudaError_t launch_lane_descriptors<double>(const DevTables&, const DevBatch&, const BsoParams&, int, int,
                                                     const void*, double*, cudaStream_t);
template cudaError_t launch_lane_descriptors<float>(const DevTables&, const DevBatch&, const BsoParams&, int, int,
                                                    const void*, float*, cudaStream_t);
template cudaError_t launch_lane_y<double>(const DevTables&, const DevBatch&, const BsoParams&, int, int, const void*,
                                           const void*, void*, cudaStream_t);
template cudaError_t launch_lane_y<float>(const DevTables&, const DevBatch&, const BsoParams&, int, int, const void*,
                                          const void*, void*, cudaStream_t);

}  // namespace mld
