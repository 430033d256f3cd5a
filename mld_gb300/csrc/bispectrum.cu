// Bispectrum-SO(4) descriptors and their derivatives in one kernel, one centre atom at a time: the route
// of batches of up to an atom per SM (larger ones: bispectrum_lanes.cu and bispectrum_deriv.cu).
//
// Per atom i with neighbours n (u_n = x_n - x_i, r_n < r_cut):
//   phase 1  c^j(p,q) = delta_pq + sum_n w_ch(type_n) f_c(r_n) U^j_pq(u_n)           (compute_bispectrum_so4.F90:288-439)
//   phase 2  Z blocks ZA/ZB/ZC by Clebsch-Gordan contraction of c, merged per (k, layer) into Y,
//            B_k = Re sum conj(c^l) ZA_k                                               (:1014-1143, :469-560)
//   phase 3  per chunk of neighbours: U, its three generator derivatives V_b = f_c U rho(T_b) + kappa_b U
//            (bispectrum.cuh; angular_functions.f90:41-273), the contraction of Y with V_b (register-tiled
//            per layer) and dB_k/du_a = w_ch(type_n) sum_b xi[a][b] (Y . V_b)   (:469-717, descriptors.F90:298-302)
// Outputs: B per atom and w_ch * dB per pair (the design rows are gathered from them by rows.cu).
// Evaluation with fitted weights has a kernel of its own (bispectrum_eval.cu).
// Only half of every layer is computed (X(-p,-q) = (-1)^((p-q)/2) conj X(p,q) for U, c, Z, V);
// full-layer sums fold into weighted sums over the half.  U runs on column chains with a lane per
// neighbour; phase 2 follows a host-balanced schedule of rounds of 32 terms of one inner extent
// per warp, each distinct Z computation evaluated once.
//
// Every floating-point sum has a fixed order: c is summed over the neighbours in order, Z terms
// land in a term buffer from which the Y rows and B are summed, and the dB contraction writes
// each layer row into the buffer of its rank (a triple's distinct layers in ascending order),
// where every triple has at most one row, so dB = (rank 0 + rank 1) + rank 2.  Results are
// therefore bitwise reproducible and do not depend on which CTA takes which atom.  (Batches of more
// atoms take other kernels, whose sums run in another order.)
//
// CTAs are persistent: they stage the small tables in shared memory once, then pull atoms from a
// queue (ordered by descending neighbour count, or in index order, whichever the launch-shape
// autotuner found faster).  Each atom's geometry records are kept from phase 1 for phase 3.
// T = double (plain FP64 method) or float (mixed method: FP32 descriptors).
#include <cuda_runtime.h>

#include <algorithm>

#include "bispectrum.cuh"

namespace mld {

template <typename T>
struct KernelArgs {
  DevTables tb;
  const GenEntry<T>* gen;
  const T* cg;
  PairSource<T> src;
  const int* nbr_off;
  // channel weights and inner cutoffs per type pair in T, converted once at launch
  T chw[kMaxCh * kMaxTypes];
  T rin[kMaxTypes * kMaxTypes];
  int nch;
  // work queue: atoms in the order given (nullptr: 0..A-1), taken through a global counter
  const int* order;
  int* counter;
  unsigned long long chains;
  // Y (the contracted Z blocks, nch * NYP complex per atom) in global memory, one slice per CTA,
  // when it does not fit in shared memory next to the rest (FP64 with several channels) or would
  // cost a resident CTA per SM (FP32 with several channels)
  void* yglobal;
  int g1;       // selects the neighbours per phase-1 pass, phase1_slots(g1)
  int geo_cap;  // neighbours whose geometry records are kept for phase 3 (the rest recompute)
  // outputs: B (A x nch*K) and w_ch * dB (P x 3 x nch*K)
  T* Bout;
  T* dBout;
};

constexpr int kNB = 16;  // neighbours per phase-3 chunk
constexpr int kScale = kMaxJ + 2;  // row scales n / d, n and d <= kMaxJ + 1

// Shared-memory carve-up, in order (every region 16-byte aligned):
//   gen[HU]  hoff[kMaxJ+2]  rowk[NROWS]  tiles[NTILE]  rank_slot[2K]  cfull[nch*NU]
//   Y[nch*NYP] (shared Y)
//   V region (phase 1: U store of a pass, zp and xp, f_c w_ch; phase 2: term buffer; both: c on half layers
//   behind them; phase 3: V_b of a chunk)
//   W region (phase 2: CG coefficients; phase 3: U of the chunk, then the chunk's contractions by
//   rank: rank 0 [cols][K], rank 1 [cols][nrank1], rank 2 [cols][nrank2])
//   Bk[nch*K]  nwt[nch*NB]  next atom
//   expand[NU]  half_diag[HU] (tables staged once per CTA)  sc[kScale^2] (row scales)
//   crec[NB*kGeoDeriv] (records of a chunk's neighbours beyond geo_cap)
//   geo[geo_cap*kGeo] (geometry records of the atom's first geo_cap neighbours)
struct SmemPlan {
  size_t gen, hoff, rowk, tiles, rslot, cfull, Y, V, p1z, p1w, p1c, W, Bk, nwt, next, sc, exp, hd, crec, geo, total;
};

__host__ __device__ inline size_t al16(size_t x) { return (x + 15) & ~(size_t)15; }

// neighbours per phase-1 pass: 64, 40, 32 or 16 for g1 = 4, 6, 8 or 16
__host__ __device__ constexpr int phase1_slots(int g1) { return kNW * (32 / g1); }

__host__ __device__ inline SmemPlan smem_plan(const DevTables& tb, int nch, int eb, bool y_in_smem, int g1 = 16,
                                              int geo_cap = 0) {
  const size_t ns = phase1_slots(g1);
  const size_t cxb = 2 * (size_t)eb;
  const size_t HS = u_stride(tb.HU);
  const size_t w1 = ns * HS;                          // phase 1: U of a pass, its zp, xp and f_c w_ch
  const size_t e1 = w1 + 2 * ns + (ns * nch + 1) / 2;
  const size_t c1 = e1 > (size_t)tb.NZT ? e1 : tb.NZT;  // c behind the U store and the term buffer
  const size_t v1 = c1 + (size_t)nch * tb.HU;
  const size_t v3 = (size_t)kNB * 3 * HS;             // phase 3
  const size_t vblock = v1 > v3 ? v1 : v3;
  const size_t wu = (size_t)kNB * HS * cxb;
  const size_t wdb = (size_t)3 * kNB * (tb.nrank[0] + tb.nrank[1] + tb.nrank[2]) * eb;
  const size_t wcg = al16((size_t)eb * tb.NCG);
  const size_t wblock = wu > wdb ? (wu > wcg ? wu : wcg) : (wdb > wcg ? wdb : wcg);
  SmemPlan s;
  size_t o = 0;
  s.gen = o;   o = al16(o + 4 * (size_t)eb * tb.HU);
  s.hoff = o;  o = al16(o + sizeof(int) * (kMaxJ + 2));
  s.rowk = o;  o = al16(o + sizeof(int16_t) * tb.NROWS);
  s.tiles = o; o = al16(o + sizeof(int) * tb.NTILE);
  s.rslot = o; o = al16(o + sizeof(int16_t) * (kRounds - 1) * tb.K);
  s.cfull = o; o = al16(o + cxb * nch * tb.NU);
  s.Y = o;     o = al16(o + (y_in_smem ? cxb * nch * tb.NYP : 0));
  s.V = o;
  s.p1z = o + cxb * w1;
  s.p1w = s.p1z + cxb * 2 * ns;
  s.p1c = o + cxb * c1;
  o = al16(o + cxb * vblock);
  s.W = o;     o = al16(o + wblock);
  s.Bk = o;    o = al16(o + (size_t)eb * nch * tb.K);
  s.nwt = o;   o = al16(o + (size_t)eb * nch * kNB);
  s.next = o;  o = al16(o + sizeof(int) * (4 + 3 * kMaxJ + 4 + kRounds));
  s.sc = o;    o = al16(o + (size_t)eb * kScale * kScale);
  s.exp = o;   o = al16(o + sizeof(int16_t) * tb.NU);
  s.hd = o;    o = al16(o + tb.HU);
  s.crec = o;  o = al16(o + (size_t)eb * kGeoDeriv * kNB);
  s.geo = o;   o = al16(o + (size_t)eb * kGeo * geo_cap);
  s.total = o;
  return s;
}

constexpr int kCT = 4;  // columns (neighbour, generator) per register tile of the dB contraction

// kYShared: Y lives in shared memory (one channel); otherwise in the per-CTA global slice
// args.yglobal (several channels), a separate instantiation so that the shared-memory
// variant keeps shared-memory addressing.
template <typename T, bool kYShared>
__global__ void __launch_bounds__(kNW * 32, sizeof(T) == 4 ? 2 : 1) k_bso4(KernelArgs<T> args, int A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const DevTables& tb = args.tb;
  const int J = tb.J, NU = tb.NU, HU = tb.HU, K = tb.K, NYP = tb.NYP;
  const int nch = args.nch;
  const int nchK = nch * K;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int nth = kNW * 32;
  const int HS = u_stride(HU);
  const SmemPlan sp = smem_plan(tb, nch, (int)sizeof(T), kYShared, args.g1, args.geo_cap);

  GenEntry<T>* sgen = reinterpret_cast<GenEntry<T>*>(smem_raw + sp.gen);
  int* shoff = reinterpret_cast<int*>(smem_raw + sp.hoff);
  int16_t* srowk = reinterpret_cast<int16_t*>(smem_raw + sp.rowk);
  int* stile = reinterpret_cast<int*>(smem_raw + sp.tiles);
  int16_t* srslot = reinterpret_cast<int16_t*>(smem_raw + sp.rslot);
  cx<T>* cfull = reinterpret_cast<cx<T>*>(smem_raw + sp.cfull);
  cx<T>* Y = kYShared ? reinterpret_cast<cx<T>*>(smem_raw + sp.Y)
                      : reinterpret_cast<cx<T>*>(args.yglobal) + (size_t)blockIdx.x * nch * NYP;
  cx<T>* V = reinterpret_cast<cx<T>*>(smem_raw + sp.V);
  T* p1z = reinterpret_cast<T*>(smem_raw + sp.p1z);
  T* p1w = reinterpret_cast<T*>(smem_raw + sp.p1w);
  cx<T>* p1c = reinterpret_cast<cx<T>*>(smem_raw + sp.p1c);
  unsigned char* W = smem_raw + sp.W;
  T* scg = reinterpret_cast<T*>(W);  // phase 2 only (restaged per atom)
  T* Bk = reinterpret_cast<T*>(smem_raw + sp.Bk);
  T* nwt = reinterpret_cast<T*>(smem_raw + sp.nwt);
  int* snext = reinterpret_cast<int*>(smem_raw + sp.next);
  T* crec = reinterpret_cast<T*>(smem_raw + sp.crec);
  T* sgeo = reinterpret_cast<T*>(smem_raw + sp.geo);
  T* ssc = reinterpret_cast<T*>(smem_raw + sp.sc);  // ssc[kScale n + d] = n / d, the row scales

  // tables, once per CTA
  for (int e = tid; e < HU; e += nth) sgen[e] = args.gen[e];
  for (int e = tid; e < kMaxJ + 2; e += nth) shoff[e] = tb.hoff[e];
  int* sMp = snext + 4;
  int* syoff = sMp + (kMaxJ + 1);
  int* srko = syoff + (kMaxJ + 1);
  int* snr = srko + (kMaxJ + 2);
  for (int e = tid; e < kMaxJ + 1; e += nth) { sMp[e] = tb.Mp[e]; syoff[e] = tb.yoff[e]; }
  for (int e = tid; e < kMaxJ + 2; e += nth) srko[e] = tb.rowk_off[e];
  for (int e = tid; e < kRounds; e += nth) snr[e] = tb.nrank[e];
  for (int e = tid; e < tb.NROWS; e += nth) srowk[e] = tb.rowk[e];
  for (int e = tid; e < tb.NTILE; e += nth) stile[e] = tb.tiles[e];
  for (int e = tid; e < (kRounds - 1) * K; e += nth) srslot[e] = tb.rank_slot[e];
  for (int e = tid; e < kScale * kScale; e += nth) ssc[e] = e % kScale ? (T)(e / kScale) / (T)(e % kScale) : T(0);
  int16_t* sexp = reinterpret_cast<int16_t*>(smem_raw + sp.exp);
  int8_t* shd = reinterpret_cast<int8_t*>(smem_raw + sp.hd);
  for (int e = tid; e < NU; e += nth) sexp[e] = tb.expand[e];
  for (int e = tid; e < HU; e += nth) shd[e] = tb.half_diag[e];
  const int zr0 = tb.zitem_off[warp], zr1 = tb.zitem_off[warp + 1];  // this warp's Z rounds

  const int slots = phase1_slots(args.g1);

  // thread 0 takes the next queue position while the current atom runs; it publishes it at the
  // top of the loop, after at least one barrier that follows every thread's read of the last one
  int nxt = first_ticket();
  for (;;) {
    if (tid == 0) snext[0] = ticket_position(nxt);
    __syncthreads();  // also orders the table staging and the previous atom's last reads
    const int qi = snext[0];
    if (qi >= A) break;
    if (tid == 0) nxt = atomicAdd(args.counter, 1);
    const int atom = args.order ? args.order[qi] : qi;
    const int ti = args.src.types[atom];
    const int p0 = args.nbr_off[atom];
    const int nn = args.nbr_off[atom + 1] - p0;

    // ---------------- phase 1: c^j on half layers ---------------------------------------------
    // (the CG coefficients of phase 2 are copied into W meanwhile by 16-byte asynchronous
    // copies, the device table being padded to whole chunks; W held the previous atom's dB)
    {
      const int n16 = (tb.NCG * (int)sizeof(T) + 15) >> 4;
      const char* src = reinterpret_cast<const char*>(args.cg);
      const unsigned dst = (unsigned)__cvta_generic_to_shared(scg);
      for (int e = tid; e < n16; e += nth)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + 16u * e), "l"(src + 16 * (size_t)e) : "memory");
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    for (int base = 0; base < nn; base += slots) {
      const int count = min(slots, nn - base);
      for (int n = tid; n < count; n += nth) {
        T g[kGeo];
        int nb, tn;
        pair_geometry<T>(args.src, args.rin, (size_t)(p0 + base + n), ti, g, &nb, &tn);
        for (int ch = 0; ch < nch; ++ch) p1w[n * nch + ch] = g[kGeoFc] * args.chw[ch * args.src.ntypes + tn];
#pragma unroll
        for (int k = 0; k < 4; ++k) p1z[n * 4 + k] = g[kGeoZx + k];
        V[(size_t)n * HS] = {T(1), T(0)};
        if (base + n < args.geo_cap) {
          T* r = sgeo + (size_t)(base + n) * kGeo;
#pragma unroll
          for (int k = 0; k < kGeoIdx; ++k) r[k] = g[k];
          put_pair<T>(r, nb, tn);
        }
      }
      __syncthreads();
      u_store<T>(V, HS, count, J, args.chains, warp, lane, [&](int n) { return p1z + n * 4; });
      __syncthreads();
      c_sum<T>(p1c, V, HS, p1w, shd, count, nch, HU, base == 0, base + slots >= nn, tid);
      __syncthreads();
    }
    if (nn == 0) {  // no neighbours: c is the identity
      for (int e = tid; e < nch * HU; e += nth) p1c[e] = {shd[e % HU] ? T(1) : T(0), T(0)};
      __syncthreads();
    }
    // expansion to full layers
    for (int e = tid; e < nch * NU; e += nth) {
      const int ch = e / NU, f = e - ch * NU;
      cfull[e] = fetch(p1c + ch * HU, sexp[f]);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();

    // ---------------- phase 2: Z terms -> term buffer -> Y rows and B -----------------------
    cx<T>* tbuf = V;
    for (int ch = 0; ch < nch; ++ch) {
      z_rounds<T>(tb.zitems, zr0, zr1, cfull + ch * NU, scg, tbuf, lane);
      __syncthreads();
      // Y rows by tiles of four, [tile][entry][row]: a warp per tile, lanes over (entry, row), so a
      // lane keeps its row's sources and a warp stores 32 consecutive values
      cx<T>* Yc = Y + (size_t)ch * NYP;
      for (int t = warp; t < tb.NTILE; t += kNW) {
        const int tile = stile[t], j = tile >> 8, rt = tile & 255;
        const int H = shoff[j + 1] - shoff[j];
        const uint4 rs = __ldg(reinterpret_cast<const uint4*>(tb.rowsrc) + srko[j] + rt * kRowTile + (lane & 3));
        // x = z0 | z1 << 16, y = z2 | nterm << 16, z = snum0..2 | sden0 << 24, w = sden1 | sden2 << 8
        const int nterm = rs.y >> 16;
        const int z0 = rs.x & 0xFFFF, z1 = rs.x >> 16, z2 = rs.y & 0xFFFF;
        const T s0 = nterm > 0 ? ssc[(rs.z & 0xFF) * kScale + (rs.z >> 24)] : T(0);
        const T s1 = nterm > 1 ? ssc[((rs.z >> 8) & 0xFF) * kScale + (rs.w & 0xFF)] : T(0);
        const T s2 = nterm > 2 ? ssc[((rs.z >> 16) & 0xFF) * kScale + ((rs.w >> 8) & 0xFF)] : T(0);
        cx<T>* o = Yc + syoff[j] + rt * kRowTile * H;
        const int centre = (j & 1) ? -1 : H - 1;  // the only entry of weight 1
        for (int i = lane; i < kRowTile * H; i += 32) {
          const int e = i >> 2;
          cx<T> v = {T(0), T(0)};
          if (nterm > 0) {
            const cx<T> z = tbuf[z0 + e];
            v = {s0 * z.x, s0 * z.y};
          }
          if (nterm > 1) {
            const cx<T> z = tbuf[z1 + e];
            v = {fma(s1, z.x, v.x), fma(s1, z.y, v.y)};
          }
          if (nterm > 2) {
            const cx<T> z = tbuf[z2 + e];
            v = {fma(s2, z.x, v.x), fma(s2, z.y, v.y)};
          }
          const T w = e == centre ? T(1) : T(2);
          o[i] = {w * v.x, w * v.y};
        }
      }
      b_sums<T>(tb.trz, K, shoff, p1c + ch * HU, tbuf, warp, lane, Bk + ch * K);
      __syncthreads();
    }
    for (int e = tid; e < nchK; e += nth) args.Bout[(size_t)atom * nchK + e] = nn == 0 ? T(0) : Bk[e];
    if (nn == 0) continue;

    // ---------------- phase 3: dB per neighbour chunk (kNB neighbours, the last one the rest) -
    cx<T>* Us = reinterpret_cast<cx<T>*>(W);
    T* dBs = reinterpret_cast<T*>(W);  // 3*kNB*K [col][k], after the chunk's V
    for (int base = 0; base < nn; base += kNB) {
      const int nb_here = min(kNB, nn - base);
      // record of the chunk's neighbour n: phase 1's, else computed again
      auto rec = [&](int n) {
        return base + n < args.geo_cap ? sgeo + (size_t)(base + n) * kGeo : crec + (size_t)n * kGeoDeriv;
      };
      if (tid < nb_here) {
        T* r = rec(tid);
        if (base + tid >= args.geo_cap) {
          T g[kGeo];
          int nb, tn;
          pair_geometry<T>(args.src, args.rin, (size_t)(p0 + base + tid), ti, g, &nb, &tn);
#pragma unroll
          for (int k = 0; k < kGeoIdx; ++k) r[k] = g[k];
          put_pair<T>(r, nb, tn);
        }
        for (int ch = 0; ch < nch; ++ch) nwt[ch * kNB + tid] = args.chw[ch * args.src.ntypes + pair_type<T>(r)];
        Us[(size_t)tid * HS] = {T(1), T(0)};
      }
      if (base + nb_here > args.geo_cap) __syncthreads();
      u_store<T>(Us, HS, nb_here, J, args.chains, warp, lane, [&](int n) { return rec(n) + kGeoZx; });
      __syncthreads();
      // V_b = f_c U rho(T_b) + kappa_b U: a warp per neighbour, lanes over the half entries
      for (int n = warp; n < nb_here; n += kNW) {
        const T* r = rec(n);
        const T fc = r[kGeoFc], k1 = r[kGeoKap], k2 = r[kGeoKap + 1], k3 = r[kGeoKap + 2];
        const cx<T>* u = Us + (size_t)n * HS;
        cx<T>* v = V + (size_t)(3 * n) * HS;
        for (int e = lane; e < HU; e += 32) {
          const GenEntry<T> g = sgen[e];
          const cx<T> u0 = u[e], um = u[max(e - 1, 0)];
          cx<T> uq = u[min(e + 1, HU - 1)];
          if (g.w == T(1)) uq = {-um.x, um.y};  // centre of an even layer
          const T fq = fc * g.q, fm = fc * g.cm, fp = fc * g.cp;
          const cx<T> a = {fm * um.x, fm * um.y};
          const cx<T> s = {fma(fp, uq.x, a.x), fma(fp, uq.y, a.y)}, d = {fma(-fp, uq.x, a.x), fma(-fp, uq.y, a.y)};
          v[e] = {fma(fq, u0.y, k1 * u0.x), fma(-fq, u0.x, k1 * u0.y)};  // T1 U = -i q U
          v[HS + e] = {fma(k2, u0.x, -s.y), fma(k2, u0.y, s.x)};         // T2 U = i (c- U[q-2] + c+ U[q+2])
          v[2 * HS + e] = {fma(k3, u0.x, d.x), fma(k3, u0.y, d.y)};      // T3 U = c- U[q-2] - c+ U[q+2]
        }
      }
      __syncthreads();  // V of the chunk complete; the U of the chunk becomes dBs
      const int ncols = 3 * nb_here;
      const int ncolt = (ncols + kCT - 1) / kCT;
      for (int ch = 0; ch < nch; ++ch) {
        const cx<T>* Yc = Y + (size_t)ch * NYP;
        // register-tiled contraction, item = (row tile of layer j, column tile), heaviest
        // layers first; each row's result goes to the buffer of its rank, where it is the
        // triple's only row, so no two items write the same element
        T* dB1 = dBs + (size_t)3 * kNB * K;
        T* dB2 = dB1 + (size_t)3 * kNB * tb.nrank[1];
        const int nitem = tb.NTILE * ncolt;
        for (int k = 0; k * nth < nitem; ++k) {
          // rounds alternate direction, so the threads with the heaviest items of one round take
          // the lightest of the next (items are ordered heaviest layers first)
          const int it = (k & 1) ? (k + 1) * nth - 1 - tid : k * nth + tid;
          if (it >= nitem) continue;
          const int tix = it / ncolt;
          const int tile = stile[tix];
          const int ct = it - tix * ncolt;
          const int j = tile >> 8, rt = tile & 255;
          const int H = shoff[j + 1] - shoff[j];
          const cx<T>* Yp = Yc + syoff[j] + rt * kRowTile * H;
          // columns ct, ct + ncolt, ...: lanes of a warp read consecutive columns of V, whose
          // odd stride spreads them over distinct shared-memory banks
          const cx<T>* Vp[kCT];
#pragma unroll
          for (int c = 0; c < kCT; ++c) {
            const int col = min(ct + c * ncolt, ncols - 1);
            Vp[c] = V + (size_t)col * HS + shoff[j];  // col = n*3 + b
          }
          cx<T> acc[kRowTile][kCT];
#pragma unroll
          for (int r = 0; r < kRowTile; ++r)
#pragma unroll
            for (int c = 0; c < kCT; ++c) acc[r][c] = {T(0), T(0)};
#pragma unroll 4
          for (int e = 0; e < H; ++e) {
            cx<T> y[kRowTile], v[kCT];
#pragma unroll
            for (int r = 0; r < kRowTile; ++r) y[r] = Yp[e * kRowTile + r];
#pragma unroll
            for (int c = 0; c < kCT; ++c) v[c] = Vp[c][e];
#pragma unroll
            for (int r = 0; r < kRowTile; ++r)
#pragma unroll
              for (int c = 0; c < kCT; ++c) acc[r][c] = fma2(y[r], v[c], acc[r][c]);
          }
#pragma unroll
          for (int r = 0; r < kRowTile; ++r) {
            const int code = srowk[srko[j] + rt * kRowTile + r];
            if (code < 0) continue;
            const int rank = code >> kRankShift, idx = code & ((1 << kRankShift) - 1);
            T* base = rank == 0 ? dBs : (rank == 1 ? dB1 : dB2);
            const int ld = snr[rank];
#pragma unroll
            for (int c = 0; c < kCT; ++c) {
              const int col = ct + c * ncolt;
              if (col < ncols) base[(size_t)col * ld + idx] = acc[r][c].x + acc[r][c].y;
            }
          }
        }
        __syncthreads();
        // S_b = (rank 0 + rank 1) + rank 2 and w_ch dB_a = w_ch sum_b xi[a][b] S_b of every pair of the
        // chunk: lanes take the components k, warps the neighbours, so a lane looks up its k's rank
        // slots once and a warp's stores are contiguous
        const int nr1 = tb.nrank[1], nr2 = tb.nrank[2];
        T* out = args.dBout + (size_t)(p0 + base) * 3 * nchK + ch * K;
        for (int k = lane; k < K; k += 32) {
          const int s1 = srslot[k * (kRounds - 1)], s2 = srslot[k * (kRounds - 1) + 1];
          for (int n = warp; n < nb_here; n += kNW) {
            T S[3];
#pragma unroll
            for (int b = 0; b < 3; ++b) {
              const int col = 3 * n + b;
              T v = dBs[col * K + k];
              if (s1 >= 0) v += dB1[col * nr1 + s1];
              if (s2 >= 0) v += dB2[col * nr2 + s2];
              S[b] = v;
            }
            const T* xi = rec(n) + kGeoXi;
            const T w = nwt[ch * kNB + n];
#pragma unroll
            for (int a = 0; a < 3; ++a)
              out[(size_t)(3 * n + a) * nchK + k] = w * fma(xi[3 * a], S[0], fma(xi[3 * a + 1], S[1], xi[3 * a + 2] * S[2]));
          }
        }
        __syncthreads();
      }
    }
  }
}

static int max_optin_smem() {
  static int v = 0;
  if (!v) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  }
  return v;
}

// Y in shared memory unless it does not fit or costs a resident CTA per SM (several channels)
static bool y_shared(const DevTables& tb, int nch, int eb) {
  const size_t ss = smem_plan(tb, nch, eb, true).total, sg = smem_plan(tb, nch, eb, false).total;
  const size_t per_sm = 228 * 1024;
  return ss <= (size_t)max_optin_smem() && per_sm / (ss + 1024) >= per_sm / (sg + 1024);
}

bool bso4_available(const DevTables& tb, int nch, int eb) {
  for (int g1 : {4, 6, 8, 16})
    for (bool y : {true, false})
      if (smem_plan(tb, nch, eb, y, g1).total <= (size_t)max_optin_smem()) return true;
  return false;
}

size_t bso4_y_scratch_bytes(const DevTables& tb, int nch, int eb, int max_ctas, bool only_if_required) {
  const bool fits = smem_plan(tb, nch, eb, true).total <= (size_t)max_optin_smem();
  if (fits && (only_if_required || y_shared(tb, nch, eb))) return 0;
  return (size_t)max_ctas * nch * tb.NYP * 2 * eb;
}

template <typename T>
cudaError_t launch_bso4(const DevTables& tb, const DevBatch& b, const BsoParams& p, T* Bout, T* dBout,
                        const int* order, int* counter, cudaStream_t st, void* yscratch, size_t yscratch_bytes,
                        const Bso4Launch* shape) {
  const Bso4Launch sh = shape ? *shape : Bso4Launch{};
  if (b.A == 0) return cudaSuccess;
  if (!counter) return cudaErrorInvalidValue;
  KernelArgs<T> a{};
  a.tb = tb;
  if constexpr (sizeof(T) == 8) {
    a.gen = tb.gen64;
    a.cg = reinterpret_cast<const T*>(tb.cg64);
  } else {
    a.gen = tb.gen32;
    a.cg = reinterpret_cast<const T*>(tb.cg32);
  }
  if (!Bout || !dBout || !a.gen) return cudaErrorInvalidValue;
  a.src = {b.types, b.nbr_idx, b.nbr_u, sizeof(T) == 4 ? b.nbr_u32 : nullptr, (T)p.rcut, (T)p.inv_r0,
           (T)p.rin_width, p.ntypes, p.has_rin, {}};
  a.src.rates.set(p.rcut, p.inv_r0);
  a.nbr_off = b.nbr_off;
  for (int e = 0; e < kMaxCh * kMaxTypes; ++e) a.chw[e] = (T)p.chw[e];
  for (int e = 0; e < kMaxTypes * kMaxTypes; ++e) a.rin[e] = (T)p.rin[e];
  a.nch = p.nch;
  a.chains = chain_order(tb.J);
  a.order = sh.sorted_queue ? order : nullptr;
  a.counter = counter;
  a.Bout = Bout;
  a.dBout = dBout;
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const size_t per_sm = 228 * 1024;
  // Y in shared memory when it fits, unless it costs a resident CTA per SM and the scratch holds
  // a global slice for every CTA of the shape without it (several channels in FP32)
  bool y_in_smem = smem_plan(tb, p.nch, sizeof(T), true).total <= (size_t)max_optin_smem();
  if (y_in_smem && yscratch && !y_shared(tb, p.nch, (int)sizeof(T))) {
    const size_t sg = smem_plan(tb, p.nch, sizeof(T), false).total;
    const long long ctas = std::min<long long>((long long)b.A, (long long)nsm * (long long)(per_sm / (sg + 1024)));
    if ((long long)(yscratch_bytes / ((size_t)p.nch * tb.NYP * 2 * sizeof(T))) >= ctas) y_in_smem = false;
  }
  // the most neighbours per phase-1 pass whose U store fits without costing a resident CTA per SM,
  // and leaves room for the geometry records of kGeoWant neighbours where any choice does
  constexpr int kGeoWant = 64;
  const size_t s16 = smem_plan(tb, p.nch, sizeof(T), y_in_smem, 16).total;
  auto keeps = [&](int g1, int cap, size_t than) {
    const size_t sg = smem_plan(tb, p.nch, sizeof(T), y_in_smem, g1, cap).total;
    return sg <= (size_t)max_optin_smem() && per_sm / (sg + 1024) >= per_sm / (than + 1024);
  };
  a.g1 = 16;
  for (int cap : {0, kGeoWant})
    for (int g1 : {4, 6, 8})
      if (keeps(g1, cap, s16)) {
        a.g1 = g1;
        break;
      }
  size_t smem = smem_plan(tb, p.nch, sizeof(T), y_in_smem, a.g1).total;
  if (smem > (size_t)max_optin_smem()) return cudaErrorInvalidConfiguration;
  // geometry records for the first geo_cap neighbours of an atom (at most 128), as many as keep
  // the resident CTAs per SM as they are.  The count depends on the configuration only, so an atom's
  // results are the same in every batch that takes this kernel (larger ones round differently).
  a.geo_cap = 0;
  for (int cap = 128; cap > 0; cap -= 8) {
    const size_t sc = smem_plan(tb, p.nch, sizeof(T), y_in_smem, a.g1, cap).total;
    if (sc <= (size_t)max_optin_smem() && per_sm / (sc + 1024) >= per_sm / (smem + 1024)) {
      a.geo_cap = cap;
      smem = sc;
      break;
    }
  }
  a.yglobal = nullptr;
  auto kern = y_in_smem ? k_bso4<T, true> : k_bso4<T, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int occ = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kNW * 32, smem);
  if (e != cudaSuccess) return e;
  if (occ < 1) return cudaErrorInvalidConfiguration;
  long long grid = std::min<long long>((long long)b.A, (long long)nsm * occ);
  if (!y_in_smem) {
    // one Y slice per persistent CTA
    const size_t per_cta = (size_t)p.nch * tb.NYP * 2 * sizeof(T);
    const long long fit = yscratch ? (long long)(yscratch_bytes / per_cta) : 0;
    grid = std::min(grid, fit);
    if (grid < 1) return cudaErrorInvalidValue;  // Y scratch required and not given
    a.yglobal = yscratch;
  }
  e = cudaMemsetAsync(counter, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  kern<<<(unsigned)grid, kNW * 32, smem, st>>>(a, b.A);
  return cudaGetLastError();
}

template cudaError_t launch_bso4<double>(const DevTables&, const DevBatch&, const BsoParams&, double*, double*,
                                         const int*, int*, cudaStream_t, void*, size_t, const Bso4Launch*);
template cudaError_t launch_bso4<float>(const DevTables&, const DevBatch&, const BsoParams&, float*, float*,
                                        const int*, int*, cudaStream_t, void*, size_t, const Bso4Launch*);

}  // namespace mld
