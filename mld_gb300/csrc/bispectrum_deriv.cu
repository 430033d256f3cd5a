// B per atom and w_ch * dB per pair from the Z terms that the atoms-on-lanes kernel has formed
// (bispectrum_lanes.cu; compute_bispectrum_so4.F90:469-717, descriptors.F90:298-302).
//
//   k_y_rows  the Y rows of every atom, each the scaled sum of up to three Z terms; reads the terms
//             with atoms on lanes and writes an atom's rows one after the other
//   k_deriv   dB_k/du_a = w_ch(type_n) sum_b xi[a][b] Re sum Y_k V_b, V_b = f_c U rho(T_b) + kappa_b U
//             (bispectrum.cuh); B = dB/dc . c / 3, since B is a cubic form of c
//
// Every sum has a fixed order that depends neither on the batch, among those that take these kernels
// (deriv_route, api.cu), nor on the launch shape.
#include <cuda_runtime.h>

#include <algorithm>

#include <cstring>

#include "bispectrum.cuh"
#include "ptx.cuh"

namespace mld {

namespace {

// ---- Y rows ---------------------------------------------------------------------------------------
// A CTA takes a tile of atoms, a channel and a share of the quads (entry, four rows of a row tile).  A
// warp forms a quad for all atoms of the tile, a lane per 16 bytes of a term (two atoms in FP32), and
// kQuads of them are turned around in shared memory so that an atom's rows are written 32 bytes per quad.
// Bound: reading the terms and writing the rows once each.
constexpr int kYWarps = 8;
constexpr int kQuads = 16;
constexpr int kScale = kMaxJ + 2;  // row scales n / d, n and d <= kMaxJ + 1

template <typename T>
struct YRowArgs {
  DevTables tb;
  const cx<T>* z;  // [tile][nch][NZTP][atoms of a tile]
  cx<T>* y;        // [position][nch][NYP]
  int count, nch, tile, per;  // per: quads of a CTA
};

template <typename T>
__global__ void __launch_bounds__(kYWarps * 32) k_y_rows(YRowArgs<T> a) {
  constexpr int kPer = 16 / (2 * (int)sizeof(T));  // atoms of a lane
  __shared__ cx<T> buf[32 * kPer][kQuads * kRowTile + 1];
  __shared__ T ssc[kScale * kScale];
  __shared__ int shoff[kMaxJ + 2], sq[kMaxJ + 2], sro[kMaxJ + 2];
  const DevTables& tb = a.tb;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int e = tid; e < kScale * kScale; e += kYWarps * 32) ssc[e] = e % kScale ? (T)(e / kScale) / (T)(e % kScale) : T(0);
  for (int e = tid; e < kMaxJ + 2; e += kYWarps * 32) {
    shoff[e] = tb.hoff[e];
    sq[e] = e <= tb.J ? tb.yoff[e] / kRowTile : tb.NYP / kRowTile;  // first quad of a layer
    sro[e] = e <= tb.J ? tb.rowk_off[e] : 0;
  }
  const int t0 = blockIdx.x / a.nch, ch = blockIdx.x - t0 * a.nch;
  const int nat = min(a.tile, a.count - t0 * a.tile), lanes = a.tile / kPer;
  const cx<T>* z = a.z + ((size_t)t0 * a.nch + ch) * tb.NZTP * a.tile + kPer * lane;
  const int nq = tb.NYP / kRowTile, qbeg = blockIdx.y * a.per, qend = min(nq, qbeg + a.per);
  __syncthreads();
  for (int q0 = qbeg; q0 < qend; q0 += kQuads) {
    const int nhere = min(kQuads, qend - q0);
#pragma unroll
    for (int i = 0; i < kQuads / kYWarps; ++i) {
      const int qi = warp + i * kYWarps, q = q0 + qi;
      if (qi >= nhere || lane >= lanes) continue;
      int j = 0;
      while (q >= sq[j + 1]) ++j;
      const int H = shoff[j + 1] - shoff[j], rt = (q - sq[j]) / H, e = (q - sq[j]) - rt * H;
      const int centre = (j & 1) ? -1 : H - 1;  // the only entry of weight 1
      const T w = e == centre ? T(1) : T(2);
#pragma unroll
      for (int r = 0; r < kRowTile; ++r) {
        // x = z0 | z1 << 16, y = z2 | nterm << 16, z = snum0..2 | sden0 << 24, w = sden1 | sden2 << 8
        const uint4 s = __ldg(reinterpret_cast<const uint4*>(tb.rowsrc2) + sro[j] + rt * kRowTile + r);
        const int nterm = s.y >> 16;
        const int zi[3] = {(int)(s.x & 0xFFFF), (int)(s.x >> 16), (int)(s.y & 0xFFFF)};
        const T sc[3] = {ssc[(s.z & 0xFF) * kScale + (s.z >> 24)], ssc[((s.z >> 8) & 0xFF) * kScale + (s.w & 0xFF)],
                         ssc[((s.z >> 16) & 0xFF) * kScale + ((s.w >> 8) & 0xFF)]};
        cx<T> v[kPer];
#pragma unroll
        for (int p = 0; p < kPer; ++p) v[p] = {T(0), T(0)};
#pragma unroll
        for (int n = 0; n < 3; ++n)
          if (n < nterm) {
            const uint4 raw = *reinterpret_cast<const uint4*>(z + (size_t)(zi[n] + e) * a.tile);
            cx<T> t[kPer];
            memcpy(t, &raw, 16);
#pragma unroll
            for (int p = 0; p < kPer; ++p) v[p] = {fma(sc[n], t[p].x, v[p].x), fma(sc[n], t[p].y, v[p].y)};
          }
#pragma unroll
        for (int p = 0; p < kPer; ++p) buf[kPer * lane + p][qi * kRowTile + r] = {w * v[p].x, w * v[p].y};
      }
    }
    __syncthreads();
    const int nval = nhere * kRowTile;
    for (int i = warp; i < nat; i += kYWarps) {
      cx<T>* o = a.y + ((size_t)(t0 * a.tile + i) * a.nch + ch) * tb.NYP + q0 * kRowTile;
      for (int v = lane; v < nval; v += 32) o[v] = buf[i][v];
    }
    __syncthreads();
  }
}

// ---- derivatives ----------------------------------------------------------------------------------
// A persistent CTA per SM takes atoms by queue position and their neighbours in equal chunks of at most
// `cap`, as many as V of the chunk leaves room for (FP32, j_max 4: 37), with four barriers per chunk:
//   U    column chains, a lane per neighbour
//   V    the three generator products of every half entry, lanes over entries
//   Y.V  register tiles of 4 kPairs rows x kCT columns (column = neighbour, generator; in the first chunk
//        c as one more, for B), jobs of 32 tiles from a counter, long layers first; beside them the
//        geometry of the next chunk or atom
//   out  S_b from the rows' ranks, times xi and w, to global memory; the next Y rows arrive meanwhile
// U and the contractions share their memory.  One wide CTA rather than two narrow ones: the phases are
// latency-bound, and a chunk that holds all neighbours passes them once per atom; the chains fill whole
// warps, and eight rows share one load of V.
//
// 185,000 Fe atoms of 36 neighbours, j_max 4, FP32: B and dB 25 ms with the terms formed per atom, 22 ms
// this way (k_deriv 15, terms 2.8, c 2.5, rows 1.6); 27 ms with two CTAs of eight warps that also sum the
// rows.  Clocks per atom: U 4,000, V 5,600, Y.V 13,000, out 3,500.  Y.V is bound by FP32 issue and
// shared-memory reads together: a register tile step, 32 packed FMAs and 8 loads, takes 116 clocks of a
// scheduler's four warps in isolation, 76 without the loads.  FP64 (16 neighbours to a chunk): the FP64
// pipe, 2 FMA per clock and SM.
constexpr int kDW = 16;
constexpr int kRec = kGeoDeriv;  // xi 0-8, f_c 9, kappa 10-12: read four at a time
static_assert(kGeoXi == 0 && kGeoFc == 9 && kGeoKap == 10 && kRec % 4 == 0, "record layout");

template <typename T>
struct DerivArgs {
  DevTables tb;
  const GenEntry<T>* gen;
  PairSource<T> src;
  const int* nbr_off;
  T chw[kMaxCh * kMaxTypes];
  T rin[kMaxTypes * kMaxTypes];
  int nch, cap;
  const int* order;  // null: atoms first, first + 1, ...
  int first, count;
  int* counter;
  unsigned long long chains;
  const cx<T>* c;    // by queue position
  const cx<T>* y;
  T* Bout;
  T* dBout;
};

struct DerivPlan {
  int dstride;  // row stride of the contractions, odd: no bank conflicts
  size_t gen, hoff, yoff, tiles, rowk, rslot, Y, V, D, rec, wt, next, total;
};

__host__ __device__ inline size_t upd(size_t x) { return (x + 15) & ~(size_t)15; }

__host__ __device__ inline DerivPlan deriv_plan(const DevTables& tb, int nch, int eb, int cap) {
  DerivPlan s;
  const size_t cxb = 2 * (size_t)eb, HS = u_stride(tb.HU);
  s.dstride = (3 * cap + 4) | 1;  // up to three columns past the last are written
  size_t o = 0;
  s.gen = o;   o = upd(o + 4 * (size_t)eb * tb.HU);
  s.hoff = o;  o = upd(o + sizeof(int) * (kMaxJ + 2));
  s.yoff = o;  o = upd(o + sizeof(int) * (2 * kMaxJ + 3));
  s.tiles = o; o = upd(o + sizeof(int16_t) * tb.NTILE);
  s.rowk = o;  o = upd(o + sizeof(uint16_t) * tb.NROWS);
  s.rslot = o; o = upd(o + sizeof(int) * (kRounds - 1) * tb.K);
  s.Y = o;     o = upd(o + cxb * tb.NYP);
  s.V = o;     o = upd(o + cxb * (3 * cap + 1) * HS);
  // (one more row, for the padding rows of the tiles)
  const size_t d = (size_t)eb * s.dstride * (tb.nrank[0] + tb.nrank[1] + tb.nrank[2] + 1), u = cxb * cap * HS;
  s.D = o;     o = upd(o + (d > u ? d : u));
  s.rec = o;   o = upd(o + (size_t)eb * 2 * cap * kRec);
  s.wt = o;    o = upd(o + (size_t)eb * 2 * cap * nch);
  s.next = o;  o = upd(o + 16);
  s.total = o;
  return s;
}

// four values from a 16-byte aligned place
__device__ __forceinline__ void load4(const float* p, float* o) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  o[0] = v.x, o[1] = v.y, o[2] = v.z, o[3] = v.w;
}
__device__ __forceinline__ void load4(const double* p, double* o) {
  const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 2);
  o[0] = a.x, o[1] = a.y, o[2] = b.x, o[3] = b.y;
}

// kPairs: row tiles of four of a register tile
template <typename T, int kPairs, int kCT>
__global__ void __launch_bounds__(kDW * 32, 1) k_deriv(DerivArgs<T> args) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const DevTables& tb = args.tb;
  const int J = tb.J, HU = tb.HU, K = tb.K, nch = args.nch, nchK = nch * K, cap = args.cap;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int nth = kDW * 32;
  const int HS = u_stride(HU);
  const DerivPlan sp = deriv_plan(tb, nch, (int)sizeof(T), cap);
  GenEntry<T>* sgen = reinterpret_cast<GenEntry<T>*>(smem_raw + sp.gen);
  int* shoff = reinterpret_cast<int*>(smem_raw + sp.hoff);
  int* syoff = reinterpret_cast<int*>(smem_raw + sp.yoff);
  int* srko = syoff + (kMaxJ + 1);
  int16_t* stile = reinterpret_cast<int16_t*>(smem_raw + sp.tiles);  // j << 8 | first row tile, 128: two of them
  uint16_t* sslot = reinterpret_cast<uint16_t*>(smem_raw + sp.rowk);  // place of each row in D
  int* srslot = reinterpret_cast<int*>(smem_raw + sp.rslot);        // places of a triple's ranks 1 and 2, -1: none
  cx<T>* Y = reinterpret_cast<cx<T>*>(smem_raw + sp.Y);
  cx<T>* V = reinterpret_cast<cx<T>*>(smem_raw + sp.V);
  cx<T>* U = reinterpret_cast<cx<T>*>(smem_raw + sp.D);
  T* D = reinterpret_cast<T*>(smem_raw + sp.D);
  T* srec = reinterpret_cast<T*>(smem_raw + sp.rec);
  T* swt = reinterpret_cast<T*>(smem_raw + sp.wt);
  int* snext = reinterpret_cast<int*>(smem_raw + sp.next);
  int* sjob = snext + 1;
  int* sntile = snext + 2;
  const int DS = sp.dstride;

  for (int e = tid; e < HU; e += nth) sgen[e] = args.gen[e];
  for (int e = tid; e < kMaxJ + 2; e += nth) {
    shoff[e] = tb.hoff[e];
    srko[e] = tb.rowk_off[e];
  }
  for (int e = tid; e < kMaxJ + 1; e += nth) syoff[e] = tb.yoff[e];
  for (int e = tid; e < tb.NROWS; e += nth) {
    const int code = tb.rowk[e], rank = code >> kRankShift, idx = code & ((1 << kRankShift) - 1);
    const int slot = code < 0 ? K + tb.nrank[1] + tb.nrank[2] : idx + (rank > 0 ? K : 0) + (rank > 1 ? tb.nrank[1] : 0);
    sslot[e] = (uint16_t)(slot * DS);
  }
  for (int e = tid; e < (kRounds - 1) * K; e += nth) {
    const int s = tb.rank_slot[e];
    srslot[e] = s < 0 ? -1 : (s + K + ((e & 1) ? tb.nrank[1] : 0)) * DS;
  }
  if (tid == 0) {
    // the row tiles of a layer follow each other in tb.tiles
    int n = 0;
    for (int t = 0; t < tb.NTILE; ++t) {
      const int code = tb.tiles[t];
      const bool two = kPairs == 2 && t + 1 < tb.NTILE && tb.tiles[t + 1] == code + 1;
      stile[n++] = (int16_t)(code | (two ? 128 : 0));
      t += two;
    }
    *sntile = n;
    snext[0] = ticket_position(first_ticket());
  }
  __syncthreads();
  const int ntile = *sntile;

  // geometry records and channel weights of neighbours [lo, hi) of a chunk that starts at pair p
  auto geometry = [&](int buf, int atom, int p, int lo, int hi) {
    const int n = lo + lane;
    if (n < hi) {
      T g[kGeo];
      int nb, tn;
      pair_geometry<T>(args.src, args.rin, (size_t)(p + n), args.src.types[atom], g, &nb, &tn);
      const int s = buf * cap + n;
      T* r = srec + s * kRec;
#pragma unroll
      for (int i = 0; i < kGeoIdx; ++i) r[i] = g[i];
      for (int ch = 0; ch < nch; ++ch) swt[s * nch + ch] = args.chw[ch * args.src.ntypes + tn];
    }
  };
  auto atom_of = [&](int qi) { return args.order ? args.order[qi] : args.first + qi; };
  // Y rows of channel ch of a queue position, 16 bytes per copy
  auto load_y = [&](int qi, int ch) {
    const unsigned char* g = reinterpret_cast<const unsigned char*>(args.y + ((size_t)qi * nch + ch) * tb.NYP);
    const uint32_t s = ptx::smem_u32(Y);
    const int n = (int)(sizeof(cx<T>) * tb.NYP / 16);
    for (int i = tid; i < n; i += nth)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s + 16u * i), "l"(g + 16 * (size_t)i) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // n / d for n < 2^16 through the multiplier of d (which wraps to 0 for d = 1)
  auto divider = [](int d) { return (unsigned)((0x100000000ull + d - 1) / d); };
  auto quotient = [](int n, unsigned m) { return m ? (int)__umulhi((unsigned)n, m) : n; };
  auto chunks = [&](int nn) { return max(1, (nn + cap - 1) / cap); };

  int qi = snext[0], unit = 0, nxt = 0;
  if (tid == 0) nxt = atomicAdd(args.counter, 1);
  bool primed = false;
  __syncthreads();
  while (qi < args.count) {
    const int atom = atom_of(qi);
    const int p0 = args.nbr_off[atom], nn = args.nbr_off[atom + 1] - p0;
    const int nchunk = chunks(nn), csize = (nn + nchunk - 1) / nchunk;
    if (!primed) {  // the CTA's first atom
      load_y(qi, 0);
      for (int lo = 32 * warp; lo < csize; lo += nth) geometry(unit & 1, atom, p0, lo, csize);
      primed = true;
      __syncthreads();
    }
    int qn = 0;
    for (int k = 0; k < nchunk; ++k, ++unit) {
      const int buf = (unit & 1) * cap, nb = min(csize, nn - k * csize);
      const int pk = p0 + k * csize;
      const bool with_c = k == 0;
      // ---- U -----------------------------------------------------------------------------------
      {
        const int ng = (nb + 31) >> 5, njob = ng * J;
        for (int it = warp; it < njob; it += kDW) {
          const int ci = it / ng, n = (it - ci * ng) * 32 + lane;
          if (n < nb)
            u_chain_of<T>((int)(args.chains >> (4 * ci)) & 15, srec + (buf + n) * kRec + kGeoZx, J, U + (size_t)n * HS);
        }
        for (int n = tid; n < nb; n += nth) U[(size_t)n * HS] = {T(1), T(0)};
        if (tid == 0) {
          *sjob = 0;
          if (k == 0) {
            snext[0] = ticket_position(nxt);  // asked for one atom ahead
            nxt = atomicAdd(args.counter, 1);
          }
        }
      }
      __syncthreads();
      if (k == 0) qn = snext[0];
      // ---- V: items (32 entries, four neighbours) -------------------------------------------------
      if (with_c)
        for (int e = tid; e < HU; e += nth) V[(size_t)(3 * nb) * HS + e] = args.c[(size_t)qi * nch * HU + e];
      {
        const int nec = (HU + 31) >> 5, ngr = (nb + 3) >> 2;
        const unsigned mgr = divider(max(1, ngr));
        for (int it = warp; it < nec * ngr; it += kDW) {
          const int ec = quotient(it, mgr), n0 = (it - ec * ngr) * 4, e = ec * 32 + lane;
          if (e >= HU) continue;
          const GenEntry<T> g = sgen[e];
          const int em = max(e - 1, 0) - e, ep = min(e + 1, HU - 1) - e;
          const bool mirror = g.w == T(1);  // centre of an even layer
          const T* r = srec + (buf + n0) * kRec;
          const cx<T>* u = U + (size_t)n0 * HS + e;
          cx<T>* v = V + (size_t)(3 * n0) * HS + e;
          const int m = nb - n0;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (i >= m) break;
            T w[4], k3 = r[kGeoKap + 2];  // xi[8], f_c, kappa
            load4(r + kGeoXi + 8, w);
            const T fc = w[1], k1 = w[2], k2 = w[3];
            const cx<T> u0 = u[0], um = u[em];
            cx<T> uq = u[ep];
            if (mirror) uq = {-um.x, um.y};
            const T fq = fc * g.q, fm = fc * g.cm, fp = fc * g.cp;
            const cx<T> a = {fm * um.x, fm * um.y};
            const cx<T> s = {fma(fp, uq.x, a.x), fma(fp, uq.y, a.y)}, d = {fma(-fp, uq.x, a.x), fma(-fp, uq.y, a.y)};
            v[0] = {fma(fq, u0.y, k1 * u0.x), fma(-fq, u0.x, k1 * u0.y)};  // T1 U = -i q U
            v[HS] = {fma(k2, u0.x, -s.y), fma(k2, u0.y, s.x)};             // T2 U = i (c- U[q-2] + c+ U[q+2])
            v[2 * HS] = {fma(k3, u0.x, d.x), fma(k3, u0.y, d.y)};          // T3 U = c- U[q-2] - c+ U[q+2]
            r += kRec;
            u += HS;
            v += 3 * HS;
          }
        }
      }
      // the next chunk, of this atom or the next
      int na = atom, np = pk + nb, nnb = 0;
      if (k + 1 < nchunk) {
        nnb = min(csize, nn - (k + 1) * csize);
      } else if (qn < args.count) {
        na = atom_of(qn);
        np = args.nbr_off[na];
        const int m = args.nbr_off[na + 1] - np, c = chunks(m);
        nnb = (m + c - 1) / c;
      }
      for (int ch = 0; ch < nch; ++ch) {
        if (with_c && ch > 0)
          for (int e = tid; e < HU; e += nth) V[(size_t)(3 * nb) * HS + e] = args.c[((size_t)qi * nch + ch) * HU + e];
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        // ---- Y . V ---------------------------------------------------------------------------------
        const int ncols = 3 * nb + (with_c ? 1 : 0), ncolt = (ncols + kCT - 1) / kCT, nitem = ntile * ncolt;
        const unsigned mcol = divider(ncolt);
        const int ngeo = ch == 0 ? (nnb + 31) >> 5 : 0, njob = ngeo + ((nitem + 31) >> 5);
        for (;;) {
          int job = 0;
          if (lane == 0) job = atomicAdd(sjob, 1);
          job = __shfl_sync(0xffffffffu, job, 0);
          if (job >= njob) break;
          if (job < ngeo) {
            geometry((unit + 1) & 1, na, np, 32 * job, nnb);
            continue;
          }
          const int it = (job - ngeo) * 32 + lane;
          if (it >= nitem) continue;
          const int tix = quotient(it, mcol), ct = it - tix * ncolt;
          const int code = stile[tix], j = code >> 8, rt = code & 127;
          const int H = shoff[j + 1] - shoff[j];
          const cx<T>* Yp = Y + syoff[j] + rt * kRowTile * H;
          const int second = code & 128 ? kRowTile * H : 0;
          // columns ct, ct + ncolt, ...: lanes of a warp read consecutive columns of V, whose odd
          // stride spreads them over distinct shared-memory banks
          const cx<T>* Vp[kCT];
#pragma unroll
          for (int c = 0; c < kCT; ++c) Vp[c] = V + (size_t)min(ct + c * ncolt, ncols - 1) * HS + shoff[j];
          cx<T> acc[kPairs * kRowTile][kCT];
#pragma unroll
          for (int r = 0; r < kPairs * kRowTile; ++r)
#pragma unroll
            for (int c = 0; c < kCT; ++c) acc[r][c] = {T(0), T(0)};
#pragma unroll 2
          for (int e = 0; e < H; ++e) {
            cx<T> y[kPairs * kRowTile], v[kCT];
#pragma unroll
            for (int h = 0; h < kPairs; ++h)
#pragma unroll
              for (int r = 0; r < kRowTile; r += 16 / (int)sizeof(cx<T>)) {
                const uint4 raw = *reinterpret_cast<const uint4*>(Yp + h * second + e * kRowTile + r);
                memcpy(&y[h * kRowTile + r], &raw, 16);
              }
#pragma unroll
            for (int c = 0; c < kCT; ++c) v[c] = Vp[c][e];
#pragma unroll
            for (int r = 0; r < kPairs * kRowTile; ++r)
#pragma unroll
              for (int c = 0; c < kCT; ++c) acc[r][c] = fma2(y[r], v[c], acc[r][c]);
          }
          // a register tile without a second row tile has formed the first one twice
#pragma unroll
          for (int h = 0; h < kPairs; ++h) {
            const uint2 sl = *reinterpret_cast<const uint2*>(sslot + srko[j] + (rt + (second ? h : 0)) * kRowTile);
            const int o[kRowTile] = {(int)(sl.x & 0xFFFF), (int)(sl.x >> 16), (int)(sl.y & 0xFFFF), (int)(sl.y >> 16)};
#pragma unroll
            for (int r = 0; r < kRowTile; ++r) {
              T* d = D + o[r] + ct;
#pragma unroll
              for (int c = 0; c < kCT; ++c) d[c * ncolt] = acc[h * kRowTile + r][c].x + acc[h * kRowTile + r][c].y;
            }
          }
        }
        __syncthreads();
        // the next Y rows: of the next channel, of the first one again for the next chunk, of the next atom
        if (ch + 1 < nch) load_y(qi, ch + 1);
        else if (k + 1 < nchunk) { if (nch > 1) load_y(qi, 0); }
        else if (qn < args.count) load_y(qn, 0);
        if (tid == 0) *sjob = 0;
        // ---- out: w_ch dB_a = w_ch sum_b xi[a][b] S_b, S = (rank 0 + rank 1) + rank 2 ----------------
        // (lanes over k, a warp keeps its k)
        const int kc = (K + 31) >> 5, g = warp / kc, i = (warp - g * kc) * 32 + lane;
        if (i < K && warp < kDW / kc * kc) {
          const int s1 = srslot[i * 2], s2 = srslot[i * 2 + 1];
          const T* d0 = D + i * DS;
          const T* d1 = D + max(s1, 0);
          const T* d2 = D + max(s2, 0);
          auto sum = [&](int col) {
            T v = d0[col];
            if (s1 >= 0) v += d1[col];
            if (s2 >= 0) v += d2[col];
            return v;
          };
          T* out = args.dBout + (size_t)(pk + g) * 3 * nchK + ch * K + i;
          const T* r = srec + (buf + g) * kRec + kGeoXi;
          const T* wp = swt + (buf + g) * nch + ch;
          const int step = kDW / kc;
          for (int n = g; n < nb; n += step) {
            T x[8];
            load4(r, x);
            load4(r + 4, x + 4);
            const T x8 = r[8], w = *wp;
            const T S0 = sum(3 * n), S1 = sum(3 * n + 1), S2 = sum(3 * n + 2);
            out[0] = w * fma(x[0], S0, fma(x[1], S1, x[2] * S2));
            out[nchK] = w * fma(x[3], S0, fma(x[4], S1, x[5] * S2));
            out[2 * nchK] = w * fma(x[6], S0, fma(x[7], S1, x8 * S2));
            out += (size_t)3 * nchK * step;
            r += kRec * step;
            wp += nch * step;
          }
          if (with_c && g == step - 1)
            args.Bout[(size_t)atom * nchK + ch * K + i] = nn == 0 ? T(0) : sum(3 * nb) * (T(1) / T(3));
        }
        if (ch + 1 < nch) __syncthreads();
      }
      __syncthreads();
    }
    qi = qn;
  }
}

int optin_d() {
  static int v = 0;
  if (!v) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  }
  return v;
}

// neighbours of a chunk: as many as fit, up to 64 (0: not even four do)
int deriv_cap(const DevTables& tb, int nch, int eb) {
  for (int cap = 64; cap >= 4; --cap)
    if (deriv_plan(tb, nch, eb, cap).total <= (size_t)optin_d()) return cap;
  return 0;
}

}  // namespace

bool deriv_available(const DevTables& tb, int nch, int eb) {
  return deriv_cap(tb, nch, eb) > 0 && lane_tile(tb, eb) > 0;
}

template <typename T>
cudaError_t launch_y_rows(const DevTables& tb, int nch, int count, const void* z, void* y, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  YRowArgs<T> a{};
  a.tb = tb;
  a.z = static_cast<const cx<T>*>(z);
  a.y = static_cast<cx<T>*>(y);
  a.count = count;
  a.nch = nch;
  a.tile = lane_tile(tb, (int)sizeof(T));
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  // few tiles: their quads are shared out over enough CTAs for four on every SM
  const int nq = tb.NYP / kRowTile, rounds = (nq + kQuads - 1) / kQuads;
  const int cols = ((count + a.tile - 1) / a.tile) * nch;
  const int slices = std::min(rounds, std::max(1, (4 * nsm + cols - 1) / cols));
  a.per = (rounds + slices - 1) / slices * kQuads;
  k_y_rows<T><<<dim3((unsigned)cols, (unsigned)((nq + a.per - 1) / a.per)), kYWarps * 32, 0, st>>>(a);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_deriv(const DevTables& tb, const DevBatch& b, const BsoParams& p, int first, int count,
                         const int* order, int* counter, const void* c, const void* y, T* Bout, T* dBout,
                         const Bso4Launch& shape, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  if (!counter || !Bout || !dBout || !tb.gen32) return cudaErrorInvalidValue;
  DerivArgs<T> a{};
  a.tb = tb;
  if constexpr (sizeof(T) == 8) a.gen = tb.gen64;
  else a.gen = tb.gen32;
  a.src = {b.types, b.nbr_idx, b.nbr_u, sizeof(T) == 4 ? b.nbr_u32 : nullptr, (T)p.rcut, (T)p.inv_r0,
           (T)p.rin_width, p.ntypes, p.has_rin, {}};
  a.src.rates.set(p.rcut, p.inv_r0);
  a.nbr_off = b.nbr_off;
  for (int e = 0; e < kMaxCh * kMaxTypes; ++e) a.chw[e] = (T)p.chw[e];
  for (int e = 0; e < kMaxTypes * kMaxTypes; ++e) a.rin[e] = (T)p.rin[e];
  a.nch = p.nch;
  a.cap = deriv_cap(tb, p.nch, (int)sizeof(T));
  if (!a.cap) return cudaErrorInvalidConfiguration;
  a.order = order;
  a.first = first;
  a.count = count;
  a.counter = counter;
  a.chains = chain_order(tb.J);
  a.c = static_cast<const cx<T>*>(c);
  a.y = static_cast<const cx<T>*>(y);
  a.Bout = Bout;
  a.dBout = dBout;
  const size_t smem = deriv_plan(tb, p.nch, (int)sizeof(T), a.cap).total;
  constexpr int kPairs = sizeof(T) == 4 ? 2 : 1;  // FP64: registers
  auto kern = shape.col_tile == 2 ? k_deriv<T, kPairs, 2> : k_deriv<T, kPairs, 4>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  e = cudaMemsetAsync(counter, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  kern<<<(unsigned)std::min(count, nsm), kDW * 32, smem, st>>>(a);
  return cudaGetLastError();
}

#define MLD_INST(T)                                                                                                  \
  template cudaError_t launch_y_rows<T>(const DevTables&, int, int, const void*, void*, cudaStream_t);               \
  template cudaError_t launch_deriv<T>(const DevTables&, const DevBatch&, const BsoParams&, int, int, const int*,    \
                                       int*, const void*, const void*, T*, T*, const Bso4Launch&, cudaStream_t);
MLD_INST(double)
MLD_INST(float)
#undef MLD_INST

}  // namespace mld
