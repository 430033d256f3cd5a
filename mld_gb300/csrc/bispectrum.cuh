// Device code shared by the descriptor kernel (bispectrum.cu) and the evaluation kernel
// (bispectrum_eval.cu): neighbour geometry, the U recursion by column chains, the
// Clebsch-Gordan (Z) terms, packed FP32 arithmetic.
#pragma once
#include <cuda_runtime.h>

#include "mld_internal.h"

namespace mld {

template <typename T>
struct alignas(2 * sizeof(T)) cx {
  T x, y;
};

template <typename T>
__device__ __forceinline__ cx<T> cmul(cx<T> a, cx<T> b) {
  return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}
template <typename T>
__device__ __forceinline__ cx<T> cfma(cx<T> a, cx<T> b, cx<T> c) {  // a*b + c
  return {fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y))};
}
// decode an encoded half-layer reference: (idx << 2) | (conj << 1) | neg
template <typename T>
__device__ __forceinline__ cx<T> fetch(const cx<T>* base, int code) {
  const cx<T> v = base[code >> 2];
  const T sy = (code & 2) ? T(-1) : T(1);
  const T sn = (code & 1) ? T(-1) : T(1);
  return {sn * v.x, sn * sy * v.y};
}

// acc + (a.x b.x, a.y b.y): one packed FP32 instruction, two FP64 ones
__device__ __forceinline__ cx<float> fma2(cx<float> a, cx<float> b, cx<float> c) {
  cx<float> d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)),
        "l"(reinterpret_cast<unsigned long long&>(c)));
  return d;
}
__device__ __forceinline__ cx<double> fma2(cx<double> a, cx<double> b, cx<double> c) {
  return {fma(a.x, b.x, c.x), fma(a.y, b.y, c.y)};
}

constexpr int kNW = 8;  // warps per CTA (== kZWarps)
static_assert(kNW == kZWarps, "phase-2 schedule is built for the CTA's warps");

// ---- work queue --------------------------------------------------------------------------------
// A persistent CTA starts with the position of its block index; the counter hands out those behind the
// grid.  Taken from the counter too, the first positions went to the CTAs that started first, which ask
// for their second atom at once: of as many CTAs as atoms some took two and others none (derivatives of
// 16 / 54 / 152 Fe atoms in FP64 at j_max 4: 860 / 900 / 925 us in most calls, 460 / 500 / 530 now).  A
// ticket becomes a position where it is used: an addition behind the counter's read would wait for it.
__device__ __forceinline__ int first_ticket() { return (int)blockIdx.x - (int)gridDim.x; }
__device__ __forceinline__ int ticket_position(int ticket) { return ticket + (int)gridDim.x; }

// ---- neighbour geometry --------------------------------------------------------------------
// Record of a neighbour (kGeo values, a multiple of 4 so that records stay 16-byte aligned); the first
// kGeoDeriv are what the derivatives need:
//   kGeoXi   xi[3][3]: d/du_a of U is U sum_b xi[a][b] rho(T_b) (the generators below)
//   kGeoFc   f_c, kGeoKap kappa[3] with f_c' e_a = sum_b xi[a][b] kappa[b]
//   kGeoZx   zp and xp, the matrix of U^1; kGeoIdx the neighbour's index and type (two ints)
//   kGeoDfr  f_c' e_a; kGeoU displacement u and 1/r
constexpr int kGeo = 28, kGeoDeriv = 20;
constexpr int kGeoXi = 0, kGeoFc = 9, kGeoKap = 10, kGeoZx = 13, kGeoIdx = 17, kGeoDfr = 20, kGeoU = 23;

// angular_functions.f90:66-107 (the geometric set-up of spherical_4d) and the cutoff of
// compute_bispectrum_so4.F90:337-377 (type-2 cosine outer cut times (1 - inner type-3 cut)).
//
// U^j is a representation of the SU(2) matrix G = cos th + sin th N(e), e = u / r, with
// G = [[zp, -i xp], [-i xm, zm]].  Its derivative is U^j rho(G^-1 dG), a combination of the three
// generators T1 = diag(i, -i), T2 = [[0, i], [i, 0]], T3 = [[0, 1], [-1, 0]]:
//   G^-1 d_a G = th' e_a N + sin th cos th / r (N(a) - e_a N) - sin^2 th / r N(e x a)
// and N(v) has the components (v_z, -v_x, v_y) on (T1, T2, T3).  kappa expresses the derivative of
// the cutoff (along e) on the same three: only the first term of xi has a component along e.
//
// The constants that every pair shares (th', 1 / r_cut and the slope of the cutoff) carry their rounding
// as a second value in FP32: rounded once, they shift all forces of a structure alike, and the sum of a
// small stress keeps that shift (54 Fe atoms: median error of the stress 8.1e-7 -> 1.4e-7).
template <typename T>
struct PairRates {
  T rate, rate_lo;    // th' (th = r th')
  T icut, icut_lo;    // 1 / r_cut
  T slope, slope_lo;  // pi / (2 r_cut)
  void set(double rcut, double inv_r0) {
    auto split = [](double v, T* h, T* l) {
      *h = (T)v;
      *l = (T)(v - (double)*h);
    };
    split(inv_r0 / rcut, &rate, &rate_lo);
    split(1.0 / rcut, &icut, &icut_lo);
    split(0.5 * 3.14159265358979323846 / rcut, &slope, &slope_lo);
  }
};
template <typename T>
__device__ __forceinline__ void nbr_geometry(T x0, T x1, T x2, T rinv, T rcut, const PairRates<T>& k, T rin, T rin_w, T* g) {
  const T PI = (T)3.14159265358979323846;
  const T rr = sqrt(x0 * x0 + x1 * x1 + x2 * x2);
  const T rate = k.rate;
  T th;
  if constexpr (sizeof(T) == 8) th = rr * rate;
  else th = fmaf(rr, rate, rr * k.rate_lo);
  T s, c;
  if constexpr (sizeof(T) == 8) sincos(th, &s, &c);
  else sincosf(th, &s, &c);
  const T e[3] = {x0 * rinv, x1 * rinv, x2 * rinv};
  g[kGeoZx + 0] = c;
  g[kGeoZx + 1] = e[2] * s;
  g[kGeoZx + 2] = e[0] * s;
  g[kGeoZx + 3] = e[1] * s;
  const T tr = s * c * rinv, cr = s * s * rinv;
  T radial = rate - tr;
  if constexpr (sizeof(T) == 4) radial += k.rate_lo;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    T v[3];
#pragma unroll
    for (int b = 0; b < 3; ++b) v[b] = radial * e[a] * e[b];
    v[a] += tr;
    // - cr (e x a)
    v[(a + 1) % 3] = fma(-cr, e[(a + 2) % 3], v[(a + 1) % 3]);
    v[(a + 2) % 3] = fma(cr, e[(a + 1) % 3], v[(a + 2) % 3]);
    g[kGeoXi + 3 * a + 0] = v[2];
    g[kGeoXi + 3 * a + 1] = -v[0];
    g[kGeoXi + 3 * a + 2] = v[1];
  }
  // cutoff (neighbours.F90:598-645, types 2 and 3)
  T fo = 0, dfo = 0;
  if (rr <= rcut) {
    T sp, cp;
    if constexpr (sizeof(T) == 8) {
      const T xx = rr / rcut;
      sincos(PI * xx, &sp, &cp);
      dfo = -T(0.5) * PI * sp / rcut;
    } else {
      sincospif(fmaf(rr, k.icut, rr * k.icut_lo), &sp, &cp);
      dfo = -fmaf(sp, k.slope, sp * k.slope_lo);
    }
    fo = T(0.5) * (cp + T(1));
  }
  T fi = 0, dfi = 0;
  if (rin > T(0)) {
    const T rc2 = rin + rin_w, w = rin_w;
    if (rr <= rc2) {
      if (rr < rc2 - w) {
        fi = 1;
        dfi = 0;
      } else {
        const T xx = PI * (rr - rc2 + w) / w;
        fi = T(0.5) * (cos(xx) + T(1));
        dfi = -T(0.5) * sin(xx) * PI / w;
      }
    }
  }
  g[kGeoFc] = (T(1) - fi) * fo;
  const T dfc = -dfi * fo + (T(1) - fi) * dfo;
#pragma unroll
  for (int a = 0; a < 3; ++a) g[kGeoDfr + a] = dfc * e[a];
  T dk = dfc / rate;
  if constexpr (sizeof(T) == 4) dk = fmaf(-dk, k.rate_lo / rate, dk);
  g[kGeoKap + 0] = dk * e[2];
  g[kGeoKap + 1] = -dk * e[0];
  g[kGeoKap + 2] = dk * e[1];
}

// one complex value from global to shared memory, asynchronously (cp.async)
__device__ __forceinline__ void copy_async(cx<float>* dst, const cx<float>* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async(cx<double>* dst, const cx<double>* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// ---- U by column chains --------------------------------------------------------------------
// Column q of layer j follows from column q - 1 of layer j - 1 alone (angular_functions.f90:108-272),
// so the layers fall into independent chains: chain d starts with column 0 (q = -j) of layer d, a
// binomial in zp and -i xm, and continues with column 1 of layer d + 1, and so on.  Columns q <= 0
// of every layer hold a half of it (the rest follows by X(-p,-q) = (-1)^((p-q)/2) conj X(p,q)), so
// chain d ends at layer min(J, 2 d).  With U(p,q) = sqrt(ip! (j-ip)! / (iq! (j-iq)!)) W(p,q) the
// recursion has no coefficients: W_j(ip,iq) = zm W_{j-1}(ip-1,iq-1) - i xp W_{j-1}(ip,iq-1).
// A lane runs one chain of one neighbour with the column in registers and every index and
// factor known at compile time: about 12 instructions per entry, against 35 of a table-driven
// recursion through shared memory.
constexpr double c_fact(int n) { return n <= 1 ? 1.0 : n * c_fact(n - 1); }
constexpr double c_sqrt(double x) {
  double r = x > 1.0 ? x : 1.0;
  for (int i = 0; i < 200; ++i) r = 0.5 * (r + x / r);
  return r;
}
constexpr int c_hoff(int j) {
  int o = 0;
  for (int i = 0; i < j; ++i) o += ((i + 1) * (i + 1) + 1) / 2;
  return o;
}
template <int J, int IP, int IQ>
struct ChainNorm {
  static constexpr double value = c_sqrt(c_fact(IP) * c_fact(J - IP) / (c_fact(IQ) * c_fact(J - IQ)));
};

// store entries ip = IP..LAST of column iq of layer j, each at its place in the stored half
template <int J, int IQ, int IP, int LAST, typename T>
__device__ __forceinline__ void chain_store(const cx<T>* col, cx<T>* __restrict__ u) {
  if constexpr (IP <= LAST) {
    constexpr int e = IP * (J + 1) + IQ, H = ((J + 1) * (J + 1) + 1) / 2;
    constexpr double n = ChainNorm<J, IP, IQ>::value;
    if constexpr (e < H) {
      u[c_hoff(J) + e] = {(T)n * col[IP].x, (T)n * col[IP].y};
    } else {  // conj of the entry at (-p, -q)
      constexpr double sn = (IP - IQ) % 2 ? -n : n;
      u[c_hoff(J) + (J + 1) * (J + 1) - 1 - e] = {(T)sn * col[IP].x, (T)(-sn) * col[IP].y};
    }
    chain_store<J, IQ, IP + 1, LAST>(col, u);
  }
}

template <int D, int S, typename T>
__device__ __forceinline__ void chain_step(cx<T>* col, cx<T> zm, cx<T> t, int J, cx<T>* __restrict__ u) {
  constexpr int j = D + S;
  chain_store<j, S, 0, (S == D ? D : j)>(col, u);
  if constexpr (S < D && j < kMaxJ) {
    if (j + 1 > J) return;
    col[j + 1] = cmul(zm, col[j]);
#pragma unroll
    for (int ip = j; ip > 0; --ip) col[ip] = cfma(zm, col[ip - 1], cmul(t, col[ip]));
    col[0] = cmul(t, col[0]);
    chain_step<D, S + 1>(col, zm, t, J, u);
  }
}

// column 0 of layer D: col[k] = C(D, k) zp^(D-k) y^k, from col[k] = zp^(D-k) and w = y^k
template <int D, int K, typename T>
__device__ __forceinline__ void chain_spine(cx<T>* col, cx<T> w, cx<T> y) {
  if constexpr (K < D) {
    constexpr double b = c_fact(D) / (c_fact(K) * c_fact(D - K));
    const cx<T> v = cmul(col[K], w);
    col[K] = {(T)b * v.x, (T)b * v.y};
    chain_spine<D, K + 1>(col, cmul(w, y), y);
  } else {
    col[D] = w;
  }
}

template <int D, typename T>
__device__ __forceinline__ void u_chain(cx<T> z, cx<T> x, int J, cx<T>* __restrict__ u) {
  constexpr int N = 2 * D < kMaxJ ? 2 * D : kMaxJ;
  cx<T> col[N + 1];
  const cx<T> y = {-x.y, -x.x};  // -i xm
  cx<T> w = z;
#pragma unroll
  for (int k = D - 1; k > 0; --k) {
    col[k] = w;  // zp^(D-k)
    w = cmul(w, z);
  }
  col[0] = w;
  chain_spine<D, 1>(col, y, y);
  chain_step<D, 0>(col, {z.x, -z.y}, {x.y, -x.x}, J, u);
}

// Chains in descending order of their length (entries), for every J: 4 bits each.
inline unsigned long long chain_order(int J) {
  int d[kMaxJ], n[kMaxJ];
  for (int i = 0; i < J; ++i) {
    d[i] = i + 1;
    n[i] = 2 * (i + 1);  // the powers of column 0
    for (int s = 0; s <= d[i] && d[i] + s <= J; ++s) n[i] += d[i] + s + 1;
  }
  unsigned long long o = 0;
  for (int i = 0; i < J; ++i) {
    int b = i;
    for (int k = i + 1; k < J; ++k)
      if (n[k] > n[b]) b = k;
    const int td = d[i], tn = n[i];
    d[i] = d[b];
    n[i] = n[b];
    d[b] = td;
    n[b] = tn;
    o |= (unsigned long long)d[i] << (4 * i);
  }
  return o;
}

// Row stride of the U store: a neighbour's half layers, odd so that lanes writing the same entry
// of consecutive neighbours use distinct banks.
__host__ __device__ constexpr int u_stride(int HU) { return HU | 1; }

// Chain d of a neighbour with zp, xp at zx into its row u of the store.
template <typename T>
__device__ __forceinline__ void u_chain_of(int d, const T* zx, int J, cx<T>* u) {
  const cx<T> z = {zx[0], zx[1]}, x = {zx[2], zx[3]};
  switch (d) {
    case 1: u_chain<1>(z, x, J, u); break;
    case 2: u_chain<2>(z, x, J, u); break;
    case 3: u_chain<3>(z, x, J, u); break;
    case 4: u_chain<4>(z, x, J, u); break;
    case 5: u_chain<5>(z, x, J, u); break;
    case 6: u_chain<6>(z, x, J, u); break;
    case 7: u_chain<7>(z, x, J, u); break;
    case 8: u_chain<8>(z, x, J, u); break;
    case 9: u_chain<9>(z, x, J, u); break;
    default: u_chain<10>(z, x, J, u); break;
  }
}

// U (all half layers but the first, which is 1) of neighbours 0..count-1 into Us[n][u_stride]; zx(n)
// points to the neighbour's zp and xp.  Work items (chain, 32 neighbours) go to the warps longest
// first, every second round in reverse.  No synchronisation inside.
template <typename T, class Zx>
__device__ __forceinline__ void u_store(cx<T>* Us, int HS, int count, int J, unsigned long long order, int warp,
                                        int lane, Zx zx) {
  const int nb = (count + 31) >> 5, nitem = J * nb;
  for (int r = 0; r * kNW < nitem; ++r) {
    const int it = (r & 1) ? (r + 1) * kNW - 1 - warp : r * kNW + warp;
    if (it >= nitem) continue;
    const int ci = it / nb, n = (it - ci * nb) * 32 + lane;
    if (n < count) u_chain_of<T>((int)(order >> (4 * ci)) & 15, zx(n), J, Us + (size_t)n * HS);
    __syncwarp();
  }
}

// ---- Z terms -------------------------------------------------------------------------------
// One Z term: sum_a c1_a sum_b c2_b c[i1 + a s1 + b] c[i2 - a s2 - b] with NB = nb known at compile
// time, so that the b loop unrolls and the term's NB coefficients c2 stay in registers.
template <int NB, typename T>
__device__ __forceinline__ cx<T> zterm(const cx<T>* __restrict__ cc, const T* __restrict__ cgs, uint4 zi) {
  // the item's 16 bytes: x = i1 | i2 << 16, y = cg1 | cg2 << 16, z = na | nb << 8 | s1 << 16 | s2 << 24
  const int cg1 = zi.y & 0xFFFF, cg2 = zi.y >> 16, na = zi.z & 0xFF, s1 = (zi.z >> 16) & 0xFF, s2 = zi.z >> 24;
  T c2[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) c2[b] = cgs[cg2 + b];
  cx<T> zs = {T(0), T(0)};
  int i1a = zi.x & 0xFFFF, i2a = zi.x >> 16;
#pragma unroll (NB <= 2 ? 4 : (NB <= 5 ? 2 : 1))
  for (int a = 0; a < na; ++a) {
    const T c1 = cgs[cg1 + a];
    cx<T> part = {T(0), T(0)};
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const cx<T> pr = cmul(cc[i1a + b], cc[i2a - b]);
      part.x = fma(c2[b], pr.x, part.x);
      part.y = fma(c2[b], pr.y, part.y);
    }
    zs.x = fma(c1, part.x, zs.x);
    zs.y = fma(c1, part.y, zs.y);
    i1a += s1;
    i2a -= s2;
  }
  return zs;
}

// The rounds [r0, r1) of a warp: lane l of a round computes one Z term into the term buffer; the 32
// terms of a round share their inner extent nb and have outer extents na in descending order, so
// the warp diverges only at the end of the a loop.  Entries are prefetched two rounds ahead.
template <typename T>
__device__ __forceinline__ void z_rounds(const ZItem* __restrict__ items, int r0, int r1, const cx<T>* __restrict__ cc,
                                         const T* __restrict__ scg, cx<T>* __restrict__ tbuf, int lane) {
  const uint4* zit = reinterpret_cast<const uint4*>(items);
  uint4 n1 = make_uint4(0u, 0u, 0u, 0u), n2 = n1;
  if (r0 < r1) n1 = __ldg(zit + (size_t)r0 * 32 + lane);
  if (r0 + 1 < r1) n2 = __ldg(zit + (size_t)(r0 + 1) * 32 + lane);
  for (int r = r0; r < r1; ++r) {
    const uint4 zi = n1;
    n1 = n2;
    if (r + 2 < r1) n2 = __ldg(zit + (size_t)(r + 2) * 32 + lane);
    cx<T> zs;
    switch ((zi.z >> 8) & 0xFF) {  // nb, uniform over the round
      case 1: zs = zterm<1, T>(cc, scg, zi); break;
      case 2: zs = zterm<2, T>(cc, scg, zi); break;
      case 3: zs = zterm<3, T>(cc, scg, zi); break;
      case 4: zs = zterm<4, T>(cc, scg, zi); break;
      case 5: zs = zterm<5, T>(cc, scg, zi); break;
      case 6: zs = zterm<6, T>(cc, scg, zi); break;
      case 7: zs = zterm<7, T>(cc, scg, zi); break;
      case 8: zs = zterm<8, T>(cc, scg, zi); break;
      case 9: zs = zterm<9, T>(cc, scg, zi); break;
      case 10: zs = zterm<10, T>(cc, scg, zi); break;
      default: zs = zterm<11, T>(cc, scg, zi); break;
    }
    if ((zi.w & 0xFFFF) != kNoTerm) tbuf[zi.w & 0xFFFF] = zs;
  }
}

// B_k of the triples by warps (lane = half entry of the ZA block): sum_e w_e Re(conj(c^l[e]) Z[e]), a
// fixed tree over the lanes.
template <typename T>
__device__ __forceinline__ void b_sums(const TripleZ* __restrict__ trz, int K, const int* __restrict__ shoff,
                                       const cx<T>* __restrict__ chalf, const cx<T>* __restrict__ tbuf, int warp,
                                       int lane, T* __restrict__ Bk) {
  for (int k = warp; k < K; k += kNW) {
    const TripleZ t = trz[k];
    const int l = t.l, H = shoff[l + 1] - shoff[l];
    const cx<T>* c = chalf + shoff[l];
    const cx<T>* z = tbuf + t.za;
    T b = T(0);
    for (int e = lane; e < H; e += 32) {
      const T w = (e == H - 1 && !(l & 1)) ? T(1) : T(2);  // the centre of an even layer counts once
      b = fma(w, c[e].x * z[e].x + c[e].y * z[e].y, b);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
    if (lane == 0) Bk[k] = b;
  }
}

// Displacement of pair q and 1/r in T.
template <typename T>
__device__ __forceinline__ void pair_u_rinv(const double* __restrict__ nbr_u, const float4* __restrict__ u32, size_t q,
                                            T* x, T* rinv) {
  if constexpr (sizeof(T) == 4) {
    if (u32) {
      const float4 v = u32[q];
      x[0] = v.x;
      x[1] = v.y;
      x[2] = v.z;
      *rinv = v.w;
      return;
    }
  }
  const double* u3 = nbr_u + 3 * q;
  x[0] = (T)u3[0];
  x[1] = (T)u3[1];
  x[2] = (T)u3[2];
  *rinv = (T)(1.0 / sqrt(u3[0] * u3[0] + u3[1] * u3[1] + u3[2] * u3[2]));
}

// Batch inputs of a pair's geometry record.
template <typename T>
struct PairSource {
  const int* types;
  const int* nbr_idx;
  const double* nbr_u;
  const float4* u32;  // (u, 1/r) in FP32 for T = float (null: converted from nbr_u)
  T rcut, inv_r0, rin_w;
  int ntypes, has_rin;
  PairRates<T> rates;
};

// Geometry record of pair q with a centre of type ti, but for the neighbour's index and type, which
// come back in *nb and *tn (put_pair stores them).
template <typename T>
__device__ __forceinline__ void pair_geometry(const PairSource<T>& s, const T* rin, size_t q, int ti, T* g, int* nb,
                                              int* tn) {
  *nb = s.nbr_idx[q];
  *tn = s.types[*nb];
  T x[3], rinv;
  pair_u_rinv<T>(s.nbr_u, s.u32, q, x, &rinv);
  nbr_geometry<T>(x[0], x[1], x[2], rinv, s.rcut, s.rates, s.has_rin ? rin[ti * s.ntypes + *tn] : T(0), s.rin_w, g);
  g[kGeoU + 0] = x[0];
  g[kGeoU + 1] = x[1];
  g[kGeoU + 2] = x[2];
  g[kGeoU + 3] = rinv;
}

template <typename T>
__device__ __forceinline__ void put_pair(T* g, int nb, int tn) {
  reinterpret_cast<int*>(g + kGeoIdx)[0] = nb;
  reinterpret_cast<int*>(g + kGeoIdx + 1)[0] = tn;
}
template <typename T>
__device__ __forceinline__ int pair_type(const T* g) {
  return reinterpret_cast<const int*>(g + kGeoIdx + 1)[0];
}

// c on half layers from the U store of neighbours 0..count-1 of a pass: chalf += sum over them in
// order of fcw * U, the diagonal's +1 after the last pass.
template <typename T>
__device__ __forceinline__ void c_sum(cx<T>* __restrict__ chalf, const cx<T>* __restrict__ Us, int HS,
                                      const T* __restrict__ fcw, const int8_t* __restrict__ half_diag, int count,
                                      int nch, int HU, bool first, bool last, int tid) {
  for (int e = tid; e < nch * HU; e += kNW * 32) {
    const int ch = e / HU, h = e - ch * HU;
    cx<T> acc = first ? cx<T>{T(0), T(0)} : chalf[e];
#pragma unroll 8
    for (int n = 0; n < count; ++n) {
      const T w = fcw[n * nch + ch];
      const cx<T> u = Us[(size_t)n * HS + h];
      acc.x = fma(w, u.x, acc.x);
      acc.y = fma(w, u.y, acc.y);
    }
    if (last && half_diag[h]) acc.x += T(1);
    chalf[e] = acc;
  }
}

}  // namespace mld
