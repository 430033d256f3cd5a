// Evaluation with fitted weights: per-pair forces, per-atom stress and energy, without dB.
//
// With beta = dE/dB_i the force of pair (i, n) is f_c' and U' contracted with the effective
// y = dE/dc, a sum of the distinct Z blocks with weights gamma (eval.cu), so the K contractions of dB
// collapse into one per direction.  The directions are the three generators of SU(2)
// (bispectrum.cuh): dU = U sum_b xi_b rho(T_b), and the generators move to the y side, once per atom:
//   S_b = Re sum y conj(U rho(T_b)) = sum_e y_b[e] . U[e],   y_0 = y, y_1 = i q y,
//   y_2 = -i (c- y[q-2] + c+ y[q+2]),  y_3 = c+ y[q+2] - c- y[q-2]
//   force_a = f_c sum_b xi[a][b] S_b + f_c' e_a S_0.
// A pair then costs its U (computed once, kept in shared memory from the sum for c) and four dot
// products of HU complex entries.
//
// Linear model: c and y come from the atoms-on-lanes kernels (bispectrum_lanes.cu); here, per atom,
// the energy (c . y / 3: the energy is of third degree in c), the generators' y_b, and in passes of
// as many neighbours as the U store holds their geometry, U and dot products.  Bound: latency of
// the short phases and shared-memory reads.
//
// Quadratic model: its stress takes the neighbour's beta (the neighbour's B in the quadratic stress
// rows, mld_stress.F90:580-603): y is formed per neighbour from the Z terms (one real by complex
// product per term, a third of a dB contraction), and its dot products are taken with the generators
// applied to U.  Neighbours are lanes and four half entries a step of a warp, so the Z terms are
// broadcast, a neighbour's block weights are read without conflicts, and its y never leaves the
// registers.  The Z terms come from the atoms-on-lanes kernel, a channel at a time and asynchronously:
// formed here, they took 37 % of the kernel.  Bound: shared memory reads and FP32 arithmetic of the
// neighbours' y.
//
// Persistent CTAs take atoms from a queue.  Every sum has a fixed order that does not depend on the
// batch.
#include <cuda_runtime.h>

#include <algorithm>

#include "bispectrum.cuh"
#include "ds.cuh"

namespace mld {

namespace {

constexpr int kBatch = 32;              // neighbours (lanes) whose own y is formed at a time
constexpr int kGrow = kBatch + 1;       // row stride of their block weights (odd: no bank conflicts)
constexpr int kStressRows = 42;         // neighbours per round of the stress sums, times six components

// A sum of products of three: FP64, or a double-FP32 pair (products and sums of FP32 values are then
// as exact as FP64 ones without its 64 times slower issue).
template <typename T>
struct ExactSum;
template <>
struct ExactSum<double> {
  double v = 0.0;
  __device__ __forceinline__ void add(double f, double u, double rinv) { v += f * rinv * u; }
  __device__ __forceinline__ void add(const ExactSum& o) { v += o.v; }
  __device__ __forceinline__ ExactSum down(int d) const { return {__shfl_down_sync(0xffffffffu, v, d)}; }
  __device__ __forceinline__ double value() const { return v; }
};
template <>
struct ExactSum<float> {
  float h = 0.f, l = 0.f;
  __device__ __forceinline__ void add(float f, float u, float rinv) {
    const float p = f * rinv, pe = fmaf(f, rinv, -p);
    ds_fma(h, l, u, p, pe);
  }
  __device__ __forceinline__ void add(const ExactSum& o) { ds_add(h, l, o.h, o.l); }
  __device__ __forceinline__ ExactSum down(int d) const {
    return {__shfl_down_sync(0xffffffffu, h, d), __shfl_down_sync(0xffffffffu, l, d)};
  }
  __device__ __forceinline__ double value() const { return (double)h + (double)l; }
};

template <typename T>
struct EvalArgs {
  DevTables tb;
  const GenEntry<T>* gen;
  PairSource<T> src;
  const int* atom_struct;
  const int* small;
  const int* nbr_off;
  T chw[kMaxCh * kMaxTypes];
  T rin[kMaxTypes * kMaxTypes];
  T sign_big;
  int nch;
  const int* order;
  int* counter;
  unsigned long long chains;
  int slots;  // neighbours of the U store
  int tile;   // atoms of a tile of Z terms
  DevEval<T> ev;
};

struct EvalPlan {
  size_t hoff, quads, gamma, tbuf, yb, yt, geo, red, grow, next, U, total;
};

__host__ __device__ inline size_t up16(size_t x) { return (x + 15) & ~(size_t)15; }

__host__ __device__ inline EvalPlan eval_plan(const DevTables& tb, int nch, int eb, int slots, bool quad) {
  const size_t cxb = 2 * (size_t)eb;
  EvalPlan s;
  size_t o = 0;
  s.hoff = o;  o = up16(o + sizeof(int) * (kMaxJ + 2));
  s.quads = o; o = up16(o + sizeof(int16_t) * (tb.HU / 4 + kMaxJ + 2));
  s.gamma = o; o = up16(o + (quad ? (size_t)eb * nch * tb.NBLKP : 0));
  // Z terms of a channel, y, and the block weights of a batch, which the generators' y_b and the
  // sums over the warps follow in the same place
  s.tbuf = o;  o = up16(o + (quad ? cxb * tb.NZTP : 0));
  s.yt = o;    o = up16(o + (quad ? cxb * nch * tb.HU : 0));
  size_t w = cxb * 4 * nch * tb.HU;
  if (quad) {
    const size_t g = (size_t)eb * tb.NBLKP * kGrow, r = (size_t)eb * kNW * 2 * kBatch * 4;
    w = w > g ? w : g;
    w = w > r ? w : r;
  }
  s.yb = o;
  s.grow = o;  o = up16(o + w);
  s.geo = o;   o = up16(o + (size_t)eb * kGeo * slots);
  s.red = o;   o = up16(o + 8 * 256);
  s.next = o;  o = up16(o + 16);
  s.U = o;     o = up16(o + cxb * u_stride(tb.HU) * slots);
  s.total = o;
  return s;
}

// (aa, bb) of the stress components xx yy zz yz xz xy
__device__ __forceinline__ int stress_a(int c) { return c < 3 ? c : (c == 3 ? 1 : 0); }
__device__ __forceinline__ int stress_b(int c) { return c < 3 ? c : (c == 5 ? 1 : 2); }

template <typename T, bool kQuad>
__global__ void __launch_bounds__(kNW * 32, sizeof(T) == 4 ? 2 : 1) k_bso4_eval(EvalArgs<T> args, int A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const DevTables& tb = args.tb;
  const int J = tb.J, HU = tb.HU;
  const int nch = args.nch, nchG = nch * tb.NBLKP;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int nth = kNW * 32;
  const EvalPlan sp = eval_plan(tb, nch, (int)sizeof(T), args.slots, kQuad);
  int* shoff = reinterpret_cast<int*>(smem_raw + sp.hoff);
  int16_t* squad = reinterpret_cast<int16_t*>(smem_raw + sp.quads);  // four half entries: layer << 8 | quad
  T* sgam = reinterpret_cast<T*>(smem_raw + sp.gamma);
  cx<T>* tbuf = reinterpret_cast<cx<T>*>(smem_raw + sp.tbuf);
  cx<T>* yb = reinterpret_cast<cx<T>*>(smem_raw + sp.yb);  // [nch][HU][4]
  cx<T>* yt = reinterpret_cast<cx<T>*>(smem_raw + sp.yt);
  T* sgeo = reinterpret_cast<T*>(smem_raw + sp.geo);
  ExactSum<T>* sred = reinterpret_cast<ExactSum<T>*>(smem_raw + sp.red);
  T* grow = reinterpret_cast<T*>(smem_raw + sp.grow);
  int* snext = reinterpret_cast<int*>(smem_raw + sp.next);
  cx<T>* Us = reinterpret_cast<cx<T>*>(smem_raw + sp.U);
  const int HS = u_stride(HU);
  auto geo = [&](int n) { return sgeo + (size_t)n * kGeo; };

  // tables, once per CTA
  for (int e = tid; e < kMaxJ + 2; e += nth) shoff[e] = tb.hoff[e];
  int nquad = 0;
  for (int j = J; j >= 0; --j) {  // heaviest layers first
    const int c = (tb.hoff[j + 1] - tb.hoff[j] + 3) >> 2;
    for (int q = tid; q < c; q += nth) squad[nquad + q] = (int16_t)((j << 8) | q);
    nquad += c;
  }

  // two places for the queue position in turn: an atom without neighbours passes no other barrier, and
  // thread 0 publishes the next position while other warps may still read this one
  int nxt = first_ticket();
  for (int turn = 0;; turn ^= 1) {
    if (tid == 0) snext[turn] = ticket_position(nxt);
    __syncthreads();  // also orders the table staging and the previous atom's last reads
    const int qi = snext[turn];
    if (qi >= A) break;
    if (tid == 0) nxt = atomicAdd(args.counter, 1);
    const int atom = args.order ? args.order[qi] : qi;
    const int ti = args.src.types[atom];
    const int p0 = args.nbr_off[atom];
    const int nn = args.nbr_off[atom + 1] - p0;
    if constexpr (kQuad) {
      for (int e = tid; e < nchG; e += nth) sgam[e] = args.ev.gamma[(size_t)atom * nchG + e];
    }
    const int npass = (nn + args.slots - 1) / args.slots;
    // geometry and U of the neighbours of one pass
    auto load_pass = [&](int base, int count) {
      for (int n = tid; n < count; n += nth) {
        T* g = geo(n);
        int nb, tn;
        pair_geometry<T>(args.src, args.rin, (size_t)(p0 + base + n), ti, g, &nb, &tn);
        put_pair<T>(g, nb, tn);
        Us[(size_t)n * HS] = {T(1), T(0)};
      }
      __syncthreads();
      u_store<T>(Us, HS, count, J, args.chains, warp, lane, [&](int n) { return geo(n) + kGeoZx; });
      __syncthreads();
    };
    if (nn == 0) {  // no neighbours: the constant alone
      if (tid < 6) args.ev.Satom[(size_t)atom * 6 + tid] = 0.0;
      if (!kQuad && tid == 0) args.ev.Eatom[atom] = args.ev.w0;
      continue;
    }
    const cx<T>* ysrc = kQuad ? yt : static_cast<const cx<T>*>(args.ev.y) + (size_t)atom * nch * HU;
    // quadratic model: the atom's Z terms of a channel into tbuf, a copy per term
    auto load_z = [&](int ch) {
      const cx<T>* z = static_cast<const cx<T>*>(args.ev.z) +
                       ((size_t)(qi / args.tile) * nch + ch) * tb.NZTP * args.tile + qi % args.tile;
      for (int t = tid; t < tb.NZTP; t += nth) copy_async(tbuf + t, z + (size_t)t * args.tile);
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (!kQuad && warp == kNW - 1) {  // energy of the atom, w0 + w_lin . B = w0 + c . y / 3
      const cx<T>* csrc = static_cast<const cx<T>*>(args.ev.c) + (size_t)atom * nch * HU;
      ExactSum<T> s;
      for (int e = lane; e < nch * HU; e += 32) {
        const T w = args.gen[e % HU].w;
        const cx<T> cv = csrc[e], yv = ysrc[e];
        s.add(cv.x, yv.x, w);
        s.add(cv.y, yv.y, w);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s.add(s.down(o));
      if (lane == 0) args.ev.Eatom[atom] = args.ev.w0 + s.value() / 3.0;
    }
    // the generators' y_b, weighted for sums over the half layers
    auto form_yb = [&]() {
      for (int e = tid; e < nch * HU; e += nth) {
        const int ch = e / HU, h = e - ch * HU;
        const GenEntry<T> g = args.gen[h];
        const cx<T>* y = ysrc + ch * HU;
        const cx<T> y0 = y[h], ym = y[max(h - 1, 0)];
        cx<T> yp = y[min(h + 1, HU - 1)];
        if (g.w == T(1)) yp = {-ym.x, ym.y};  // centre of an even layer: y(0, 2) = -conj y(0, -2)
        const cx<T> a = {g.cm * ym.x, g.cm * ym.y}, b = {g.cp * yp.x, g.cp * yp.y};
        const T w = g.w, qw = g.q * g.w;
        cx<T>* o = yb + (size_t)e * 4;
        o[0] = {w * y0.x, w * y0.y};
        o[1] = {-qw * y0.y, qw * y0.x};
        o[2] = {w * (a.y + b.y), -w * (a.x + b.x)};
        o[3] = {w * (b.x - a.x), w * (b.y - a.y)};
      }
    };
    if constexpr (!kQuad) form_yb();  // (each pass begins with barriers)
    // ---- pairs: forces (and, linear model, stress) ---------------------------------------------
    const T lev = args.small[args.atom_struct[atom]] ? T(1) : -args.sign_big;  // stress lever arm: sign * u
    ExactSum<T> sacc;  // of this thread's (pair slot, component)
    const int srow = tid / 6, scomp = tid - srow * 6;  // quadratic model: its neighbours and component
    for (int ps = npass - 1; ps >= 0; --ps) {
      const int base = ps * args.slots, count = min(args.slots, nn - base);
      if constexpr (kQuad) load_z(0);  // (arrives beside the geometry and U)
      load_pass(base, count);
      if constexpr (kQuad) {
        // stress sums S_b of the pass's neighbours with their own beta, channel by channel
        T st[2][4];
#pragma unroll
        for (int i = 0; i < 8; ++i) st[i >> 2][i & 3] = T(0);
        for (int ch = 0; ch < nch; ++ch) {
          asm volatile("cp.async.wait_group 0;" ::: "memory");
          __syncthreads();
          if (ps == npass - 1) {
            // y of the atom: the blocks of each layer with its own weights, in order
            for (int h = tid; h < HU; h += nth) {
              int j = 0;
              while (shoff[j + 1] <= h) ++j;
              const int H = shoff[j + 1] - shoff[j];
              const cx<T>* z = tbuf + tb.zoffp[j] + (h - shoff[j]);
              const T* g = sgam + ch * tb.NBLKP + tb.blkp_off[j];
              const int nb = tb.blkp_off[j + 1] - tb.blkp_off[j];
              cx<T> v = {T(0), T(0)};
#pragma unroll 4
              for (int r = 0; r < nb; ++r) {
                const cx<T> zr = z[r * H];
                v.x = fma(g[r], zr.x, v.x);
                v.y = fma(g[r], zr.y, v.y);
              }
              yt[ch * HU + h] = v;
            }
          }
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const int b0 = b * kBatch;
            if (b0 >= count) continue;
            for (int n = warp; n < min(kBatch, count - b0); n += kNW) {
              const int nb = reinterpret_cast<const int*>(geo(b0 + n) + kGeoIdx)[0];
              const T* src = args.ev.gamma + (size_t)nb * nchG + ch * tb.NBLKP;
              for (int r = lane; r < tb.NBLKP; r += 32) grow[r * kGrow + n] = src[r];
            }
            __syncthreads();
            const int n = min(b0 + lane, count - 1);
            const cx<T>* u = Us + (size_t)n * HS;
            const T wn = args.chw[ch * args.src.ntypes + pair_type<T>(geo(n))];
            for (int it = warp; it < nquad; it += kNW) {
              const int q = squad[it], j = q >> 8, e0 = (q & 255) * 4;
              const int H = shoff[j + 1] - shoff[j], nb = tb.blkp_off[j + 1] - tb.blkp_off[j];
              const cx<T>* z = tbuf + tb.zoffp[j] + e0;
              const T* g = grow + tb.blkp_off[j] * kGrow + (n - b0);
              cx<T> y[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) y[i] = {T(0), T(0)};
              // (the last step of a layer reads up to three values past its entries; they are not used)
#pragma unroll 2
              for (int r = 0; r < nb; ++r) {
                const T w = g[r * kGrow];
                const cx<T> ww = {w, w};
#pragma unroll
                for (int i = 0; i < 4; ++i) y[i] = fma2(ww, z[r * H + i], y[i]);
              }
              const int h0 = shoff[j] + e0;
              cx<T> um = u[max(h0 - 1, 0)], u0 = u[h0];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                if (e0 + i < H) {
                  const GenEntry<T> ge = args.gen[h0 + i];
                  const cx<T> up = u[min(h0 + i + 1, HU - 1)];
                  // w y . (U, T1 U, T2 U, T3 U)
                  cx<T> uq = up;
                  if (ge.w == T(1)) uq = {-um.x, um.y};
                  const cx<T> a = {ge.cm * um.x, ge.cm * um.y}, c = {ge.cp * uq.x, ge.cp * uq.y};
                  const cx<T> s = {a.x + c.x, a.y + c.y}, d = {a.x - c.x, a.y - c.y};
                  const T wg = ge.w * wn;
                  const cx<T> yw = {wg * y[i].x, wg * y[i].y};
                  st[b][0] = fma(yw.x, u0.x, fma(yw.y, u0.y, st[b][0]));
                  st[b][1] = fma(ge.q, fma(yw.x, u0.y, -(yw.y * u0.x)), st[b][1]);
                  st[b][2] = fma(-yw.x, s.y, fma(yw.y, s.x, st[b][2]));
                  st[b][3] = fma(yw.x, d.x, fma(yw.y, d.y, st[b][3]));
                  um = u0;
                  u0 = up;
                }
              }
            }
            __syncthreads();  // the weights have been read (and, after the last batch, the Z terms)
          }
          if (ch + 1 < nch) load_z(ch + 1);
        }
        // sums over the warps, in order; then the stress of (neighbour, component)
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int i = 0; i < 4; ++i) grow[((warp * 2 + b) * kBatch + lane) * 4 + i] = st[b][i];
        __syncthreads();
        if (srow < kStressRows) {
          const int aa = stress_a(scomp), bb = stress_b(scomp);
          for (int n = srow; n < count; n += kStressRows) {
            T S[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) {
              S[b] = T(0);
#pragma unroll
              for (int w = 0; w < kNW; ++w) S[b] += grow[((w * 2 + n / kBatch) * kBatch + n % kBatch) * 4 + b];
            }
            const T* g = geo(n);
            const T* xi = g + kGeoXi + 3 * aa;
            const T f = fma(g[kGeoFc], fma(xi[0], S[1], fma(xi[1], S[2], xi[2] * S[3])), g[kGeoDfr + aa] * S[0]);
            sacc.add(f, lev * g[kGeoU + bb], g[kGeoU + 3]);
          }
        }
        __syncthreads();
        form_yb();  // where the sums were
        __syncthreads();
      }
      for (int g4 = warp * 4; g4 < count; g4 += kNW * 4) {
        // a warp takes four pairs, its lanes the half entries
        T tot[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) tot[i] = T(0);
        const cx<T>* up[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) up[i] = Us + (size_t)min(g4 + i, count - 1) * HS;
        for (int ch = 0; ch < nch; ++ch) {
          cx<T> acc[4][4];
#pragma unroll
          for (int i = 0; i < 16; ++i) acc[i >> 2][i & 3] = {T(0), T(0)};
          const cx<T>* yc = yb + (size_t)ch * HU * 4;
          for (int e = lane; e < HU; e += 32) {
            cx<T> y[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) y[b] = yc[e * 4 + b];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const cx<T> u = up[i][e];
#pragma unroll
              for (int b = 0; b < 4; ++b) acc[i][b] = fma2(y[b], u, acc[i][b]);
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int tn = pair_type<T>(geo(min(g4 + i, count - 1)));
            const T w = args.chw[ch * args.src.ntypes + tn];
#pragma unroll
            for (int b = 0; b < 4; ++b) tot[i * 4 + b] = fma(w, acc[i][b].x + acc[i][b].y, tot[i * 4 + b]);
          }
        }
        // sums over the lanes: lane l ends with value l / 2 (pair l / 8, direction (l / 2) % 4)
#pragma unroll
        for (int s = 8; s > 0; s >>= 1) {
          const bool hi = lane & (2 * s);
#pragma unroll
          for (int i = 0; i < s; ++i) {
            const T keep = hi ? tot[i + s] : tot[i], send = hi ? tot[i] : tot[i + s];
            tot[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * s);
          }
        }
        const T v = tot[0] + __shfl_xor_sync(0xffffffffu, tot[0], 1);
        // forces on lanes (pair, component) = (l / 3, l % 3) < 12
        const int fi = min(lane / 3, 3), fa = lane % 3;
        T S[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) S[b] = __shfl_sync(0xffffffffu, v, (fi * 4 + b) * 2);
        const T* g = geo(min(g4 + fi, count - 1));
        const T* xi = g + kGeoXi + 3 * fa;
        const T f = fma(g[kGeoFc], fma(xi[0], S[1], fma(xi[1], S[2], xi[2] * S[3])), g[kGeoDfr + fa] * S[0]);
        if (lane < 12 && g4 + fi < count) args.ev.pair[(size_t)(p0 + base + g4 + fi) * 3 + fa] = f;
        if constexpr (!kQuad) {
          // stress on lanes (pair, component) = (l / 6, l % 6) < 24
          const int si = min(lane / 6, 3), sc = lane % 6;
          const T fs = __shfl_sync(0xffffffffu, f, si * 3 + stress_a(sc));
          const T* gs = geo(min(g4 + si, count - 1));
          if (lane < 24 && g4 + si < count)
            sacc.add(fs, lev * gs[kGeoU + stress_b(sc)], gs[kGeoU + 3]);
        }
      }
      if (ps > 0) __syncthreads();  // the pass's U and geometry have been read
    }
    // stress of the atom: the partial sums of (slot, component), slots in order
    if constexpr (kQuad) {
      if (srow < kStressRows) sred[tid] = sacc;
      __syncthreads();
      if (tid < 6) {
        ExactSum<T> v;
        for (int n = 0; n < kStressRows; ++n) v.add(sred[n * 6 + tid]);
        args.ev.Satom[(size_t)atom * 6 + tid] = v.value();
      }
    } else {
      if (lane < 24) sred[warp * 24 + lane] = sacc;
      __syncthreads();
      if (warp == 0) {
        ExactSum<T> v;
        if (lane < 24)
          for (int w = 0; w < kNW; ++w) v.add(sred[w * 24 + lane]);
        v.add(v.down(12));  // slots (0 + 2) and (1 + 3), then both
        v.add(v.down(6));
        if (lane < 6) args.ev.Satom[(size_t)atom * 6 + lane] = v.value();
      }
    }
  }
}

int max_optin() {
  static int v = 0;
  if (!v) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  }
  return v;
}

}  // namespace

template <typename T>
cudaError_t launch_bso4_eval(const DevTables& tb, const DevBatch& b, const BsoParams& p, const DevEval<T>& ev,
                             const int* order, int count, int* counter, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  const bool quad = ev.gamma != nullptr;
  if (!counter || !ev.pair || !ev.Satom || !tb.gen32 || (quad ? !ev.z : !ev.c || !ev.y)) return cudaErrorInvalidValue;
  EvalArgs<T> a{};
  a.tb = tb;
  if constexpr (sizeof(T) == 8) {
    a.gen = reinterpret_cast<const GenEntry<T>*>(tb.gen64);
  } else {
    a.gen = reinterpret_cast<const GenEntry<T>*>(tb.gen32);
  }
  a.src = {b.types, b.nbr_idx, b.nbr_u, sizeof(T) == 4 ? b.nbr_u32 : nullptr, (T)p.rcut, (T)p.inv_r0,
           (T)p.rin_width, p.ntypes, p.has_rin, {}};
  a.src.rates.set(p.rcut, p.inv_r0);
  a.atom_struct = b.atom_struct;
  a.small = b.small;
  a.nbr_off = b.nbr_off;
  for (int e = 0; e < kMaxCh * kMaxTypes; ++e) a.chw[e] = (T)p.chw[e];
  for (int e = 0; e < kMaxTypes * kMaxTypes; ++e) a.rin[e] = (T)p.rin[e];
  a.sign_big = (T)p.sign_big;
  a.nch = p.nch;
  a.order = order;
  a.counter = counter;
  a.chains = chain_order(tb.J);
  a.ev = ev;
  a.tile = quad ? lane_tile(tb, (int)sizeof(T)) : 1;
  if (!a.tile) return cudaErrorInvalidConfiguration;
  // the largest U store (up to 64 neighbours) that keeps the CTAs per SM of a 32-neighbour one (at
  // most two: registers); it depends on the configuration only, not on the batch
  const size_t per_sm = 228 * 1024;
  auto bytes = [&](int slots) { return eval_plan(tb, p.nch, (int)sizeof(T), slots, quad).total; };
  const size_t want = std::min<size_t>(sizeof(T) == 4 ? 2 : 1, per_sm / (bytes(32) + 1024));
  a.slots = 8;
  for (int s = 64; s > 8; s -= 4)
    if (bytes(s) <= (size_t)max_optin() && per_sm / (bytes(s) + 1024) >= std::max<size_t>(want, 1)) {
      a.slots = s;
      break;
    }
  const size_t smem = bytes(a.slots);
  if (smem > (size_t)max_optin()) return cudaErrorInvalidConfiguration;
  auto kern = quad ? k_bso4_eval<T, true> : k_bso4_eval<T, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int dev = 0, nsm = 0, occ = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kNW * 32, smem);
  if (e != cudaSuccess) return e;
  if (occ < 1) return cudaErrorInvalidConfiguration;
  const long long grid = std::min<long long>(count, (long long)nsm * occ);
  e = cudaMemsetAsync(counter, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  kern<<<(unsigned)grid, kNW * 32, smem, st>>>(a, count);
  return cudaGetLastError();
}

template cudaError_t launch_bso4_eval<double>(const DevTables&, const DevBatch&, const BsoParams&,
                                              const DevEval<double>&, const int*, int, int*, cudaStream_t);
template cudaError_t launch_bso4_eval<float>(const DevTables&, const DevBatch&, const BsoParams&,
                                             const DevEval<float>&, const int*, int, int*, cudaStream_t);

}  // namespace mld
