// Internal declarations shared by the CUDA translation units of libmld_gpu.
// Nothing here is part of the public C ABI (include/mld_gpu.h).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <stdint.h>
#include <string>
#include <vector>

namespace mld {

constexpr int kMaxJ = 10;          // doubled angular momentum bound (j_max <= 5)
constexpr int kMaxTypes = 8;       // element types per handle
constexpr int kMaxCh = 3;          // plain, weighted, weighted_3ch
constexpr int kRowTile = 4;        // rows (triples) per register tile of the dB contraction


// Symmetry used throughout: U^j(-p,-q) = (-1)^((p-q)/2) conj(U^j(p,q)); the same holds for c,
// the Z blocks and vecall.  Only the "half" of each layer is stored: the first
// H_j = ceil((j+1)^2/2) entries in row-major (p, q) order.  A source reference into a half
// layer is encoded as (half_index << 2) | (conj << 1) | negate, or -1 when absent.

// One output element of the Z contraction (compute_bispectrum_so4.F90:1014-1143).
// Z(m1,m2) = sum_{a<na, b<nb} cg1[a]*cg2[b] * c[i1 + a*s1 + b] * c[i2 - a*s2 - b]
// (full-layer indices of c) where layer jA supplies the first factor and jB the second.
struct ZTerm {
  uint16_t i1, i2;         // flattened c index of the first (ma,mb) / matching second factor
  uint16_t cg1, cg2;       // offsets into the 1-D CG coefficient table
  uint8_t na, nb, s1, s2;  // loop extents and layer strides (j+1)
  uint8_t snum, sden;      // scale snum/sden: 1 for ZA, (l+1)/(l1+1) for ZB, (l+1)/(l2+1) for ZC
  uint16_t pad;
};

// One slot of the folded Y array: triple k, layer j, half entry e.  Y = wgt * sum of the scaled
// Z blocks of k living on layer j at that entry; wgt = 2 off the symmetry centre, 1 on it.
struct YSlot {
  uint16_t term[3];
  uint8_t nterm;
  uint8_t is_a;            // term[0] is the ZA block (contributes to B_k)
  uint16_t ufull;          // full (j,p,q) index into c
  uint16_t k;              // triple index
  uint16_t ypos;           // position in the layer-blocked Y array
  uint8_t wgt;             // 2 or 1
  uint8_t pad;
};

// One lane of a phase-2 round (16 bytes): the Z term's c indices of its first product, CG
// offsets, loop extents and strides, and the term's index in the per-atom term buffer
// (kNoTerm marks a padding lane).
struct alignas(16) ZItem {
  uint16_t i1, i2, cg1, cg2;  // first (ma,mb) c index / matching second factor, CG offsets
  uint8_t na, nb, s1, s2;     // loop extents and layer strides (j+1)
  uint16_t term;              // index of the term (its Z value) in the term buffer
  uint16_t pad;
};
static_assert(sizeof(ZItem) == 16, "phase-2 entries are 16 bytes");
// the descriptor kernel decodes entries from their four 32-bit words at these byte offsets
static_assert(offsetof(ZItem, i2) == 2 && offsetof(ZItem, cg1) == 4 && offsetof(ZItem, cg2) == 6 &&
                  offsetof(ZItem, na) == 8 && offsetof(ZItem, nb) == 9 && offsetof(ZItem, s1) == 10 &&
                  offsetof(ZItem, s2) == 11 && offsetof(ZItem, term) == 12,
              "ZItem layout");
constexpr uint16_t kNoTerm = 0xFFFF;

// One folded Y slot with its distinct terms (host only; the kernels take the rows' sources instead, whose
// order tests compare with it): Y[ypos] = wgt * sum_t (snum_t / sden_t) Z[term_t].
struct SlotEntry {
  uint16_t term[3];
  uint16_t ypos;
  uint8_t nterm, wgt;
  uint8_t snum[3], sden[3];
};

// One ZA half entry of a triple (host only, as SlotEntry): B_k = sum over its entries of
// wgt * Re(conj(c[ufull]) Z[term]).
struct BkItem {
  uint16_t term, ufull;
  uint8_t wgt, pad[3];
};

// A record of the atoms-on-lanes sums (bispectrum_lanes.cu; 32 bytes): for an operand pair jA >= jB and
// an output position (m1, m2), the Z terms of nj of the pair's output layers in descending jO,
//   Z_o = sum_{a<na} cgv[cg1 + a st1 + o] sum_{b<nb} cgv[cg2 + b st2 + o] c[i1 + a s1 + b] c[i2 - a s2 - b].
constexpr int kMaxZOut = kMaxJ / 2 + 1;
struct alignas(16) LaneRec {
  uint16_t i1, i2, cg1, cg2;
  uint8_t na, nb, s1, s2;
  uint8_t st1, st2, nj, off;  // off (y): the job's output of Z_0
  uint16_t out[kMaxZOut];     // y: the terms' blocks; B: c indices of the output position
  uint16_t w;                 // B: weight of the position in a sum over full layers
  uint16_t pad;
};
static_assert(sizeof(LaneRec) == 32, "lane records are two 16-byte words");
static_assert(offsetof(LaneRec, na) == 8 && offsetof(LaneRec, st1) == 12 && offsetof(LaneRec, out) == 16 &&
                  offsetof(LaneRec, w) == 28,
              "LaneRec layout (decoded from its words)");
// A job: its records in four parts of about equal work, and its outputs (y: half entries of the
// layers jO in descending order; B: triples)
struct LaneJob {
  int rec[5];
  uint16_t nout;
  uint16_t out[kMaxZOut];
  uint16_t pad;
};

// Layer l of a triple and the first term of its ZA block: B_k = sum_e w_e Re(conj(c^l[e]) Z[za + e]).
struct TripleZ {
  uint16_t za;
  uint16_t l;
};
// A contribution of triple k to the weight of a Z block.
struct GammaItem {
  uint16_t k;
  uint8_t snum, sden;
};
// A contraction row (triple, layer): Y[e] = w_e sum_t (snum_t / sden_t) Z[z_t + e], nterm <= 3 (0: padding).
struct alignas(16) RowSource {
  uint16_t z[3];
  uint16_t nterm;
  uint8_t snum[3], sden[3];
  uint16_t pad;
};
static_assert(sizeof(RowSource) == 16, "row sources are 16 bytes");

constexpr int kZWarps = 8;   // warps of the phase-2 schedule (= warps of a k_bso4 CTA)
constexpr int kRounds = 3;   // ranks of a triple's layer rows (its distinct layers in ascending order)
constexpr int kRankShift = 12;  // row destination code: (rank << kRankShift) | index within the rank's buffer

// Host-built constant tables of the SO(4) bispectrum for a given j_max.
struct Bso4Tables {
  std::vector<ZItem> zitems;    // phase-2 rounds of 32 terms of one nb (na descending), grouped per warp (LPT)
  std::vector<int> zitem_off;   // kZWarps + 1 round offsets (a round is 32 consecutive zitems)
  int J = 0, NU = 0, HU = 0, K = 0, NYP = 0;
  int off[kMaxJ + 2] = {0};     // full-layer offsets
  int hoff[kMaxJ + 2] = {0};    // half-layer offsets
  int Mp[kMaxJ + 1] = {0};      // padded row count per layer (multiple of kRowTile per round group)
  int yoff[kMaxJ + 1] = {0};    // Y offset of each layer block (complex elements)
  std::vector<int> l1, l2, l;   // triples (reference order)
  std::vector<double> cg;       // 1-D CG coefficient lists
  std::vector<ZTerm> zterms;    // ZA/ZB/ZC outputs on half layers
  int nzu = 0;                  // distinct Z computations among them (the term buffer's entries)
  std::vector<YSlot> yslots;    // folded slots
  std::vector<SlotEntry> slots; // the same slots with their distinct terms and Y positions
  std::vector<int> bk_off;      // K + 1 offsets into bk_items
  std::vector<BkItem> bk_items; // ZA entries of each triple
  // per layer-block row: destination code (rank << kRankShift) | index, -1 for padding; the
  // index is the triple for rank 0 and the triple's slot in the rank-1 / rank-2 buffers
  std::vector<int16_t> rowk;
  int rowk_off[kMaxJ + 2] = {0};  // offset of each layer's rows in rowk
  std::vector<int> tiles;       // row tiles (j << 8 | rt), heaviest layers first
  int nrank[kRounds] = {0};     // triples with a row of rank r (rank 0: all K)
  std::vector<int16_t> rank_slot;  // K x (kRounds - 1): slot of triple k in the rank-1 / rank-2 buffers, -1 none
  // recursion on half layers, U = tz*Zsel*U[src_z] + tx*(-i)*Xsel*U[src_x] (host only: the kernels run
  // column chains)
  std::vector<double> rec_tz, rec_tx;
  std::vector<int16_t> rec_sz, rec_sx;
  std::vector<int8_t> rec_qneg;
  std::vector<int16_t> expand;  // full index -> encoded half source
  // generators on the half layers (4 values per entry (j, p, q)): c- = sqrt((j+q)/2 ((j-q)/2 + 1)) and
  // c+ = sqrt((j-q)/2 ((j+q)/2 + 1)), the weights of the entries at q - 2 and q + 2; q; the entry's
  // weight in a sum over full layers (2; 1 on the centre (0, 0) of an even layer, whose entry at
  // q + 2 is -conj of the one at q - 2)
  std::vector<double> gen;
  // the distinct Z blocks (jA, jB -> jO), grouped by output layer: block r of layer j holds the terms
  // zoff[j] + r * H_j + e of its half entries e
  int zoff[kMaxJ + 1] = {0};
  // the blocks with their operands in descending order (blocks that differ by the exchange are one),
  // as the atoms-on-lanes sums count them, layer by layer.  dE/dB_k = beta_k weighs block b with
  // gamma_b = sum over [gamp_off[b], gamp_off[b + 1]) of (snum / sden) beta_k
  int nblk_pair = 0;
  std::vector<int> gamp_off;
  std::vector<GammaItem> gamp;
  // atoms-on-lanes sums: CG coefficients of a pair by (m, first index, jO descending), the records and
  // jobs of B (a job per operand pair) and y (a job per output position), heaviest jobs first
  std::vector<double> cgv;
  std::vector<LaneRec> brecs, yrecs, zrecs;  // zrecs: yrecs with the terms' places in place of their blocks
  int nztp = 0;                   // terms of the pair blocks, by layer, block and half entry
  int blkp_off[kMaxJ + 2] = {0};  // first pair block and term of every layer
  int zoffp[kMaxJ + 1] = {0};
  std::vector<TripleZ> trzp;      // trz on these terms
  std::vector<LaneJob> bjobs, yjobs;
  std::vector<TripleZ> trz;       // the ZA block and layer of each triple
  std::vector<RowSource> rowsrc;  // the blocks of every contraction row, indexed as rowk
  std::vector<RowSource> rowsrc2; // the same on the terms of the pair blocks
  std::vector<int8_t> half_diag;  // half entries on the diagonal p == q (get the +1 of c)
  long long cg_terms = 0;       // CG products evaluated per channel (half outputs)
  long long cg_terms_full = 0;  // CG products of the unfolded contraction (reference count)
  long long u_one = 0, u_two = 0;  // half-layer recursion entries with one / two source terms
};

bool build_bso4_tables(double j_max, Bso4Tables* t, std::string* err);
double cg_coefficient(int j1, int m1, int j2, int m2, int j, int m);  // doubled indices

// A half-layer entry's generator weights and weight in full-layer sums (Bso4Tables::gen).
template <typename T>
struct alignas(16) GenEntry {
  T cm, cp, q, w;
};

// Device copies of the tables.
struct DevTables {
  int J = 0, NU = 0, HU = 0, K = 0, NYP = 0, NTILE = 0, NZT = 0, NROWS = 0;
  int NCG = 0;  // entries of the 1-D CG coefficient table
  int NCGV = 0, NBJ = 0, NYJ = 0, NBLKP = 0, NZTP = 0;
  int blkp_off[kMaxJ + 2] = {0};
  int zoffp[kMaxJ + 1] = {0};
  double* cgv64 = nullptr;        // NCGV
  float2* cgv32x2 = nullptr;      // every coefficient twice
  LaneRec* brecs = nullptr;
  LaneJob* bjobs = nullptr;       // NBJ
  LaneRec* yrecs = nullptr;       // (fill_deriv_tables)
  LaneJob* yjobs = nullptr;       // NYJ
  LaneRec* zrecs = nullptr;
  RowSource* rowsrc2 = nullptr;
  TripleZ* trzp = nullptr;        // K
  TripleZ* trz = nullptr;         // K
  RowSource* rowsrc = nullptr;    // NROWS
  int hoff[kMaxJ + 2] = {0};
  int Mp[kMaxJ + 1] = {0};
  int yoff[kMaxJ + 1] = {0};
  int rowk_off[kMaxJ + 2] = {0};
  int nrank[kRounds] = {0};
  int16_t* rowk = nullptr;
  int16_t* rank_slot = nullptr;  // K x (kRounds - 1)
  int* tiles = nullptr;
  double* cg64 = nullptr;
  float* cg32 = nullptr;
  int16_t* expand = nullptr;
  int8_t* half_diag = nullptr;
  ZItem* zitems = nullptr;
  int* zitem_off = nullptr;     // kZWarps + 1
  // tables of the derivatives and the evaluation (fill_deriv_tables)
  GenEntry<float>* gen32 = nullptr;   // HU
  GenEntry<double>* gen64 = nullptr;  // HU
  int* gamp_off = nullptr;      // NBLKP + 1
  GammaItem* gamp = nullptr;
};

// Fill the scalar part of *d from t and place every device table through put(vector, &ptr),
// which allocates (or carves) device memory of the vector's size and copies it there.
template <class Put>
cudaError_t fill_dev_tables(const Bso4Tables& t, DevTables* d, Put put) {
  *d = DevTables();
  d->J = t.J;
  d->NU = t.NU;
  d->HU = t.HU;
  d->K = t.K;
  d->NYP = t.NYP;
  d->NTILE = (int)t.tiles.size();
  d->NZT = t.nzu;
  d->NROWS = (int)t.rowk.size();
  d->NCG = (int)t.cg.size();
  for (int j = 0; j <= t.J + 1; ++j) {
    d->hoff[j] = t.hoff[j];
    d->rowk_off[j] = t.rowk_off[j];
  }
  for (int j = 0; j <= t.J; ++j) {
    d->Mp[j] = t.Mp[j];
    d->yoff[j] = t.yoff[j];
  }
  for (int r = 0; r < kRounds; ++r) d->nrank[r] = t.nrank[r];
  // the CG table padded to whole 16-byte chunks (the descriptor kernel stages it with 16-byte
  // asynchronous copies)
  std::vector<double> cg64(t.cg);
  cg64.resize((cg64.size() + 1) / 2 * 2, 0.0);
  std::vector<float> cg32(t.cg.begin(), t.cg.end());
  cg32.resize((cg32.size() + 3) / 4 * 4, 0.0f);
  cudaError_t e = cudaSuccess;
  if (e == cudaSuccess) e = put(t.rowk, &d->rowk);
  if (e == cudaSuccess) e = put(t.rank_slot, &d->rank_slot);
  if (e == cudaSuccess) e = put(t.tiles, &d->tiles);
  if (e == cudaSuccess) e = put(cg64, &d->cg64);
  if (e == cudaSuccess) e = put(cg32, &d->cg32);
  if (e == cudaSuccess) e = put(t.expand, &d->expand);
  if (e == cudaSuccess) e = put(t.half_diag, &d->half_diag);
  if (e == cudaSuccess) e = put(t.zitems, &d->zitems);
  d->NCGV = (int)t.cgv.size();
  d->NBJ = (int)t.bjobs.size();
  std::vector<float2> cgv32x2;
  for (double v : t.cgv) cgv32x2.push_back(make_float2((float)v, (float)v));
  if (e == cudaSuccess) e = put(t.cgv, &d->cgv64);
  if (e == cudaSuccess) e = put(cgv32x2, &d->cgv32x2);
  if (e == cudaSuccess) e = put(t.brecs, &d->brecs);
  if (e == cudaSuccess) e = put(t.bjobs, &d->bjobs);
  if (e == cudaSuccess) e = put(t.trz, &d->trz);
  if (e == cudaSuccess) e = put(t.rowsrc, &d->rowsrc);
  if (e == cudaSuccess) e = put(t.zitem_off, &d->zitem_off);
  return e;
}

// Device tables that only derivatives and evaluation need, placed like those of fill_dev_tables.
template <class Put>
cudaError_t fill_deriv_tables(const Bso4Tables& t, DevTables* d, Put put) {
  std::vector<GenEntry<float>> g32(t.HU);
  std::vector<GenEntry<double>> g64(t.HU);
  for (int h = 0; h < t.HU; ++h) {
    const double* g = &t.gen[4 * (size_t)h];
    g32[h] = {(float)g[0], (float)g[1], (float)g[2], (float)g[3]};
    g64[h] = {g[0], g[1], g[2], g[3]};
  }
  cudaError_t e = put(g32, &d->gen32);
  if (e == cudaSuccess) e = put(g64, &d->gen64);
  d->NBLKP = t.nblk_pair;
  if (e == cudaSuccess) e = put(t.gamp_off, &d->gamp_off);
  if (e == cudaSuccess) e = put(t.gamp, &d->gamp);
  d->NYJ = (int)t.yjobs.size();
  if (e == cudaSuccess) e = put(t.yrecs, &d->yrecs);
  if (e == cudaSuccess) e = put(t.yjobs, &d->yjobs);
  d->NZTP = t.nztp;
  if (e == cudaSuccess) e = put(t.zrecs, &d->zrecs);
  if (e == cudaSuccess) e = put(t.rowsrc2, &d->rowsrc2);
  if (e == cudaSuccess) e = put(t.trzp, &d->trzp);
  for (int j = 0; j <= t.J + 1; ++j) d->blkp_off[j] = t.blkp_off[j];
  for (int j = 0; j <= t.J; ++j) d->zoffp[j] = t.zoffp[j];
  return e;
}

// Per-batch structure description on the device.
struct DevBatch {
  int S = 0;                 // structures
  int A = 0;                 // atoms
  int* atom_start = nullptr; // S+1
  int* atom_struct = nullptr;// A
  int* types = nullptr;      // A
  double* pos = nullptr;     // 3A
  double* cell = nullptr;    // 9S  (cell[9s+3i+c] = a_i[c])
  double* recip = nullptr;   // 9S  (b_k with a_i.b_k = delta)
  int* small = nullptr;      // S
  int* nsize = nullptr;      // 3S
  double* volume = nullptr;  // S
  // FP32 copies for the neighbour pre-filter (written by the counting pass)
  float4* pos32 = nullptr;   // A  (x, y, z, 0)
  float4* frac32 = nullptr;  // A  (fractional coordinates b_k . x, 0)
  // neighbour list (CSR over atoms)
  int* nn = nullptr;         // A
  int* nbr_off = nullptr;    // A+1
  int* nbr_idx = nullptr;    // P
  double* nbr_u = nullptr;   // 3P  (x_neighbour - x_centre, FP64)
  float4* nbr_u32 = nullptr; // P (x, y, z, 1/r) rounded from the FP64 values, for the FP32
                             // descriptor kernel (null: it converts nbr_u itself)
  long long P = 0;
  int maxnn = 0;             // largest neighbour count (after the counting pass)
  // linked cells of large boxes (null cnc: every structure scans all its atoms)
  int* cnc = nullptr;        // 3S cells per lattice direction, 0 for a structure without cells
  int* cell_off = nullptr;   // S+1 first cell of each structure
  int ncells = 0;
  int* cell_of = nullptr;    // A cell of each atom (-1 without cells)
  int* cell_start = nullptr; // ncells+1 first entry of each cell in cell_atoms (then a cursor of ncells)
  int* cell_atoms = nullptr; // A atoms grouped by cell
  int* sort_tmp = nullptr;   // P  neighbour indices while the lists of celled structures are sorted
  // single-pass search: each atom's pairs (neighbour, packed image) in a row of nbr_cap entries
  int2* nbr_tmp = nullptr;   // A * nbr_cap
  int nbr_cap = 0;
};

// Design-row placement of each structure (-1 when a block is absent).
struct DevRows {
  long long M = 0;           // rows
  int D = 0;                 // row width (1 + nch*K for linear)
  int ldx = 0;               // row stride of the design matrix (D rounded up to 4)
  long long* rowE = nullptr; // S
  long long* rowF = nullptr; // S (first of 3*nat force rows)
  long long* rowS = nullptr; // S (first of 6 stress rows)
};

struct BsoParams {
  double rcut, inv_r0;       // inv_r0 = pi * inv_r0_input
  int nch, ntypes;
  double chw[kMaxCh * kMaxTypes];
  double rin[kMaxTypes * kMaxTypes];
  double rin_width;
  int has_rin;
  double sign_stress, sign_big;
};

inline int round_up4(int d) { return (d + 3) & ~3; }

// Kernels / launchers (return cudaError_t of the launch).
// pass 0 counts and 1 fills the CSR lists (two scans of the candidates); pass 2 counts and
// writes each atom's pairs into b.nbr_tmp in one scan, pass 3 then compacts them into the CSR.
// Passes 1 and 3 end with the sorted lists of celled structures and the displacements.
cudaError_t launch_neighbours(const DevBatch& b, double rcut, int* counts, int* maxcount, cudaStream_t st,
                              int pass);
cudaError_t launch_scan(const int* in, int* out, int n, int* d_tmp, cudaStream_t st);
// Bin the atoms of celled structures (b.cnc) into their cells; scan_tmp as for launch_scan over
// b.ncells entries.  Then launch_neighbours scans the 27 (or fewer, unique) cells around each
// atom, and launch_sort_lists restores the ascending neighbour order of those atoms' lists.
cudaError_t launch_cells(const DevBatch& b, int* scan_tmp, cudaStream_t st);
cudaError_t launch_sort_lists(const DevBatch& b, cudaStream_t st);

// Y scratch the descriptor kernel needs in global memory for up to max_ctas CTAs (0 when Y fits
// in shared memory); pass it to launch_bso4, which then runs at most that many persistent CTAs.
// Bytes of the descriptor kernel's global Y slices for max_ctas persistent CTAs: needed when Y
// does not fit in shared memory, and preferred (unless only_if_required) when it would cost a
// resident CTA per SM; 0 otherwise.
size_t bso4_y_scratch_bytes(const DevTables& tb, int nch, int eb, int max_ctas, bool only_if_required = false);
// whether the kernel's shared memory fits at all (FP64 at j_max 5 does not)
bool bso4_available(const DevTables& tb, int nch, int eb);
// Launch shape of the descriptor kernel, chosen per handle by the autotuner (api.cu); every
// shape gives bitwise the same results.
struct Bso4Launch {
  int col_tile = 2;      // columns per register tile of k_deriv's contraction: 2 or 4 (492,000 Fe atoms: 58
                         // against 62 ms; wider tiles leave long jobs to few warps at the end of a phase)
  int sorted_queue = 1;  // atoms longest first (1) or in index order (0)
};
// c (count x nch x HU complex of T) of atoms first .. first + count - 1, or of order[0 .. count - 1]
// (first = 0).  Rows by atom (atom - first) or by position in the queue.  counter: one int of device
// memory, reset by the launch.
template <typename T>
cudaError_t launch_c_half(const DevTables& tb, const DevBatch& b, const BsoParams& p, int first, int count,
                          const int* order, bool by_position, int* counter, void* c, cudaStream_t st);
// B (whole-batch array) of the same atoms from their c.
template <typename T>
cudaError_t launch_lane_descriptors(const DevTables& tb, const DevBatch& b, const BsoParams& p, int first, int count,
                                    const void* c, T* B, cudaStream_t st);
// y = dE/dc (as c) of the same atoms with the pair-block weights gamma (nch * NBLKP, from
// launch_block_weights).
template <typename T>
cudaError_t launch_lane_y(const DevTables& tb, const DevBatch& b, const BsoParams& p, int first, int count,
                          const void* c, const void* gamma, void* y, cudaStream_t st);

// Y rows of `count` rows of Z terms, [position][nch][NYP], and from them and c (by position) B and
// w_ch * dB (whole-batch arrays) of atoms first .. first + count - 1, or of order[0 .. count - 1]
// (bispectrum_deriv.cu).
template <typename T>
cudaError_t launch_y_rows(const DevTables& tb, int nch, int count, const void* z, void* y, cudaStream_t st);
template <typename T>
cudaError_t launch_deriv(const DevTables& tb, const DevBatch& b, const BsoParams& p, int first, int count,
                         const int* order, int* counter, const void* c, const void* y, T* Bout, T* dBout,
                         const Bso4Launch& shape, cudaStream_t st);
bool deriv_available(const DevTables& tb, int nch, int eb);
// Z terms of `count` rows of c, [tile][nch][NZTP][atoms of a tile] complex of T; lane_tile: atoms of a
// tile (0: the tables do not fit).
int lane_tile(const DevTables& tb, int eb);
// B (whole-batch array) of atoms order[0 .. count - 1] from their c and Z terms by position.
template <typename T>
cudaError_t launch_z_descriptors(const DevTables& tb, const DevBatch& b, const BsoParams& p, const int* order, int count,
                                 const void* c, const void* z, T* B, cudaStream_t st);
template <typename T>
cudaError_t launch_lane_z(const DevTables& tb, int nch, int count, const void* c, void* z, cudaStream_t st);

// Evaluation with fitted weights (bispectrum_eval.cu): per-pair forces and per-atom stress of
// dE/dB_a (beta_a = w_lin for the linear model; w_lin + (W + W^T) B_a for the quadratic one),
// gathered into E/F/S by launch_eval_gather.
template <typename T>
struct DevEval {
  const void* c = nullptr;       // c of every atom (A x nch x HU complex of T)
  const void* y = nullptr;       // linear model: y of every atom, as c; the kernel writes Eatom
  double w0 = 0.0;
  const T* gamma = nullptr;      // quadratic model: pair-block weights, nch * NBLKP per atom
  const void* z = nullptr;       // quadratic model: Z terms by queue position (launch_lane_z)
  T* pair = nullptr;             // P x 3: the pair's force contribution
  double* Satom = nullptr;       // A x 6: sum over the atom's pairs of the stress products (xx yy zz yz xz xy)
  double* Eatom = nullptr;       // A: energy of each atom (written for the linear model)
  double* part = nullptr;        // eval_part_doubles: sums over parts of large structures
};

// Descriptor kernel (bispectrum.cu): B (A x nch*K) and w_ch * dB (P x 3 x nch*K) of the batch.  Atoms are taken in `order` (null: index order) through `counter` (one int
// of device memory, reset by the launch).
template <typename T>
cudaError_t launch_bso4(const DevTables& tb, const DevBatch& b, const BsoParams& p, T* Bout, T* dBout,
                        const int* order, int* counter, cudaStream_t st, void* yscratch = nullptr,
                        size_t yscratch_bytes = 0, const Bso4Launch* shape = nullptr);
// Evaluation kernel (bispectrum_eval.cu) of the batch.
template <typename T>
cudaError_t launch_bso4_eval(const DevTables& tb, const DevBatch& b, const BsoParams& p, const DevEval<T>& ev,
                             const int* order, int count, int* counter, cudaStream_t st);
// Linear design rows of the batch from B, w_ch * dB and the reverse pairs (rows.cu); Sp is a
// workspace of A x 6 x KK stress partials.  Columns [1, 1 + KK) of the energy, force and stress
// rows are written.
template <typename T>
cudaError_t launch_lin_rows(const DevBatch& b, const DevRows& rows, const BsoParams& p, int KK, const int* rev,
                            const T* B, const T* dB, T* Sp, T* X, cudaStream_t st);
// E (S), F (3A) and S (6S) from the atoms' energies and stresses and the pairs' forces of evaluation.
size_t eval_part_doubles(int A, int S);
// max_atoms: atoms of the largest structure
template <typename T>
cudaError_t launch_eval_gather(const DevBatch& b, const BsoParams& p, const int* rev, const DevEval<T>& ev,
                               int max_atoms, double* E,
                               double* F, double* S, cudaStream_t st);
// Atoms ordered by descending neighbour count (the descriptor kernel's queue); tmp holds
// atom_order_tmp_ints(maxnn) ints.
size_t atom_order_tmp_ints(int maxnn);
cudaError_t launch_atom_order(const int* nn, int A, int maxnn, int* order, int* tmp, cudaStream_t st);
// The pair-block weights gamma (nch * NBLKP per atom) of beta_a = w_lin + Wsym B_a and the energies
// Eatom_a = w0 + B_a . (beta_a + w_lin) / 2 (eval.cu).  wsym32: Wsym as double-FP32 pairs
// (launch_split_pairs), for T = float.
template <typename T>
cudaError_t launch_eval_gamma(const DevTables& tb, const T* B, int A, int nch, const double* wlin, const double* wsym,
                              const float2* wsym32, double w0, T* gamma, double* Eatom, cudaStream_t st);
// The pair-block weights (nch * NBLKP) of beta = w_lin: FP64, or double-FP32 pairs for T = float.
template <typename T>
cudaError_t launch_block_weights(const DevTables& tb, int nch, const double* wlin, void* gamma, cudaStream_t st);
cudaError_t launch_split_pairs(const double* in, float2* out, size_t n, cudaStream_t st);

// FP64 Gram and rhs on the CUDA cores; with ws (gram_workspace_doubles(M, D) doubles) the
// row-chunk partials are summed in a fixed order (bitwise reproducible), else with atomics
size_t gram_workspace_doubles(long long M, int D);
template <typename T>
cudaError_t launch_gram(const T* X, int ldx, const double* w, const double* y, long long M, int D, double* G,
                        double* h, cudaStream_t st, double* ws = nullptr);
cudaError_t launch_solve_sym(double* G, const double* h, int D, double lambda, double rcond, double* wout,
                             double* evals, int* info, cudaStream_t st);
template <typename T>
cudaError_t launch_rhs(const T* X, int ldx, const double* w, const double* y, long long M, int D, double* h,
                       int nsm, cudaStream_t st, float2* sv, double* ws = nullptr);
cudaError_t launch_symmetrize(double* G, int D, cudaStream_t st);
// ws: at least kSumsqBlocks doubles (per-block partials, added in block order)
constexpr int kSumsqBlocksMax = 1024;
cudaError_t launch_weighted_sumsq(const double* w, const double* y, long long M, double* out, double* ws,
                                  cudaStream_t st);
cudaError_t launch_split_weights(const double* w, long long M, float2* wds, cudaStream_t st);
// ws: normal_matvec_workspace_doubles(M, D, nsm) doubles for the per-block partial column sums,
// reduced in block order (null: FP64 atomics, order not fixed)
size_t normal_matvec_workspace_doubles(long long M, int D, int nsm);
cudaError_t launch_normal_matvec(const float* X, int ldx, int c0, int D, const double* w, const double* p, long long M,
                                 double lambda, float2* sv, double* q, double* ws, int nsm, cudaStream_t st,
                                 int* launches, int* err);
// doubles of the squared-error buffer of launch_predict_sq (3 sums, 3 counts, per-CTA partials)
size_t predict_sq_doubles();
template <typename T>
cudaError_t launch_predict_sq(const T* X, int ldx, const double* w, long long M, int D, double* pred, const double* y,
                              const int* kind, double* sq, cudaStream_t st);
template <typename T>
cudaError_t launch_rows_prep(int S, const int* atom_start, const DevRows& rows, const double* E, const double* F,
                             const double* Sv, const double* wefs, T* X, double* y, double* wrow, int* kind,
                             cudaStream_t st);
template <typename T>
cudaError_t launch_quad_rows(const DevBatch& b, const DevRows& rows, const BsoParams& p, int KK, const int* rev,
                             const T* B, const T* dB, T* H, T* X, int qoff, cudaStream_t st);
cudaError_t launch_reverse_pairs(const DevBatch& b, int* rev, cudaStream_t st);

// dense FP64 factorisation / solves (solve.cu)
// ds_update: trailing updates in double-FP32 on the FP32 pipe (preconditioner factors)
cudaError_t launch_cholesky(double* A, int D, double shift, int* info, cudaStream_t st, bool ds_update = false);
cudaError_t launch_chol_solve(const double* L, int D, const double* b, double* x, cudaStream_t st);
cudaError_t launch_chol_solve_blocked(const double* L, int D, const double* b, double* x, double* tmp,
                                      cudaStream_t st);
inline int chol_solve_launches(int D) { return 2 * ((D + 63) / 64); }
cudaError_t launch_cholesky_inverse(const double* L, int D, double* R, double* Rt, cudaStream_t st, int* launches);
cudaError_t launch_precond_apply(const double* R, const double* Rt, int D, const double* r, double* z, double* tmp,
                                 cudaStream_t st);
inline int cholesky_launches(int D) { return 3 * ((D + 31) / 32) - 2; }

// FP32 inverse of a wide block's preconditioner factor (precond32.cu)
size_t precond32_workspace_bytes(int D);
cudaError_t launch_precond32_from_factor(const double* Lf, int D, void* ws, cudaStream_t st, int* launches);
cudaError_t launch_precond32_apply(const void* ws, int D, const double* r, double* z, double* tmp, cudaStream_t st);
cudaError_t launch_residual(const double* G, int D, double lambda, const double* w, const double* h, double* r,
                            cudaStream_t st);
cudaError_t launch_axpy(int n, double a, const double* x, double* y, cudaStream_t st);
cudaError_t launch_shift_diag_rel(double* A, int D, double lambda, double rel, cudaStream_t st);
cudaError_t launch_pcg_alpha(int D, const double* p, const double* q, double* x, double* r, double* scal,
                             cudaStream_t st);
cudaError_t launch_pcg_beta(int D, const double* z, const double* r, double* p, double* scal, int first,
                            cudaStream_t st);

// kernel ridge regression rows (kernel_rows.cu)
size_t krr_workspace_elems(int A, int nk, int KK);
template <typename T>
cudaError_t launch_krr_rows(const DevBatch& b, const DevRows& rows, const int* rev, const T* Bq, const T* dBq,
                            const T* Z, int nk, int KK, double power, double length, double sigma,
                            double sign_stress, double sign_big, T* ws, T* X, int c0, cudaStream_t st,
                            int* launches, void* tcws = nullptr, size_t tcws_bytes = 0, int* err = nullptr,
                            int nsm = 0);
// kernel-block force rows on the tensor cores (krr_tc.cu); the workspace that holds all `atoms`
// (maxnv derivative vectors at most) in one chunk
// sketched preconditioner of wide mixed blocks (sketch.cu)
constexpr int kSketchZeta = 8;
struct SketchParams {
  int zeta;        // signed copies of each row of X
  int s;           // sketch rows
  long long M;     // rows of X
  uint64_t seed;   // signs
  long long a[kSketchZeta], ainv[kSketchZeta], b[kSketchZeta];  // affine permutations of the rows
};
SketchParams sketch_params(long long M, int D, uint64_t seed);
size_t sketch_workspace_bytes(long long M, int D);
// G (D x D, FP64, full) = Y^T Y of the sketch Y = S W^1/2 X[:, c0 : c0 + D]
cudaError_t launch_sketch_gram(const float* X, int ldx, int c0, int D, const double* w, long long M,
                               const SketchParams& P, void* ws, double* G, cudaStream_t st, int* launches);
constexpr int kKrrTcMaxK = 192;  // three K blocks of 64 in shared memory
bool krr_force_tc_available();
size_t krr_force_tc_workspace_bytes(long long atoms, int maxnv, int nk, int KK);
cudaError_t launch_krr_force_tc(const DevBatch& b, const DevRows& rows, const int* rev, const float* Bq,
                                const float* dBq, const float* Z, const float* F, const float* at, const float* szz,
                                const float* Ts, const float* tx, double sign_stress, int nk, int KK, double power,
                                double length, double sigma, void* ws, size_t ws_bytes, float* X, int c0, int* err,
                                int nsm, cudaStream_t st, int* launches);

// tensor-core Gram in BF16 split precision (gram_tc.cu)
size_t gram_tc_min_workspace(int D);
// doubles of the per-split partial tiles launch_gram_tc needs for a deterministic sum (0: none)
size_t gram_tc_part_doubles(int D, int nsm);
void gram_tc_test_timeout(int skip_loads, long long wait_limit);
bool gram_tc_available();
template <typename T>
cudaError_t launch_gram_tc(const T* X, int ldx, int c0, int D, const double* w, long long M, double* G, void* ws,
                           size_t ws_bytes, int* err, int nsm, cudaStream_t st, double* part = nullptr,
                           size_t part_doubles = 0);

}  // namespace mld
