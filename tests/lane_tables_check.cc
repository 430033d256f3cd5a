// Invariants of the host-built tables that the atoms-on-lanes kernels, the Y rows and the derivatives
// rely on without checking them: indices of c, coefficients, blocks and terms in range, every term of a
// pair block formed exactly once, every output of a job written once, jobs covering their records.
// Built and run by tests/test_lane_tables.py (host code only; no GPU).  Prints "ok <j_max>" and the sizes
// that the work model counts, or the first failure and exits 1.
#include <cstdio>
#include <cstdlib>
#include <set>
#include <string>
#include <vector>

#include "../mld_gb300/csrc/mld_internal.h"

using namespace mld;

static int fail(double jm, const std::string& what) {
  std::printf("FAIL j_max=%.1f: %s\n", jm, what.c_str());
  return 1;
}

static int check(double jm) {
  Bso4Tables t;
  std::string err;
  if (!build_bso4_tables(jm, &t, &err)) return fail(jm, "build: " + err);
  auto H = [&](int j) { return t.hoff[j + 1] - t.hoff[j]; };
  const int no = t.J / 2 + 1;
  // --- records: first and last operands inside c, coefficients inside their table
  auto records = [&](const std::vector<LaneRec>& recs, const char* name) {
    for (const LaneRec& r : recs) {
      if (r.na < 1 || r.nb < 1 || r.nj < 1 || r.nj > no || r.nj > kMaxZOut) return fail(jm, std::string(name) + ": extents");
      const int hi = r.i1 + (r.na - 1) * r.s1 + r.nb - 1, lo = r.i2 - (r.na - 1) * r.s2 - (r.nb - 1);
      if (hi >= t.NU || lo < 0 || r.i2 >= t.NU) return fail(jm, std::string(name) + ": c index");
      if (r.cg1 + (r.na - 1) * r.st1 + r.nj > (int)t.cgv.size() || r.cg2 + (r.nb - 1) * r.st2 + r.nj > (int)t.cgv.size())
        return fail(jm, std::string(name) + ": coefficient");
      if (r.nj > r.st1 || r.nj > r.st2) return fail(jm, std::string(name) + ": more layers than coefficients of an entry");
    }
    return 0;
  };
  if (records(t.brecs, "B") || records(t.yrecs, "y") || records(t.zrecs, "z")) return 1;
  if (t.zrecs.size() != t.yrecs.size()) return fail(jm, "z records are not the y records");
  // --- jobs: four parts each, one after the other, covering the records
  auto jobs = [&](const std::vector<LaneJob>& jobs, size_t nrec, const char* name) {
    size_t at = 0;
    for (const LaneJob& j : jobs) {
      if (j.rec[0] != (int)at || j.nout > no) return fail(jm, std::string(name) + " job start or outputs");
      for (int q = 0; q < 4; ++q)
        if (j.rec[q] > j.rec[q + 1]) return fail(jm, std::string(name) + " job parts");
      at = j.rec[4];
    }
    return at == nrec ? 0 : fail(jm, std::string(name) + " jobs do not cover the records");
  };
  if (jobs(t.bjobs, t.brecs.size(), "B") || jobs(t.yjobs, t.yrecs.size(), "y")) return 1;
  // --- outputs
  std::set<int> k_seen, y_seen;
  long long products = 0, sums = 0;
  std::vector<int> z_seen(t.nztp, 0);
  for (const LaneJob& j : t.bjobs) {
    for (int o = 0; o < j.nout; ++o)
      if (j.out[o] >= t.K || !k_seen.insert(j.out[o]).second) return fail(jm, "B output out of range or repeated");
    for (int r = j.rec[0]; r < j.rec[4]; ++r) {
      if (t.brecs[r].nj > j.nout || t.brecs[r].w < 1 || t.brecs[r].w > 2) return fail(jm, "B record's outputs or weight");
      for (int o = 0; o < t.brecs[r].nj; ++o)
        if (t.brecs[r].out[o] >= t.NU) return fail(jm, "B record's c index");
    }
  }
  if ((int)k_seen.size() != t.K) return fail(jm, "a triple without a job");
  for (const LaneJob& j : t.yjobs) {
    for (int o = 0; o < j.nout; ++o)
      if (j.out[o] >= t.HU || !y_seen.insert(j.out[o]).second) return fail(jm, "y output out of range or repeated");
    for (int r = j.rec[0]; r < j.rec[4]; ++r) {
      const LaneRec &y = t.yrecs[r], &z = t.zrecs[r];
      if (y.off + y.nj > j.nout) return fail(jm, "y record beyond its job's outputs");
      for (int o = 0; o < y.nj; ++o) {
        if (y.out[o] >= t.nblk_pair) return fail(jm, "y record's block");
        if (z.out[o] >= t.nztp) return fail(jm, "z record's term");
        z_seen[z.out[o]]++;
      }
      products += y.na * y.nb;
      sums += (long long)y.nj * (y.na * y.nb + y.na);
    }
  }
  if ((int)y_seen.size() != t.HU) return fail(jm, "a half entry without a y job");
  for (int n : z_seen)
    if (n != 1) return fail(jm, "term not formed exactly once");
  // --- block weights, triples and rows on the terms
  if ((int)t.gamp_off.size() != t.nblk_pair + 1 || t.gamp_off[0] != 0 || t.gamp_off.back() != (int)t.gamp.size())
    return fail(jm, "block weight offsets");
  for (const GammaItem& g : t.gamp)
    if (g.k >= t.K || g.snum < 1 || g.sden < 1) return fail(jm, "block weight item");
  if ((int)t.trzp.size() != t.K || t.rowsrc2.size() != t.rowk.size()) return fail(jm, "triples or rows");
  for (const TripleZ& z : t.trzp)
    if (z.l > t.J || z.za + H(z.l) > t.nztp) return fail(jm, "triple's terms out of range");
  long long row_entries = 0, row_terms = 0;
  for (int j = 0; j <= t.J; ++j)
    for (int r = 0; r < t.Mp[j]; ++r) {
      const RowSource& s = t.rowsrc2[t.rowk_off[j] + r];
      if (s.nterm > 3 || (s.nterm == 0) != (t.rowk[t.rowk_off[j] + r] < 0)) return fail(jm, "row terms");
      for (int n = 0; n < s.nterm; ++n)
        if (s.z[n] + H(j) > t.nztp || s.snum[n] < 1 || s.sden[n] < 1 || s.snum[n] > kMaxJ + 1 || s.sden[n] > kMaxJ + 1)
          return fail(jm, "row source out of range");
      if (s.nterm) row_entries += H(j);
      row_terms += (long long)s.nterm * H(j);
    }
  std::printf("ok %.1f products=%lld sums=%lld row_entries=%lld row_terms=%lld\n", jm, products, sums, row_entries, row_terms);
  return 0;
}

int main(int argc, char** argv) {
  int bad = 0;
  for (int i = 1; i < argc; ++i) bad |= check(std::atof(argv[i]));
  return bad;
}
