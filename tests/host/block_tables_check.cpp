// Checks the block kernel's host tables (block_tables.hpp) of one model against its terms, without
// a device: argv[1] is a namelist.def of a canonical model of at most 24 bits, or "crowded"; with
// "no_memory" as argv[2], whether the plans decline without a device.  Every index the
// kernel would form is compared with the room it has, and H*v put together from the tables, the
// way the kernel does it, with H*v from the terms.  Prints what the tables are like; the exit
// status is 1, with a message, when something is wrong.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <random>

#include "block_tables.hpp"
#include "hv_blocks.hpp"
#include "hv_gc.hpp"

using namespace hphi;
using Z = std::complex<double>;

static void fail(const char *what, long a = 0, long b = 0) {
  printf("%s (%ld, %ld)\n", what, a, b);
  exit(1);
}

// The tables of these terms; row_of: row of a configuration, -1 outside the sector.
static void check(const std::vector<BitTerm> &terms, int lo_bits, const std::vector<uint32_t> &l22,
                  const std::vector<SectorBlock> &blk, const std::vector<uint32_t> &low,
                  const std::vector<uint64_t> &list_1, const std::vector<int64_t> &row_of) {
  const uint64_t lo_mask = (1ull << lo_bits) - 1;
  const int64_t dim = (int64_t)list_1.size();
  std::mt19937_64 rng(5);
  std::normal_distribution<double> gauss;
  std::vector<Z> v(dim);
  for (Z &x : v) x = Z(gauss(rng), gauss(rng));
  for (int two_pass = 0; two_pass < 2; two_pass++) {
    BlockTables t;
    if (!block_tables(terms, lo_bits, l22, blk, low, dim, two_pass != 0, &t)) {
      printf("no plan ");
      continue;
    }
    const BkShapeDef &S = kBkShapeDefs[t.shape];
    // the tasks: every position once, every record inside the room of its block
    int longest = 0;
    for (int cv = 0; cv < 2; cv++)
      for (int ctas : {148, 740, 1480}) {
        std::vector<std::vector<char>> seen(t.b_row0.size());
        for (const BkTask &k : block_tasks(t, cv != 0, ctas)) {
          const int n = t.cls[k.cls].n, npad = (n + 31) / 32 * 32;
          const uint32_t bs[2] = {k.b0, k.b1};
          uint32_t xmax = 0;
          for (uint32_t b : bs)
            if (b != ~0u) {
              if (b < (uint32_t)t.cls[k.cls].boff || b >= (uint32_t)(t.cls[k.cls].boff + t.cls[k.cls].nblk))
                fail("block of another class", b);
              xmax = std::max(xmax, t.b_list[b].y >> 16);
            }
          for (uint32_t b : bs) {
            if (b == ~0u) continue;
            const uint32_t nh = t.b_list[b].y & 0xFFFFu, nx = t.b_list[b].y >> 16;
            longest = std::max(longest, (int)(nh + nx));
            if ((int)(nh + nx) > t.nlist) fail("list longer than its room", nh + nx, t.nlist);
            for (uint32_t i = 0; i < xmax; i += S.U)
              if ((int)(nh + i + S.U) > t.nlist) fail("records read past their room", nh + i + S.U, t.nlist);
            seen[b].resize(npad, 0);
            const uint32_t p0 = k.span & 0xFFFFu, p1 = k.span >> 16;
            if (p0 % 32 || p1 % 32 || (int)p1 > npad) fail("span", p0, p1);
            for (uint32_t p = p0; p < p1; p++)
              if (seen[b][p]++) fail("position done twice", b, p);
          }
        }
        for (size_t b = 0; b < seen.size(); b++) {
          if (seen[b].empty()) fail("block without a task", (long)b);
          for (char c : seen[b])
            if (!c) fail("position left out", (long)b);
        }
      }
    // H*v
    double worst = 0.0, big = 0.0;
    for (size_t c = 0; c < t.cls.size(); c++) {
      const BkClass &C = t.cls[c];
      if (C.n + 16 > S.stride) fail("block longer than a plane", C.n, S.stride);
      for (int b = C.boff; b < C.boff + C.nblk; b++) {
        const Z *x = v.data() + t.b_row0[b];
        for (int p = 0; p < C.n; p++) {
          Z y = 0.0, want = 0.0;
          const uint2 h = t.head[C.head + (p >> 5)];
          size_t at = (size_t)C.gat + (size_t)(p >> 5) * C.sets * 32 + (p & 31);
          for (size_t g = 0; g < t.cf.size(); g++) {
            const int ns = ((g < 4 ? h.x : h.y) >> (8 * (g & 3))) & 255u;
            Z s = 0.0;
            for (int j = 0; j < ns; j += 8, at += 32) {
              const uint32_t w[4] = {t.gat.at(at).x, t.gat.at(at).y, t.gat.at(at).z, t.gat.at(at).w};
              for (int q = 0; q < (j + 4 < ns ? 8 : 4); q++) {
                const uint32_t e = (w[q / 2] >> (16 * (q % 2))) & 0xFFFFu, word = e & 0x7FFFu;
                if ((int)word >= C.n + 16) fail("gather past the plane", word, C.n);
                if ((int)word < C.n) s += (e >> 15 ? -1.0 : 1.0) * x[word];
              }
            }
            y += Z(t.cf[g].x, t.cf[g].y) * s;
          }
          if (at >= t.gat.size()) fail("set read ahead past the table", (long)at);
          const uint2 li = t.b_list[b];
          for (uint32_t k = 0; k < (li.y & 0xFFFFu) + (li.y >> 16); k++) {
            const BkRec &r = t.rec.at(li.x + k);
            const Z cf(r.re, t.im ? t.rec_im.at(li.x + k) : 0.0);
            if (k < (li.y & 0xFFFFu)) {
              y += cf * v.at(r.row + p);
            } else {
              const uint32_t e = t.tab.at(r.tab + p);
              if ((e & 0x7FFFu) != kBkNone) y += (e >> 15 ? -1.0 : 1.0) * cf * v.at(r.row + (e & 0x7FFFu));
            }
          }
          const uint64_t cfg = list_1[t.b_row0[b] + p];
          for (const BitTerm &q : terms) {
            if (two_pass && ((q.cm | q.flip | q.sm) & lo_mask) == 0) continue;
            if ((cfg & q.cm) != q.cv || row_of[cfg ^ q.flip] < 0) continue;
            want += ((__builtin_popcountll(cfg & q.sm) & 1) ? -1.0 : 1.0) * Z(q.re, q.im) * v[row_of[cfg ^ q.flip]];
          }
          worst = std::max(worst, std::abs(y - want));
          big = std::max(big, std::abs(want));
        }
      }
    }
    // a row sums a few hundred products of numbers of order 1 in another order
    if (worst > 1e-13 * std::max(1.0, big)) fail("H*v differs");
    printf("shape %d longest list %d room %d ", t.shape, longest, t.nlist);
  }
}

// One block of 512 rows whose first 16 rows read the same 20 words each, all on one of the 16 bank
// pairs: 320 entries that no two slots of a half-warp can share.
static void crowded() {
  std::vector<BitTerm> terms;
  for (uint64_t r = 0; r < 16; r++)
    for (uint64_t k = 0; k < 20; k++) terms.push_back(BitTerm{511, r, r ^ (32 + 16 * k), 0, 1.0, 0.0});
  std::vector<uint32_t> low;
  std::vector<uint64_t> list_1;
  std::vector<int64_t> row_of(1024, -1);
  for (uint32_t ia = 0; ia < 512; ia++) {
    low.push_back(ia);
    list_1.push_back(ia);
    row_of[ia] = ia;
  }
  check(terms, 9, {1, 0}, {SectorBlock{0, 0, 0, 512}}, low, list_1, row_of);
}

// A plan that cannot have device memory (there is no device) leaves the sector without one: the caller goes
// on with the kernels that need none.
static void no_memory(const char *namelist) {
  Sector s;
  std::string err;
  if (read_expert(namelist, &s.model, &err) != 0) fail(err.c_str());
  s.num_sms = 148;
  s.gc = s.model.rows_are_configs();
  s.lo_bits = (s.model.nbits + 1) / 2;
  s.hi_bits = s.model.nbits - s.lo_bits;
  s.ihfbit = 1ull << s.lo_bits;
  s.sdim = 1ull << s.hi_bits;
  s.dim = sector_dim(s.model);
  std::vector<uint64_t> list_1((size_t)s.dim);
  std::vector<uint32_t> l21(s.ihfbit), l22(s.sdim);
  s.d_list_1 = list_1.data();
  s.d_list_2_1 = l21.data();
  s.d_list_2_2 = l22.data();
  bk_plan_build(&s, false);
  gc_plan_build(&s);
  if (s.bk || s.gcp) fail("a plan without a device");
}

int main(int argc, char **argv) {
  if (argc == 3 && std::string(argv[2]) == "no_memory") {
    no_memory(argv[1]);
    return 0;
  }
  if (argc == 2 && std::string(argv[1]) == "crowded") {
    crowded();
    printf("\n");
    return 0;
  }
  Model m;
  std::string err;
  if (argc < 2 || read_expert(argv[1], &m, &err) != 0) fail(err.c_str());
  const int lo_bits = (m.nbits + 1) / 2, hi_bits = m.nbits - lo_bits;
  const uint64_t lo_mask = (1ull << lo_bits) - 1, even = 0x5555555555555555ull;
  auto in_sector = [&](uint64_t c) {
    if (m.calc_model == kHubbard)
      return __builtin_popcountll(c & even) == m.nup && __builtin_popcountll(c & ~even) == m.ndown;
    return __builtin_popcountll(c) == m.ne;
  };
  // HPhi's rows: by upper half, then lower half
  std::vector<uint64_t> list_1;
  std::vector<uint32_t> l22(1ull << hi_bits, 0), low;
  std::vector<SectorBlock> blk;
  std::map<std::vector<uint32_t>, uint32_t> cls;
  std::vector<int64_t> row_of(1ull << m.nbits, -1);
  for (uint64_t ib = 0; ib < (1ull << hi_bits); ib++) {
    std::vector<uint32_t> mine;
    const uint32_t row0 = (uint32_t)list_1.size();
    for (uint64_t ia = 0; ia <= lo_mask; ia++)
      if (in_sector(ib << lo_bits | ia)) {
        mine.push_back((uint32_t)ia);
        row_of[ib << lo_bits | ia] = (int64_t)list_1.size();
        list_1.push_back(ib << lo_bits | ia);
      }
    if (mine.empty()) continue;
    l22[ib] = row0 + 1;
    const auto it = cls.emplace(mine, (uint32_t)low.size());
    if (it.second) low.insert(low.end(), mine.begin(), mine.end());
    blk.push_back(SectorBlock{(uint32_t)ib, row0, it.first->second, (uint32_t)mine.size()});
  }
  check(m.offdiag, lo_bits, l22, blk, low, list_1, row_of);
  printf("\n");
  return 0;
}
