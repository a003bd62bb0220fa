#include "block_tables.hpp"

#include <algorithm>
#include <array>
#include <atomic>
#include <map>

#include "gather_table.hpp"
#include "host_parallel.hpp"

namespace hphi {

bool block_tables(const std::vector<BitTerm> &terms, int lo_bits, const std::vector<uint32_t> &l22,
                  const std::vector<SectorBlock> &blk, const std::vector<uint32_t> &low, int64_t dim, bool two_pass,
                  BlockTables *out) {
  BlockTables &T = *out;
  const uint64_t nlo = 1ull << lo_bits, lo_mask = nlo - 1;
  uint32_t max_n = 0;
  for (const SectorBlock &b : blk) max_n = std::max(max_n, b.n);
  if (max_n + 16 > 12896) return false;
  // classes, longest blocks first; block lists by class; each lower half's class and position
  std::map<uint32_t, std::vector<int>> by_low;
  for (size_t b = 0; b < blk.size(); b++) by_low[blk[b].low0].push_back((int)b);
  std::vector<uint32_t> order_c;
  for (const auto &kv : by_low) order_c.push_back(kv.first);
  std::stable_sort(order_c.begin(), order_c.end(),
                   [&](uint32_t x, uint32_t y) { return blk[by_low[x][0]].n > blk[by_low[y][0]].n; });
  std::vector<int> cls_of(nlo, -1), pos_of(nlo, -1);
  std::vector<BkClass> &cls = T.cls;
  std::vector<uint32_t> b_ib, &b_row0 = T.b_row0;
  for (size_t c = 0; c < order_c.size(); c++) {
    const std::vector<int> &bl = by_low[order_c[c]];
    BkClass k{};
    k.n = (int)blk[bl[0]].n;
    k.nblk = (int)bl.size();
    k.boff = (int)b_ib.size();
    k.uoff = (int)order_c[c];
    for (int p = 0; p < k.n; p++) {
      const uint32_t ia = low[k.uoff + p];
      if (cls_of[ia] >= 0) return false;  // classes that share lower halves: not this layout
      cls_of[ia] = (int)c;
      pos_of[ia] = p;
    }
    for (int b : bl) {
      b_ib.push_back(blk[b].ib);
      b_row0.push_back(blk[b].row0);
    }
    cls.push_back(k);
  }
  // lower-half terms by coefficient up to sign
  struct LoTerm {
    const BitTerm *t;
    bool neg;
  };
  std::vector<std::vector<LoTerm>> lo;  // by group
  std::vector<double2> &cf = T.cf;
  // upper-half and crossing terms, in bits of the upper half; a crossing term's lower-half pattern
  // (condition, flip, sign) is a table of source positions per class
  struct HiTerm {
    uint32_t cm, cv, flip, sm;
    int pat;  // lower-half pattern, -1: upper-half term
    double re, im;
  };
  std::vector<HiTerm> hi;
  std::vector<std::array<uint32_t, 4>> pats;
  for (const BitTerm &t : terms) {
    const uint64_t all = t.cm | t.flip | t.sm;
    if ((all & ~lo_mask) == 0) {
      size_t g = 0;
      bool neg = false;
      for (; g < cf.size(); g++) {
        if (t.re == cf[g].x && t.im == cf[g].y) break;
        if (t.re == -cf[g].x && t.im == -cf[g].y) { neg = true; break; }
      }
      if (g == cf.size()) {
        if (g == (size_t)kBkGroups) return false;
        cf.push_back(make_double2(t.re, t.im));
        lo.emplace_back();
      }
      lo[g].push_back(LoTerm{&t, neg});
      continue;
    }
    HiTerm h{(uint32_t)(t.cm >> lo_bits), (uint32_t)(t.cv >> lo_bits), (uint32_t)(t.flip >> lo_bits),
             (uint32_t)(t.sm >> lo_bits), -1, t.re, t.im};
    if ((all & lo_mask) != 0) {
      const std::array<uint32_t, 4> pt{(uint32_t)(t.cm & lo_mask), (uint32_t)(t.cv & lo_mask), (uint32_t)(t.flip & lo_mask),
                                       (uint32_t)(t.sm & lo_mask)};
      h.pat = (int)(std::find(pats.begin(), pats.end(), pt) - pats.begin());
      if (h.pat == (int)pats.size()) pats.push_back(pt);
      if (pats.size() > 4 * (size_t)kBkCross) return false;
    }
    hi.push_back(h);
  }
  const size_t np = pats.size();
  std::vector<uint16_t> &tab = T.tab;
  std::vector<uint32_t> tab_at(cls.size() * std::max<size_t>(1, np), 0);
  std::vector<int> tab_to(tab_at.size(), -1);  // the class the pattern leads to: one for all its positions
  for (size_t c = 0; c < cls.size(); c++)
    for (size_t q = 0; q < np; q++) {
      tab_at[c * np + q] = (uint32_t)tab.size();
      int &to = tab_to[c * np + q];
      for (int p = 0; p < cls[c].n; p++) {
        const uint32_t ia = low[cls[c].uoff + p], src = ia ^ pats[q][2];
        uint16_t v = (uint16_t)kBkNone;
        if ((ia & pats[q][0]) == pats[q][1] && cls_of[src] >= 0) {
          if (to < 0) to = cls_of[src];
          if (cls_of[src] != to) return false;
          v = (uint16_t)((uint32_t)pos_of[src] | ((__builtin_popcount(ia & pats[q][3]) & 1) ? 0x8000u : 0u));
        }
        tab.push_back(v);
      }
    }
  // per block the upper-half and crossing terms that act on it
  std::vector<int> class_of_block(l22.size(), -1);
  for (size_t c = 0; c < cls.size(); c++)
    for (int b = 0; b < cls[c].nblk; b++) class_of_block[b_ib[cls[c].boff + b]] = (int)c;
  std::vector<uint2> &b_list = T.b_list;
  b_list.resize(b_ib.size());
  std::vector<uint64_t> ib_sorted(b_ib.size());
  std::vector<BkRec> &rec = T.rec;
  std::vector<double> &rec_im = T.rec_im;
  for (const HiTerm &h : hi) T.im = T.im || (h.im != 0.0 && !(two_pass && h.pat < 0));
  std::stable_sort(hi.begin(), hi.end(), [](const HiTerm &x, const HiTerm &y) { return (x.pat >= 0) < (y.pat >= 0); });
  const size_t n_up = std::find_if(hi.begin(), hi.end(), [](const HiTerm &h) { return h.pat >= 0; }) - hi.begin();
  struct List {  // a block's records, upper-half terms first
    const BkRec *rec;
    const double *im;
    uint32_t nh, nx;
  };
  const uint32_t longest = two_pass ? kBkListRows : kBkList;
  constexpr int kRun = 64;  // blocks of a piece
  struct Run {
    std::vector<BkRec> rec;
    std::vector<double> im;
  };
  std::vector<Run> runs((b_ib.size() + kRun - 1) / kRun);
  std::vector<List> lists(b_ib.size());
  const int ng = (int)cf.size();
  struct Warp {
    int cls, warp;
    std::vector<std::vector<uint16_t>> code;  // by group
    std::vector<int> slots;
  };
  std::vector<Warp> warps;
  for (size_t c = 0; c < cls.size(); c++)
    for (int w = 0; w < (cls[c].n + 31) / 32; w++) warps.push_back(Warp{(int)c, w, {}, {}});
  std::atomic<bool> fits{true};
  auto list_run = [&](size_t u) {
    Run &r = runs[u];
    r.rec.reserve((size_t)kRun * std::min<size_t>(hi.size(), longest));
    const size_t q0 = (size_t)u * kRun, q1 = std::min(b_ib.size(), q0 + kRun);
    for (size_t q = q0; q < q1 && fits; q++) {
      const uint32_t ib = b_ib[q];
      const int c = class_of_block[ib];
      List &l = lists[q];
      l.nh = l.nx = 0;
      for (size_t k = two_pass ? n_up : 0; k < hi.size(); k++) {
        const HiTerm &h = hi[k];
        if ((ib & h.cm) != h.cv) continue;
        const uint32_t to = ib ^ h.flip;
        if (l22[to] == 0) continue;
        const bool cross = h.pat >= 0;
        const int lead = cross ? tab_to[c * np + h.pat] : c;  // a moved block keeps its lower halves
        if (lead < 0) continue;                               // no row of the class matches
        if (class_of_block[to] != lead) fits = false;
        const bool neg = h.sm && (__builtin_popcount(ib & h.sm) & 1);
        r.rec.push_back(BkRec{l22[to] - 1u, cross ? tab_at[c * np + h.pat] : 0u, neg ? -h.re : h.re});
        if (T.im) r.im.push_back(neg ? -h.im : h.im);
        (cross ? l.nx : l.nh)++;
      }
      if (l.nh + l.nx > longest) fits = false;
    }
    size_t at = 0;  // the run's vectors do not move any more
    for (size_t q = q0; q < q1; at += lists[q].nh + lists[q].nx, q++) {
      lists[q].rec = r.rec.data() + at;
      lists[q].im = T.im ? r.im.data() + at : nullptr;
    }
  };
  auto gather = [&](Warp &w) {
    std::vector<uint32_t> ptr, ent;
    const BkClass &k = cls[w.cls];
    w.code.resize(ng);
    for (int g = 0; g < ng; g++) {
      ptr.assign(1, 0);
      ent.clear();
      for (int p = 32 * w.warp; p < 32 * (w.warp + 1); p++) {
        const uint32_t ia = p < k.n ? low[k.uoff + p] : 0;
        for (const LoTerm &t : lo[g]) {
          if (p >= k.n || (ia & t.t->cm) != t.t->cv) continue;
          const uint32_t src = ia ^ (uint32_t)t.t->flip;
          if (cls_of[src] < 0) continue;  // list_2_1 == 0: outside the sector
          if (cls_of[src] != w.cls) fits = false;
          const bool neg = (t.t->sm && (__builtin_popcount(ia & (uint32_t)t.t->sm) & 1)) != t.neg;
          ent.push_back((uint32_t)pos_of[src] | (neg ? 0x10000u : 0u));
        }
        ptr.push_back((uint32_t)ent.size());
      }
      w.slots.push_back(gather_warp(ptr.data(), ent.data(), k.n, &w.code[g]));
    }
  };
  // lists first: their limits decline without the gather tables.  ~6 ns per block and term, 500 per
  // warp and lower-half term (up to 32 entries, about half of them there)
  size_t n_lo = 0;
  for (const auto &g : lo) n_lo += g.size();
  host_parallel((int64_t)(runs.size() + warps.size()), 0.006 * (double)(b_ib.size() * hi.size()) + 0.5 * (double)(warps.size() * n_lo),
                [&](int64_t k) {
                  if (!fits) return;
                  if (k < (int64_t)runs.size()) list_run((size_t)k);
                  else gather(warps[k - runs.size()]);
                });
  if (!fits) return false;
  size_t total = 0;
  for (const Run &r : runs) total += r.rec.size();
  if (total > (1u << 26)) return false;
  rec.reserve(total);
  std::vector<uint32_t> r0;
  std::vector<std::pair<uint64_t, int>> order;
  for (const BkClass &k : cls) {
    order.clear();
    for (int b = 0; b < k.nblk; b++) {
      const List &l = lists[k.boff + b];
      order.push_back({((uint64_t)l.nh << 32) | (l.nh + l.nx), b});
    }
    std::stable_sort(order.begin(), order.end());  // blocks of equal list lengths side by side
    r0.resize(k.nblk);
    for (int b = 0; b < k.nblk; b++) {
      r0[b] = b_row0[k.boff + order[b].second];
      ib_sorted[k.boff + b] = b_ib[k.boff + order[b].second];
    }
    for (int b = 0; b < k.nblk; b++) {
      const List &l = lists[k.boff + order[b].second];
      b_row0[k.boff + b] = r0[b];
      b_list[k.boff + b] = make_uint2((uint32_t)rec.size(), l.nh | (l.nx << 16));
      rec.insert(rec.end(), l.rec, l.rec + l.nh + l.nx);
      if (T.im) rec_im.insert(rec_im.end(), l.im, l.im + l.nh + l.nx);
    }
  }
  // one table per class: a warp's sets, group after group, at a fixed stride (with one set past
  // the last, read ahead), so that the first set's address does not wait for the slot counts
  std::vector<uint4> &gat = T.gat;
  std::vector<uint2> &head = T.head;
  for (const Warp &w : warps) {
    int n = 1;
    for (int ns : w.slots) {
      if (ns > 255) return false;  // counts are packed in 8 bits
      n += (ns + 7) / 8;
    }
    cls[w.cls].sets = std::max(cls[w.cls].sets, n);
  }
  for (const Warp &w : warps) {
    BkClass &k = cls[w.cls];
    if (w.warp == 0) {
      k.gat = (int)gat.size();
      k.head = (int)head.size();
    }
    uint64_t cnt = 0;
    for (int g = 0; g < ng; g++) {
      cnt |= (uint64_t)w.slots[g] << (8 * g);
      for (int j = 0; j < w.slots[g]; j += 8)
        for (int lane = 0; lane < 32; lane++) {
          const GatherSet s = gather_set(w.code[g], j, lane);
          gat.push_back(make_uint4(s.w[0], s.w[1], s.w[2], s.w[3]));
        }
    }
    gat.resize((size_t)k.gat + (size_t)(w.warp + 1) * k.sets * 32, make_uint4(0, 0, 0, 0));
    head.push_back(make_uint2((uint32_t)cnt, (uint32_t)(cnt >> 32)));
  }
  double mean = 0.0;  // block length a row sees on average
  for (const SectorBlock &b : blk) mean += (double)b.n * b.n / (double)dim;
  for (int id = kBkShapes - 1; id >= 0; id--)
    if ((int)max_n + 16 <= kBkShapeDefs[id].stride && !(id == 2 && mean >= kBkLong)) T.shape = id;
  // Pairs of blocks of one class (complex vectors: single blocks).  Where v1 exceeds
  // L2 (two_pass), blocks whose upper halves differ only in bits that crossing terms flip read
  // each other's rows, so they come together and a group's source blocks are read while in L2;
  // else class by class, the longest first.
  uint64_t xhi = 0;
  for (const HiTerm &h : hi)
    if (h.pat >= 0) xhi |= h.flip;
  for (size_t c = 0; c < cls.size(); c++)
    for (int b = 0; b < cls[c].nblk; b++)
      T.order.push_back({two_pass ? ib_sorted[cls[c].boff + b] & ~xhi : 0, (uint32_t)c, (uint32_t)(cls[c].boff + b)});
  std::stable_sort(T.order.begin(), T.order.end(), [](const BlockTables::Place &x, const BlockTables::Place &y) {
    return x.group != y.group ? x.group < y.group : x.cls < y.cls;
  });
  // room for what the kernel's walk over the crossing terms reads: whole steps of U terms up to the
  // longest list of the task, after each block's own upper-half terms
  const uint32_t U = (uint32_t)kBkShapeDefs[T.shape].U;
  auto room = [&](uint2 own, uint2 other) {
    const uint32_t nx = std::max(own.y >> 16, other.y >> 16);
    return (own.y & 0xFFFFu) + (nx + U - 1) / U * U;
  };
  uint32_t nlist = 1;
  for (size_t q = 0; q < T.order.size(); q++) {
    const uint2 l = b_list[T.order[q].b];
    nlist = std::max(nlist, room(l, l));
    if (!block_pair(T, q)) continue;
    const uint2 m = b_list[T.order[q + 1].b];
    nlist = std::max({nlist, room(l, m), room(m, l)});
  }
  T.nlist = (int)nlist;
  return true;
}

bool block_pair(const BlockTables &t, size_t q) {
  return q + 1 < t.order.size() && t.order[q + 1].cls == t.order[q].cls && t.order[q + 1].group == t.order[q].group;
}

// Whole blocks, unless they are fewer than kBkWaves tasks per resident CTA: then at most that
// share of the rows each, but no less than one turn of the threads.  us per H*v (real) with whole
// blocks, shares for 2 tasks per CTA, and for 8: 23-site J1-J2 chain 48.7, 42.6, 44.0; 22 sites 30.9,
// 28.8, 28.7; 8-site Kondo 32.5, 29.4, 29.4; spin-1 chain of 14 sites 27.1, 24.5, 24.5.  Where there are
// more blocks the second staging costs more than the even end gives: 24 sites 77.7, 77.7, 81.4.
std::vector<BkTask> block_tasks(const BlockTables &t, bool cplx, int ctas) {
  std::vector<BkTask> tk;
  int64_t total = 0;
  for (const auto &b : t.order) total += t.cls[b.cls].n;
  const BkShapeDef &S = kBkShapeDefs[t.shape];
  const int64_t want = (int64_t)kBkWaves * ctas;
  const int whole = (int)(cplx ? t.order.size() : (t.order.size() + 1) / 2);
  const int share =
      whole >= want ? 1 << 15 : (int)std::max<int64_t>(S.Q * S.threads, (cplx ? total : total / 2) / want);
  for (size_t q = 0; q < t.order.size();) {
    const bool two = !cplx && block_pair(t, q);
    const BlockTables::Place &b = t.order[q];
    const int nw = (t.cls[b.cls].n + 31) / 32, parts = std::min(nw, (32 * nw + share - 1) / share);
    for (int k = 0; k < parts; k++)
      tk.push_back(BkTask{b.cls, b.b, two ? t.order[q + 1].b : ~0u,
                          (uint32_t)(32 * (nw * k / parts)) | ((uint32_t)(32 * (nw * (k + 1) / parts)) << 16)});
    q += two ? 2 : 1;
  }
  return tk;
}

}  // namespace hphi
