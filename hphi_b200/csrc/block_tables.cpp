#include "block_tables.hpp"

#include <algorithm>
#include <array>
#include <map>

#include "hv_product.hpp"

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
    int group;
    bool neg;
  };
  std::vector<LoTerm> lo;
  std::vector<double2> &cf = T.cf;
  for (const BitTerm &t : terms) {
    if (((t.cm | t.flip | t.sm) & ~lo_mask) != 0) continue;
    int g = 0;
    bool neg = false;
    for (; g < (int)cf.size(); g++) {
      if (t.re == cf[g].x && t.im == cf[g].y) break;
      if (t.re == -cf[g].x && t.im == -cf[g].y) { neg = true; break; }
    }
    if (g == (int)cf.size()) {
      if (g == kBkGroups) return false;
      cf.push_back(make_double2(t.re, t.im));
    }
    lo.push_back(LoTerm{&t, g, neg});
  }
  std::vector<uint4> &gat = T.gat;
  std::vector<uint2> &head = T.head;
  const int ng = (int)cf.size();
  for (size_t c = 0; c < cls.size(); c++) {
    BkClass &k = cls[c];
    std::vector<std::vector<std::vector<uint32_t>>> tab(ng, std::vector<std::vector<uint32_t>>(k.n));
    for (int p = 0; p < k.n; p++) {
      const uint32_t ia = low[k.uoff + p];
      for (const LoTerm &t : lo) {
        if ((ia & t.t->cm) != t.t->cv) continue;
        const uint32_t src = ia ^ (uint32_t)t.t->flip;
        if (cls_of[src] < 0) continue;  // list_2_1 == 0: outside the sector
        if (cls_of[src] != (int)c) return false;
        const bool neg = ((__builtin_popcountll((uint64_t)ia & t.t->sm) & 1) != 0) != t.neg;
        tab[t.group][p].push_back((uint32_t)pos_of[src] | (neg ? 0x10000u : 0u));
        if (tab[t.group][p].size() > 255) return false;
      }
    }
    // one table per class: a warp's sets, group after group, at a fixed stride (with one set past
    // the last, read ahead), so that the first set's address does not wait for the slot counts
    const int nw = (k.n + 31) / 32;
    std::vector<std::vector<uint32_t>> t(ng);
    std::vector<std::vector<uint8_t>> ws(ng);
    std::vector<int> gs(ng, 1);
    k.sets = 1;
    for (int g = 0; g < ng; g++)
      if (!build_gather_table(tab[g], k.n, &t[g], &ws[g], &gs[g])) return false;
    for (int w = 0; w < nw; w++) {
      int n = 1;
      for (int g = 0; g < ng; g++) n += (ws[g][w] + 7) / 8;
      k.sets = std::max(k.sets, n);
    }
    k.gat = (int)gat.size();
    k.head = (int)head.size();
    gat.resize(gat.size() + (size_t)nw * k.sets * 32, make_uint4(0, 0, 0, 0));
    for (int w = 0; w < nw; w++) {
      size_t at = (size_t)k.gat + (size_t)w * k.sets * 32;
      uint64_t cnt = 0;
      for (int g = 0; g < ng; g++) {
        cnt |= (uint64_t)ws[g][w] << (8 * g);
        const uint32_t *src = &t[g][(size_t)w * gs[g] * 128];
        for (int i = 0; i < (ws[g][w] + 7) / 8 * 32; i++, at++)
          gat[at] = make_uint4(src[4 * i], src[4 * i + 1], src[4 * i + 2], src[4 * i + 3]);
      }
      head.push_back(make_uint2((uint32_t)cnt, (uint32_t)(cnt >> 32)));
    }
  }
  // per block the upper-half and crossing terms that act on it; a crossing term's lower-half
  // pattern (condition, flip, sign) is a table of source positions per class
  struct HiTerm {
    const BitTerm *t;
    int pat;  // lower-half pattern, -1: upper-half term
  };
  std::vector<HiTerm> hi;
  std::vector<std::array<uint32_t, 4>> pats;
  for (const BitTerm &t : terms) {
    if (((t.cm | t.flip | t.sm) & ~lo_mask) == 0) continue;  // lower half
    HiTerm h{&t, -1};
    if (((t.cm | t.flip | t.sm) & lo_mask) != 0) {
      const std::array<uint32_t, 4> pt{(uint32_t)(t.cm & lo_mask), (uint32_t)(t.cv & lo_mask), (uint32_t)(t.flip & lo_mask),
                                       (uint32_t)(t.sm & lo_mask)};
      h.pat = (int)(std::find(pats.begin(), pats.end(), pt) - pats.begin());
      if (h.pat == (int)pats.size()) pats.push_back(pt);
    }
    hi.push_back(h);
  }
  if (pats.size() > 4 * (size_t)kBkCross) return false;
  std::vector<uint16_t> &tab = T.tab;
  std::vector<uint32_t> tab_at(cls.size() * std::max<size_t>(1, pats.size()), 0);
  for (size_t c = 0; c < cls.size(); c++)
    for (size_t q = 0; q < pats.size(); q++) {
      tab_at[c * pats.size() + q] = (uint32_t)tab.size();
      int to = -1;  // the class the pattern leads to: one for all its positions
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
  std::vector<int> class_of_block(l22.size(), -1);
  for (size_t c = 0; c < cls.size(); c++)
    for (int b = 0; b < cls[c].nblk; b++) class_of_block[b_ib[cls[c].boff + b]] = (int)c;
  std::vector<uint2> &b_list = T.b_list;
  b_list.resize(b_ib.size());
  std::vector<uint64_t> ib_sorted(b_ib.size());
  std::vector<BkRec> &rec = T.rec;
  std::vector<double> &rec_im = T.rec_im;
  bool &im = T.im;
  for (size_t c = 0; c < cls.size(); c++) {
    std::vector<std::pair<uint64_t, int>> order;  // blocks of equal list lengths side by side
    std::vector<std::vector<BkRec>> recs(cls[c].nblk);
    std::vector<std::vector<double>> ims(cls[c].nblk);
    std::vector<uint32_t> nhb(cls[c].nblk);
    for (int b = 0; b < cls[c].nblk; b++) {
      const uint64_t ib = b_ib[cls[c].boff + b], cfg = ib << lo_bits;
      for (int cross = 0; cross < 2; cross++) {
        for (const HiTerm &h : hi) {
          if ((h.pat >= 0) != (cross == 1) || (two_pass && !cross)) continue;
          if ((cfg & h.t->cm) != (h.t->cv & ~lo_mask)) continue;
          const uint64_t to = (cfg ^ h.t->flip) >> lo_bits;
          if (l22[to] == 0) continue;
          const bool neg = __builtin_popcountll(cfg & h.t->sm) & 1;
          if (cross == 0 && class_of_block[to] != (int)c) return false;  // a moved block keeps its lower halves
          if (cross == 1) {  // the source positions are those of the class the pattern leads to
            const uint32_t at = tab_at[c * pats.size() + h.pat];
            int any = -1;
            for (int p = 0; p < cls[c].n && any < 0; p++)
              if ((tab[at + p] & 0x7FFFu) != kBkNone) any = cls_of[low[cls[c].uoff + p] ^ pats[h.pat][2]];
            if (any < 0) continue;  // no row of the class matches
            if (class_of_block[to] != any) return false;
          }
          recs[b].push_back(BkRec{l22[to] - 1u, cross ? tab_at[c * pats.size() + h.pat] : 0u, neg ? -h.t->re : h.t->re});
          ims[b].push_back(neg ? -h.t->im : h.t->im);
          im = im || h.t->im != 0.0;
        }
        if (cross == 0) nhb[b] = (uint32_t)recs[b].size();
      }
      if (recs[b].size() > (size_t)kBkList) return false;
      order.push_back({((uint64_t)nhb[b] << 32) | recs[b].size(), b});
    }
    std::stable_sort(order.begin(), order.end());
    std::vector<uint32_t> r0(cls[c].nblk);
    for (int b = 0; b < cls[c].nblk; b++) {
      r0[b] = b_row0[cls[c].boff + order[b].second];
      ib_sorted[cls[c].boff + b] = b_ib[cls[c].boff + order[b].second];
    }
    for (int b = 0; b < cls[c].nblk; b++) {
      const int o = order[b].second;
      b_row0[cls[c].boff + b] = r0[b];
      b_list[cls[c].boff + b] = make_uint2((uint32_t)rec.size(), nhb[o] | ((uint32_t)(recs[o].size() - nhb[o]) << 16));
      rec.insert(rec.end(), recs[o].begin(), recs[o].end());
      rec_im.insert(rec_im.end(), ims[o].begin(), ims[o].end());
    }
    if (rec.size() > (1u << 26)) return false;
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
    if (h.pat >= 0) xhi |= h.t->flip >> lo_bits;
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
// share of the rows each, but no less than one turn of the threads (8-site Kondo chain, a step:
// 36.4 us with whole blocks, 33.8 shared out.  Where there are more tasks the second staging of
// a block costs more than the even end gives: 24-site J1-J2 chain, 2.8 tasks per CTA, 105 us
// whole and 113 in halves).
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
