#include "gather_table.hpp"

#include <algorithm>

namespace hphi {

int gather_warp(const uint32_t *ptr, const uint32_t *ent, int n, std::vector<uint16_t> *code) {
  struct Edge {
    int lane, bank, color;
    uint16_t code;
  };
  auto zero_word = [&](int bank) { return (uint16_t)(n + (((bank - n) % 16) + 16) % 16); };
  struct Scratch {  // kept by each thread: thousands of warps want the same few kilobytes
    std::vector<Edge> ed;
    std::vector<int> L, B, path;           // edge of each (lane | bank, color)
    std::vector<uint64_t> used_l, used_b;  // its colors, as bits
    std::vector<uint16_t> half[2];
  };
  static thread_local Scratch scratch;
  auto &[ed, L, B, path, used_l, used_b, half] = scratch;
  int slots[2];
  for (int hw = 0; hw < 2; hw++) {
    ed.clear();
    int ldeg[16] = {0}, bdeg[16] = {0};
    for (int l = 0; l < 16; l++) {
      const int p = 16 * hw + l;
      for (uint32_t k = ptr[p]; k < ptr[p + 1]; k++) {
        const uint32_t word = ent[k] & 0xFFFFu;
        ed.push_back(Edge{l, (int)(word % 16), -1, (uint16_t)(word | ((ent[k] >> 16 & 1u) << 15))});
        ldeg[l]++;
        bdeg[word % 16]++;
      }
    }
    int D = 0;
    for (int i = 0; i < 16; i++) D = std::max({D, ldeg[i], bdeg[i]});
    const int nw = (D + 63) / 64;
    L.assign((size_t)16 * D, -1);
    B.assign((size_t)16 * D, -1);
    used_l.assign((size_t)16 * nw, 0);
    used_b.assign((size_t)16 * nw, 0);
    auto first_free = [&](const uint64_t *u) {
      int k = 0;
      while (u[k] == ~0ull) k++;
      return 64 * k + __builtin_ctzll(~u[k]);
    };
    auto mark = [](std::vector<uint64_t> &u, int words, int node, int color, bool on) {
      uint64_t &x = u[(size_t)node * words + color / 64];
      const uint64_t bit = 1ull << (color % 64);
      x = on ? x | bit : x & ~bit;
    };
    auto place = [&](int e, bool on) {
      const Edge &x = ed[e];
      L[(size_t)x.lane * D + x.color] = on ? e : -1;
      B[(size_t)x.bank * D + x.color] = on ? e : -1;
      mark(used_l, nw, x.lane, x.color, on);
      mark(used_b, nw, x.bank, x.color, on);
    };
    for (int i = 0; i < (int)ed.size(); i++) {
      const int l = ed[i].lane, bk = ed[i].bank;
      const int a = first_free(&used_l[(size_t)l * nw]), c = first_free(&used_b[(size_t)bk * nw]);
      if (B[(size_t)bk * D + a] >= 0) {
        // alternating a/c path from bank bk; swapping it frees a at bk
        path.clear();
        int node = bk, want = a;
        bool at_bank = true;
        for (;;) {
          const int e = at_bank ? B[(size_t)node * D + want] : L[(size_t)node * D + want];
          if (e < 0) break;
          path.push_back(e);
          node = at_bank ? ed[e].lane : ed[e].bank;
          at_bank = !at_bank;
          want = (want == a) ? c : a;
        }
        for (int e : path) place(e, false);
        for (int e : path) ed[e].color = (ed[e].color == a) ? c : a;
        for (int e : path) place(e, true);
      }
      ed[i].color = a;
      place(i, true);
    }
    half[hw].resize((size_t)16 * D);
    for (int k = 0; k < D; k++) {
      int f = 0;  // next bank pair that the slot may leave free
      for (int l = 0; l < 16; l++) {
        const int e = L[(size_t)l * D + k];
        if (e < 0)
          while (B[(size_t)f * D + k] >= 0) f++;
        half[hw][(size_t)16 * k + l] = e >= 0 ? ed[e].code : zero_word(f++);
      }
    }
    slots[hw] = D;
  }
  const int total = std::max(slots[0], slots[1]), padded = (total + 7) / 8 * 8;
  code->resize((size_t)padded * 32);
  for (int k = 0; k < padded; k++)
    for (int lane = 0; lane < 32; lane++)
      (*code)[(size_t)32 * k + lane] = k < slots[lane / 16] ? half[lane / 16][(size_t)16 * k + lane % 16] : zero_word(lane % 16);
  return total;
}

}  // namespace hphi
