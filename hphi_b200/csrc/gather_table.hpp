// Edge-coloured gather tables of the row and block kernels, made on the host.
#pragma once
#include <cstdint>
#include <vector>

namespace hphi {

// Entries of one warp.  A task's n positions belong to warps of 32; the warp's position l reads the sources
// ent[ptr[l]] .. ent[ptr[l + 1]) (source position | negative << 16) from shared memory.  The entries of
// the 16 positions of a half-warp form a bipartite multigraph between lanes and shared-memory bank
// pairs (source word mod 16).  A proper edge colouring with Delta colours (Delta = its largest
// degree; Konig's theorem, built by swapping alternating paths) gives slots in which every lane
// and every bank pair carries at most one entry; a lane left without one reads a zero word
// (n .. n + 15, one per bank pair) of a bank pair that the slot leaves free.  Returns the number of
// slots; code[slot * 32 + lane] is the word | sign << 15, in whole sets of 8 slots, padded with zero
// words.
int gather_warp(const uint32_t *ptr, const uint32_t *ent, int n, std::vector<uint16_t> *code);

// The set of 8 slots beginning at `slot` as lane `lane` loads it: two entries per word.
struct GatherSet {
  uint32_t w[4];
};
inline GatherSet gather_set(const std::vector<uint16_t> &code, int slot, int lane) {
  GatherSet s;
  for (int k = 0; k < 4; k++)
    s.w[k] = (uint32_t)code[(size_t)(slot + 2 * k) * 32 + lane] | ((uint32_t)code[(size_t)(slot + 2 * k + 1) * 32 + lane] << 16);
  return s;
}

}  // namespace hphi
