// Tables of the block kernel (hv_blocks.cu), made on the host from a sector's lists and terms.
// Nothing here touches the device, so the tables can be checked against the terms on the CPU.
#pragma once
#include <cstdint>
#include <vector>

#include "engine.hpp"

namespace hphi {

constexpr int kBkGroups = 8;      // lower-half coefficients, up to sign
constexpr int kBkCross = 64;      // crossing terms
constexpr int kBkList = 96;       // upper or crossing terms acting on one block: whole products,
constexpr int kBkListRows = 256;  // row passes (as many crossing terms as the row-block plan takes)
constexpr uint32_t kBkNone = 0x7FFFu;

struct BkClass {
  int n, nblk, boff, uoff;                // rows of a block, blocks, first block in b_*, first lower half
  int gat, sets;                          // gather table (16-byte units), sets of 8 slots per warp of 32 positions
  int head;                               // per warp: slots of each group (8 bits each)
};

// A term on a block: the first row of its source block, the table of source positions (crossing
// terms; positions keep their number under an upper-half term), and the coefficient, signs of the
// upper half included.
struct BkRec {
  uint32_t row, tab;
  double re;
};

// A task: its class, two blocks (the second ~0: none, and with complex vectors), and the positions
// it computes (first | last + 1 << 16, multiples of 32): long blocks are shared by several tasks.
struct BkTask {
  uint32_t cls, b0, b1, span;
};

// Shapes by the longest block (planes of `stride` words: a block and 16 zero words) and, where a
// sector has long and short ones, by the length its rows see.  Two planes share the table entries;
// a thread takes Q positions, which share the addresses and coefficients of the listed terms, and
// has U terms per block and position in flight.  Small CTAs, several per SM: a task is staging, then
// gathers, then loads from L2, and only other CTAs fill the waits between them; five of 128
// threads with 95 registers, since the address arithmetic of the listed terms wants them (24-site
// J1-J2 chain, blocks of 924 rows, us per H*v: eight CTAs with 64 registers 107, six with 80: 89,
// five with 95: 78; four planes and 256 threads 137; the general kernel 146).
struct BkShapeDef {
  int stride, P, Q, U, threads, ctas;
};
constexpr BkShapeDef kBkShapeDefs[] = {
    {96, 2, 1, 4, 96, 6},     {288, 2, 2, 2, 128, 5},   {960, 2, 2, 2, 64, 10},    {960, 2, 2, 2, 128, 5},
    {1744, 2, 2, 2, 256, 2},  {3456, 2, 2, 2, 256, 2},  {6560, 2, 2, 2, 512, 1},   {12896, 2, 2, 2, 1024, 1},
};
constexpr int kBkShapes = 8;
// Tasks per resident CTA that long blocks are shared out to (block_tasks).
constexpr int kBkWaves = 2;
// Mean block length, as a row sees it, from which 128 threads share a task of 960-word planes
// (else 64).  us per H*v with 128 and with 64 threads, real | complex, by mean length: 23-site chain
// 757: 42 / 55 | 65 / 67, 22 sites 395: 29 / 33 | 40 / 46, spin-1 chain of 13 sites 326: 12.6 / 16.1 |
// 15.6 / 21.2; below, it depends on the sector: 24 sites with 2Sz = -12, 278: 17.2 / 21.4 | 31 / 24,
// spin-3/2 of 12 sites with 2Sz = 14, 286: 35 / 28 | 38 / 48, 8-site Kondo 234: 28.5 / 29.5 | 38.6 / 41.6,
// 24 sites with 2Sz = -14, 183: 15.5 / 14.0 | 23.6 / 19.5.
constexpr int kBkLong = 320;

struct BlockTables {
  std::vector<BkClass> cls;
  std::vector<uint32_t> b_row0;   // per block, by class: its first row
  std::vector<uint2> b_list;      // its first record, and numbers of upper (low half) and crossing terms
  std::vector<BkRec> rec;
  std::vector<double> rec_im;     // imaginary parts of the records' coefficients
  std::vector<uint4> gat;
  std::vector<uint2> head;
  std::vector<double2> cf;        // lower-half coefficients by group
  std::vector<uint16_t> tab;      // source position | sign << 15 of each position, kBkNone: not matched
  // Blocks in the order the tasks take them; real vectors pair neighbours of one class and group.
  struct Place {
    uint64_t group;
    uint32_t cls, b;
  };
  std::vector<Place> order;
  int shape = 0;                  // kBkShapeDefs
  // Records of shared memory per block of a task.  The kernel walks the crossing terms of a task's
  // two blocks side by side, U at a time up to the longer list, so a block with many upper-half
  // terms beside one with many crossing ones takes more than the longest list.
  int nlist = 0;
  bool im = false;                // complex coefficients in the lists
};

// terms: off-diagonal terms; l22: list_2_2; blk, low: sector_blocks.  two_pass: lower-half and crossing
// terms only (the row-block plan's row pass).  false: the plan does not apply (too many or
// complex-valued groups of terms, blocks longer than shared memory, another layout).
bool block_tables(const std::vector<BitTerm> &terms, int lo_bits, const std::vector<uint32_t> &l22,
                  const std::vector<SectorBlock> &blk, const std::vector<uint32_t> &low, int64_t dim, bool two_pass,
                  BlockTables *out);

// True when order[q] and order[q + 1] make one task of real vectors.
bool block_pair(const BlockTables &t, size_t q);

// The tasks for vectors with (cplx) or without imaginary parts on `ctas` resident CTAs.
std::vector<BkTask> block_tasks(const BlockTables &t, bool cplx, int ctas);

}  // namespace hphi
