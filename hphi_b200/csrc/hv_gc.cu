// Tile kernel: H*v of grand-canonical sectors whose rows are their configurations (SpinGC,
// HubbardGC), src/mltplySpin.c:450-703 and src/mltplyHubbard.c:150-330 in gather form.
//
// A term maps row r to row r ^ flip.  A pass picks K of the n bits (the lowest ones always among
// them, so that rows of a tile come in whole 64-byte pieces) and works on tiles: the 2^K rows
// that agree in the other bits, staged in shared memory.  Every term whose flip and condition
// lie in the pass's bits stays inside a tile, where its source is the word at q ^ f: a
// permutation of the lanes' words, without bank conflicts and without any table.  A few passes
// (3 or 4 for the 24-site Kitaev-Heisenberg honeycomb) cover all terms; each reads v1 once and
// updates v0 once.  The row-block passes this replaces test every term of every row one by one
// (four bit patterns per bond) and gather the crossing ones from memory.
//
// Terms are merged to groups of one flip, one sign mask and at most two condition bits; a
// group's coefficient is picked by those bits.  Bound by memory for few terms per pass, by
// instruction issue for many (about 6 instructions per group and element).  24-site
// Kitaev-Heisenberg honeycomb, complex: 4 passes of 196 us, where the row and column passes of
// the row-block plan took 973 + 369.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdint>
#include <map>
#include <string>
#include <type_traits>
#include <vector>

#include "device_util.cuh"
#include "engine.hpp"
#include "hv_gc.hpp"
#include "plan_upload.hpp"
#include "tma.cuh"

namespace hphi {
namespace {

constexpr int kTidBits = 9, kGcThreads = 1 << kTidBits;
constexpr int kGcPasses = 12;     // more passes than this cost more than the general kernels
constexpr int kGcGroups = 24;     // groups of one pass
// Smallest sectors, in bits.  A tile is a CTA's task, and below 64 to 128 of them too few of the 148
// SMs work; real vectors with fermion signs have the longest sweep per byte and wait for the sector to
// leave L2.  H*v in us, tiles against the kernel without them (the general one, the row-block
// plan at 24 bits): chains with a field, complex 18 bits 33 / 31, 19: 35 / 53; real 19: 44 / 30, 20: 46 /
// 52; Hubbard rings, complex 18: 30 / 25, 20: 48 / 68; real 20: 43 / 38, 22: 143 / 130, 24: 512 / 620.
constexpr int kGcBitsComplex = 19, kGcBitsReal = 20, kGcBitsSigned = 24;
// 64 KB of shared memory per tile, two CTAs per SM: one stages while the other computes
template <typename T> struct GcTile;
template <> struct GcTile<double> { static constexpr int K = 13, low = 3; };
template <> struct GcTile<cplx> { static constexpr int K = 12, low = 2; };

// A group in tile coordinates.  Position q of a tile is thread q % kGcThreads, element q /
// kGcThreads.  Source q ^ f; coefficient c[bit i of q + 2 * bit j of q]; sign (-1)^popcount(q & sm)
// times that of the tile's other bits, (-1)^popcount(base & smo).  The element's share of the
// condition and the sign is worked out here, one bit per element, so that the kernel tests
// constants: `at` is 0 where both condition bits are the thread's, 1 where j is the element's,
// 2 where both are.
struct GcGroup {
  uint32_t ft, sm;         // flip and sign masks among the thread's bits
  int fe;                  // flip among the elements
  int i, j, at;
  uint32_t bi, bj, sgn;    // per element: condition bits i and j, sign
  uint32_t any_sign;
  uint64_t smo;
  double re[4];
};

struct GcPass {
  int ngroup, first, last;   // first: applies acc and the diagonal; last: sums all passes' records
  int nouter;
  const uint32_t *dep;       // [2^(K - low)] the tile's bits above the lowest ones, in place
  uint8_t outer[32];         // bit positions of the other bits, increasing
  GcGroup g[kGcGroups];      // kernel parameters: uniform operands
  double im[kGcGroups][4];   // imaginary parts of the coefficients
};

__device__ __forceinline__ void gc_fma(double &y, double c, double x) { y = fma(c, x, y); }
__device__ __forceinline__ void gc_fma(cplx &y, double c, const cplx &x) {
  y.x = fma(c, x.x, y.x);
  y.y = fma(c, x.y, y.y);
}
__device__ __forceinline__ void gc_fma_i(double &, double, const double &) {}
__device__ __forceinline__ void gc_fma_i(cplx &y, double ci, const cplx &x) {
  y.x = fma(-ci, x.y, y.x);
  y.y = fma(ci, x.x, y.y);
}
__device__ __forceinline__ double gc_lds(const double *p) { return *p; }
__device__ __forceinline__ cplx gc_lds(const cplx *p) {
  const double2 z = *reinterpret_cast<const double2 *>(p);
  return cplx{z.x, z.y};
}

// y of one element (position q of the tile) without the patterns that no term matches.  The kernel
// multiplies their sources by 0 (passing them by in its sweep took the 24-site Kitaev-Heisenberg
// honeycomb, complex, from 769 to 932 us; this way it is 782), which must not spread an infinity to rows that H does not
// couple to it: a non-finite y shows in the products with x that a sweep sums anyway, and the sweep's
// elements are then left out there and worked out here.
template <typename T, bool IM>
__device__ __forceinline__ T gc_element(const GcPass &ps, const T *x, uint64_t base, int q, double diag) {
  const int tid = q % kGcThreads, qe = q / kGcThreads;
  T y = ps.first ? VT<T>::scale(diag, x[q]) : VT<T>::zero();
#pragma unroll 1
  for (int k = 0; k < ps.ngroup; k++) {
    const GcGroup &g = ps.g[k];
    const int c = ((q >> g.i) & 1) | (((q >> g.j) & 1) << 1);
    const uint32_t sg = (uint32_t)__popc((uint32_t)tid & g.sm) + (uint32_t)__popcll(base & g.smo) + (g.sgn >> qe);
    const double re = g.re[c], im = IM ? ps.im[k][c] : 0.0;
    const T z = x[(tid ^ (int)g.ft) + ((qe ^ g.fe) * kGcThreads)];
    if (re != 0.0) gc_fma(y, sg & 1u ? -re : re, z);
    if (im != 0.0) gc_fma_i(y, sg & 1u ? -im : im, z);
  }
  return y;
}

// IM: some coefficient has an imaginary part (complex vectors only).
template <typename T, bool IM>
__global__ void __launch_bounds__(kGcThreads, 2) gc_tile_kernel(const __grid_constant__ GcPass ps, int64_t ntile,
                                                                const double *__restrict__ diag,
                                                                const T *__restrict__ v1, T *__restrict__ v0,
                                                                const double *__restrict__ coef, SumOut so) {
  constexpr int K = GcTile<T>::K, LOW = GcTile<T>::low, M = (1 << K) / kGcThreads;
  constexpr int H = M < 4 ? M : 4;  // elements per thread and sweep over the groups (registers)
  extern __shared__ __align__(16) unsigned char gc_smem[];
  T *x = reinterpret_cast<T *>(gc_smem);
  const double acc = ps.first ? coef[0] : 1.0, scale = coef[1];
  const int tid = threadIdx.x;
  __shared__ uint32_t s_dep[1 << (K - LOW)];
  for (int k = tid; k < (1 << (K - LOW)); k += kGcThreads) s_dep[k] = __ldg(ps.dep + k);
  auto dep = [&](int m) {  // the thread's m-th row within a tile
    const int q = tid + m * kGcThreads;
    return s_dep[q >> LOW] | (uint32_t)(q & ((1 << LOW) - 1));
  };
  auto base_of = [&](int64_t t) {
    uint64_t base = 0;
    for (int b = 0; b < ps.nouter; b++) base |= (uint64_t)((t >> b) & 1) << ps.outer[b];
    return base;
  };
  double pr[2] = {0.0, 0.0};
  for (int64_t t = blockIdx.x; t < ntile; t += gridDim.x) {
    const uint64_t base = base_of(t);
    __syncthreads();  // the previous tile is no longer read (and s_dep is there)
    const uint32_t dst = smem_u32(x);
#pragma unroll
    for (int m = 0; m < M; m++) {
      if constexpr (sizeof(T) == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + 16 * (tid + m * kGcThreads)),
                     "l"(v1 + (base | dep(m)))
                     : "memory");
      else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst + 8 * (tid + m * kGcThreads)),
                     "l"(v1 + (base | dep(m)))
                     : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    uint32_t again = 0;  // elements whose products with x are not finite: gc_element
#pragma unroll
    for (int m0 = 0; m0 < M; m0 += H) {
      T y[H], old[H];
      uint32_t row[H];
#pragma unroll
      for (int m = 0; m < H; m++) {  // the old v0 and the diagonal arrive during the sweep
        row[m] = dep(m0 + m);
        old[m] = VT<T>::zero();
        if (acc != 0.0) old[m] = v0[base | row[m]];
        y[m] = VT<T>::zero();
      }
      if (ps.first) {
#pragma unroll
        for (int m = 0; m < H; m++)
          y[m] = VT<T>::scale(__ldg(diag + (base | row[m])), gc_lds(x + tid + (m0 + m) * kGcThreads));
      }
      for (int k = 0; k < ps.ngroup; k++) {
        const GcGroup &g = ps.g[k];
        const T *xs = x + (tid ^ (int)g.ft);
        // y += coefficient * source of the sweep's elements, coefficient(element) by kind of group
        auto sweep = [&](auto coefficient, auto imag) {
#pragma unroll
          for (int m = 0; m < H; m++) {
            const double cc = coefficient(m0 + m);
            const T z = gc_lds(xs + ((m0 + m) ^ g.fe) * kGcThreads);
            if (decltype(imag)::value) gc_fma_i(y[m], cc, z);
            else gc_fma(y[m], cc, z);
          }
        };
        auto flip = [](double c, uint32_t sg) { return __hiloint2double(__double2hiint(c) ^ (int)sg, __double2loint(c)); };
        auto part = [&](const double(&c)[4], auto imag) {
          const bool bi = (tid >> g.i) & 1;  // read where bit i is the thread's
          if (g.any_sign) {
            const uint32_t sg = ((uint32_t)__popc((uint32_t)tid & g.sm) + (uint32_t)__popcll(base & g.smo)) << 31;
            auto sign = [&](int qe) { return sg ^ ((g.sgn >> qe) << 31); };
            if (g.at == 0) {
              const double c0 = ((tid >> g.j) & 1) ? (bi ? c[3] : c[2]) : (bi ? c[1] : c[0]);
              sweep([&](int qe) { return flip(c0, sign(qe)); }, imag);
            } else if (g.at == 1) {
              const double c0 = bi ? c[1] : c[0], c1 = bi ? c[3] : c[2];
              sweep([&](int qe) { return flip(((g.bj >> qe) & 1u) ? c1 : c0, sign(qe)); }, imag);
            } else {
              sweep([&](int qe) { return flip(c[((g.bi >> qe) & 1u) | (((g.bj >> qe) & 1u) << 1)], sign(qe)); }, imag);
            }
          } else if (g.at == 0) {
            const double c0 = ((tid >> g.j) & 1) ? (bi ? c[3] : c[2]) : (bi ? c[1] : c[0]);
            sweep([&](int) { return c0; }, imag);
          } else if (g.at == 1) {
            const double c0 = bi ? c[1] : c[0], c1 = bi ? c[3] : c[2];
            sweep([&](int qe) { return ((g.bj >> qe) & 1u) ? c1 : c0; }, imag);
          } else {
            sweep([&](int qe) { return c[((g.bi >> qe) & 1u) | (((g.bj >> qe) & 1u) << 1)]; }, imag);
          }
        };
        part(g.re, std::false_type{});
        if (IM) part(ps.im[k], std::true_type{});
      }
      double d[2] = {0.0, 0.0};
#pragma unroll
      for (int m = 0; m < H; m++) {
        const T xq = gc_lds(x + tid + (m0 + m) * kGcThreads);
        d[0] += VT<T>::conj_mul_re(xq, y[m]);
        d[1] += VT<T>::conj_mul_im(xq, y[m]);
      }
      if (!isfinite(d[0])) {
        again |= ((1u << H) - 1) << m0;
        continue;
      }
      pr[0] += d[0];
      pr[1] += d[1];
#pragma unroll
      for (int m = 0; m < H; m++) {
        const T ys = VT<T>::scale(scale, y[m]);
        v0[base | row[m]] = (acc == 0.0) ? ys : VT<T>::add(VT<T>::scale(acc, old[m]), ys);
      }
    }
#pragma unroll 1
    for (; again; again &= again - 1) {
      const int q = tid + (__ffs((int)again) - 1) * kGcThreads;
      const int64_t r = (int64_t)(base | dep(q / kGcThreads));
      const T xq = gc_lds(x + q), y = gc_element<T, IM>(ps, x, base, q, ps.first ? __ldg(diag + r) : 0.0);
      pr[0] += VT<T>::conj_mul_re(xq, y);
      pr[1] += VT<T>::conj_mul_im(xq, y);
      const T ys = VT<T>::scale(scale, y);
      v0[r] = (acc == 0.0) ? ys : VT<T>::add(VT<T>::scale(acc, v0[r]), ys);
    }
  }
  if (ps.last) {
    grid_sum<2>(pr, so);
  } else {
    block_sum<2>(pr);
    if (tid == 0) {
      so.part[2 * (so.rec0 + blockIdx.x)] = pr[0];
      so.part[2 * (so.rec0 + blockIdx.x) + 1] = pr[1];
    }
  }
}

}  // namespace

struct GcPlan {
  std::vector<void *> allocs;
  std::vector<GcPass> pass[2];   // real, complex vectors
  bool im = false;
  int grid[2] = {0, 0};
  int64_t ntile[2] = {0, 0};
  double *part = nullptr;
};

void gc_plan_free(GcPlan *p) {
  if (!p) return;
  for (void *q : p->allocs) cudaFree(q);
  delete p;
}

namespace {

// A group in the configuration's bits.
struct Raw {
  uint64_t flip, sm;
  int i, j;  // condition bits (equal: one bit)
  std::array<double, 4> re{}, im{};
};

// One term into its group; false when it has more than two condition bits.
bool merge_term(const BitTerm &t, std::vector<Raw> *raw) {
  const uint64_t bits = t.cm;
  const int n = __builtin_popcountll(bits);
  if (n > 2 || t.flip == 0) return false;
  // sign bits inside the condition have fixed values: they go into the coefficient
  const double sg = (__builtin_popcountll(t.cv & t.sm & bits) & 1) ? -1.0 : 1.0;
  const uint64_t sm = t.sm & ~bits;
  int i, j;
  if (n == 0) i = j = __builtin_ctzll(t.flip);
  else {
    i = __builtin_ctzll(bits);
    j = 63 - __builtin_clzll(bits);
  }
  Raw *r = nullptr;
  for (Raw &x : *raw)
    if (x.flip == t.flip && x.sm == sm && x.i == i && x.j == j) r = &x;
  if (!r) {
    raw->push_back(Raw{t.flip, sm, i, j, {}, {}});
    r = &raw->back();
  }
  for (int k = 0; k < 4; k++) {
    const int bi = k & 1, bj = k >> 1;
    if (i == j && bi != bj) continue;  // never read
    if (n > 0 && (((t.cv >> i) & 1) != (uint64_t)bi || ((t.cv >> j) & 1) != (uint64_t)bj)) continue;
    r->re[k] += sg * t.re;
    r->im[k] += sg * t.im;
  }
  return true;
}

// Bit sets of K bits (the `low` lowest always among them) that cover every group's flip and
// condition bits: greedily the set that takes most groups, grown group by group.
std::vector<uint64_t> cover_passes(const std::vector<Raw> &raw, int n, int K, int low) {
  const uint32_t base = (1u << low) - 1u;
  std::vector<uint32_t> need;  // of the groups still to cover (n <= 32 bits)
  for (const Raw &r : raw) need.push_back((uint32_t)(r.flip | (1ull << r.i) | (1ull << r.j)));
  // groups within a set: the loop that the whole search spends its time in
  auto within = [&](uint32_t set) {
    int g = 0;
    for (uint32_t x : need) g += (x & ~set) == 0;
    return g;
  };
  std::vector<uint64_t> sets;
  while (!need.empty()) {
    uint32_t best = 0;
    int best_n = 0;
    // all seeds of up to 64 groups, 32 of more (the search grows with the cube of the groups)
    const size_t step = need.size() <= 64 ? 1 : (need.size() + 31) / 32;
    for (size_t q = 0; q < need.size(); q += step) {
      uint32_t set = base | need[q];
      if (__builtin_popcount(set) > K) continue;
      for (;;) {  // the group that adds the fewest bits, then the one that shares most with others
        int cost = 99, gain = -1;
        uint32_t pick = 0;
        for (uint32_t x : need) {
          const uint32_t add = x & ~set;
          if (add == 0) continue;
          const int c = __builtin_popcount(add);
          if (__builtin_popcount(set) + c > K) continue;
          const int g = within(set | add);
          if (g - 2 * c > gain - 2 * cost || pick == 0) { pick = add; cost = c; gain = g; }
        }
        if (pick == 0) break;
        set |= pick;
      }
      const int covered = within(set);
      if (covered > best_n) { best_n = covered; best = set; }
    }
    if (best_n == 0) return {};
    for (int b = 0; b < n && __builtin_popcount(best) < K; b++) best |= 1u << b;  // fill up with low bits
    sets.push_back(best);
    if (sets.size() > (size_t)kGcPasses) return {};
    need.erase(std::remove_if(need.begin(), need.end(), [&](uint32_t x) { return (x & ~best) == 0; }), need.end());
  }
  return sets;
}

uint64_t extract_bits(uint64_t x, uint64_t set) {  // bits of x at the places of set, packed
  uint64_t r = 0;
  int k = 0;
  for (int b = 0; b < 64; b++)
    if ((set >> b) & 1) r |= ((x >> b) & 1) << k++;
  return r;
}

// Passes of one vector type; leaves p->pass[vt] empty where the plan does not apply.
template <typename T>
void build_passes(Sector *s, GcPlan *p, const std::vector<Raw> &raw, int vt) {
  constexpr int K = GcTile<T>::K, low = GcTile<T>::low;
  const int n = s->model.nbits;
  std::vector<uint64_t> sets = raw.empty() ? std::vector<uint64_t>{(1ull << K) - 1} : cover_passes(raw, n, K, low);
  if (sets.empty()) return;
  // a group that several passes could take goes to the one with fewest, the least movable groups first
  std::vector<int> owner(raw.size(), -1), load(sets.size(), 0);
  std::vector<std::pair<int, size_t>> order;
  auto fits = [&](size_t q, size_t a) {
    return ((raw[q].flip | (1ull << raw[q].i) | (1ull << raw[q].j)) & ~sets[a]) == 0;
  };
  for (size_t q = 0; q < raw.size(); q++) {
    int n_fit = 0;
    for (size_t a = 0; a < sets.size(); a++) n_fit += fits(q, a);
    order.push_back({n_fit, q});
  }
  std::sort(order.begin(), order.end());
  for (const auto &o : order) {
    for (size_t a = 0; a < sets.size(); a++)
      if (fits(o.second, a) && (owner[o.second] < 0 || load[a] < load[owner[o.second]])) owner[o.second] = (int)a;
    load[owner[o.second]]++;
  }
  std::vector<GcPass> passes(sets.size());
  std::vector<std::vector<uint32_t>> deps(sets.size());
  PlanUpload up;
  for (size_t a = 0; a < sets.size(); a++) {
    const uint64_t set = sets[a];
    constexpr int M = (1 << K) / kGcThreads;
    GcPass &ps = passes[a];
    ps = GcPass{};
    for (size_t q = 0; q < raw.size(); q++) {
      const Raw &r = raw[q];
      if (owner[q] != (int)a) continue;
      if (ps.ngroup == kGcGroups) return;
      GcGroup &g = ps.g[ps.ngroup];
      const uint32_t f = (uint32_t)extract_bits(r.flip, set), sm = (uint32_t)extract_bits(r.sm, set);
      g.ft = f % kGcThreads;
      g.fe = (int)(f / kGcThreads);
      g.sm = sm % kGcThreads;
      g.smo = r.sm & ~set;
      g.any_sign = r.sm != 0;
      g.i = __builtin_popcountll(set & ((1ull << r.i) - 1));
      g.j = __builtin_popcountll(set & ((1ull << r.j) - 1));
      g.at = g.j < kTidBits ? 0 : g.i < kTidBits ? 1 : 2;
      for (int m = 0; m < M; m++) {
        const uint32_t qm = (uint32_t)m * kGcThreads;
        if (g.i >= kTidBits) g.bi |= ((qm >> g.i) & 1u) << m;
        if (g.j >= kTidBits) g.bj |= ((qm >> g.j) & 1u) << m;
        g.sgn |= ((uint32_t)__builtin_popcount(qm & sm) & 1u) << m;
      }
      for (int k = 0; k < 4; k++) {
        g.re[k] = r.re[k];
        ps.im[ps.ngroup][k] = r.im[k];
      }
      ps.ngroup++;
    }
    std::vector<uint32_t> &dep = deps[a];
    dep.resize(1u << (K - low));
    std::vector<int> in;
    for (int b = 0; b < n; b++) {
      if (!((set >> b) & 1)) ps.outer[ps.nouter++] = (uint8_t)b;
      else if (b >= low) in.push_back(b);
    }
    for (uint32_t q = 0; q < dep.size(); q++)
      for (size_t k = 0; k < in.size(); k++) dep[q] |= ((q >> k) & 1u) << in[k];
    ps.first = a == 0;
    ps.last = a + 1 == sets.size();
    up.add(dep, &ps.dep);
  }
  const size_t smem = sizeof(T) << K;
  int per_sm = 0;
  const void *f[2] = {(const void *)gc_tile_kernel<T, false>, (const void *)gc_tile_kernel<T, true>};
  const bool im = p->im && sizeof(T) == 16;
  if (raise_smem_limit(f[im], smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f[im], kGcThreads, smem) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    return;
  }
  if (up.run(&p->allocs) != 0) {
    cudaGetLastError();
    return;
  }
  p->ntile[vt] = 1ll << (n - K);
  p->grid[vt] = (int)std::min<int64_t>(p->ntile[vt], (int64_t)per_sm * s->num_sms);
  p->pass[vt] = passes;
}

}  // namespace

// Leaves s->gcp null where the plan does not apply or there is no memory for it: the other kernels remain.
void gc_plan_build(Sector *s) {
  s->gcp = nullptr;
  const Model &m = s->model;
  // rows within a tile are 32-bit numbers
  if (!s->gc || m.general_spin || m.nbits > 32 || m.nbits < kGcBitsComplex) return;
  std::vector<Raw> raw;
  for (const BitTerm &t : m.offdiag)
    if (!merge_term(t, &raw) || raw.size() > (size_t)kGcPasses * kGcGroups) return;
  GcPlan *p = new GcPlan();
  for (const Raw &r : raw)
    for (double x : r.im) p->im = p->im || x != 0.0;
  bool signs = false;
  for (const Raw &r : raw) signs = signs || r.sm != 0;
  const bool real = !m.complex_terms && m.nbits >= (signs ? kGcBitsSigned : kGcBitsReal);
  if (real) build_passes<double>(s, p, raw, 0);
  build_passes<cplx>(s, p, raw, 1);
  if (p->pass[0].empty() && p->pass[1].empty()) {
    gc_plan_free(p);
    return;
  }
  s->gcp = p;
  const size_t nd = std::max(gc_scratch_doubles(s, kReal64), gc_scratch_doubles(s, kComplex128));
  if (cudaMalloc(&p->part, sizeof(double) * std::max<size_t>(2, nd)) != cudaSuccess) {
    cudaGetLastError();
    gc_plan_free(p);
    s->gcp = nullptr;
    return;
  }
  p->allocs.push_back(p->part);
}

bool gc_applies(const Sector *s, VecType vt) { return s->gcp && !s->gcp->pass[vt == kReal64 ? 0 : 1].empty(); }

int gc_passes(const Sector *s, VecType vt) { return (int)s->gcp->pass[vt == kReal64 ? 0 : 1].size(); }

size_t gc_scratch_doubles(const Sector *s, VecType vt) {
  const int v = vt == kReal64 ? 0 : 1;
  return 2 * s->gcp->pass[v].size() * (size_t)s->gcp->grid[v];
}

double *gc_part(const Sector *s) { return s->gcp->part; }

int gc_hv_launch(Sector *s, VecType vt, const void *d_v1, void *d_v0, const double *d_coef, double *d_out,
                 double *d_part, const LanczosTail *lt) {
  const GcPlan *p = s->gcp;
  const int v = vt == kReal64 ? 0 : 1, grid = p->grid[v];
  for (size_t a = 0; a < p->pass[v].size(); a++) {
    const SumOut so = sum_out(d_part, (int)a * grid, (int)p->pass[v].size() * grid, s->d_done, d_out, 0, lt);
    if (v == 0)
      gc_tile_kernel<double, false><<<grid, kGcThreads, sizeof(double) << GcTile<double>::K, s->stream>>>(
          p->pass[v][a], p->ntile[v], s->d_diag, (const double *)d_v1, (double *)d_v0, d_coef, so);
    else if (p->im)
      gc_tile_kernel<cplx, true><<<grid, kGcThreads, sizeof(cplx) << GcTile<cplx>::K, s->stream>>>(
          p->pass[v][a], p->ntile[v], s->d_diag, (const cplx *)d_v1, (cplx *)d_v0, d_coef, so);
    else
      gc_tile_kernel<cplx, false><<<grid, kGcThreads, sizeof(cplx) << GcTile<cplx>::K, s->stream>>>(
          p->pass[v][a], p->ntile[v], s->d_diag, (const cplx *)d_v1, (cplx *)d_v0, d_coef, so);
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error(std::string("grand-canonical kernel: launch failed: ") + cudaGetErrorString(e));
    return -1;
  }
  return 0;
}

}  // namespace hphi
