// Green's functions <v| O_e |v> for batches of operator strings.
//
// Replaces the per-entry passes of expec_cisajs (src/expec_cisajs.c:66-641) and
// expec_cisajscktaltdc (src/expec_cisajscktaltdc.c:87-1647).  The reference makes one full
// pass over the vector for every entry, each row testing the entry's occupation pattern,
// looking up the row of the changed configuration (GetOffComp, src/bitcalc.c:195-223) and
// adding conj(v[off]) * sgn * v[j].  Here one pass serves a batch of entries: each thread
// reads its row's configuration and vector element once and evaluates every entry of the
// batch on it, accumulating in registers; the batch's masks are kernel parameters (constant
// bank operands of the unrolled entry loop); a fixed-order block reduction and a fixed-order
// sum over blocks make the result reproducible.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <map>
#include <string>
#include <vector>

#include "device_util.cuh"
#include "engine.hpp"

namespace hphi {
namespace {

constexpr int kGreenThreads = 256;
constexpr int kGreenAcc = 16;  // doubles accumulated per thread: 16 real or 8 complex entries

template <typename T> struct GreenWidth;
template <> struct GreenWidth<double> { static constexpr int w = 1; };
template <> struct GreenWidth<cplx> { static constexpr int w = 2; };

template <typename T>
__device__ __forceinline__ void green_acc(double (&acc)[kGreenAcc], int k, double sg, const T &y, const T &x);
template <>
__device__ __forceinline__ void green_acc<double>(double (&acc)[kGreenAcc], int k, double sg, const double &y,
                                                  const double &x) {
  acc[k] += sg * (y * x);
}
template <>
__device__ __forceinline__ void green_acc<cplx>(double (&acc)[kGreenAcc], int k, double sg, const cplx &y,
                                                const cplx &x) {
  // conj(y) * x
  acc[2 * k] += sg * (y.x * x.x + y.y * x.y);
  acc[2 * k + 1] += sg * (y.x * x.y - y.y * x.x);
}

// A batch of entries passed by value: the masks sit in the kernel's parameter (constant)
// bank and enter the unrolled entry loop as instruction operands.  Unused slots hold a
// pattern no configuration matches (cm = 0, cv = 1).
template <int NB> struct GreenBatch { GreenTerm t[NB]; };

// One batch over all rows (grid-stride, one row per thread); per-block sums of the kGreenAcc
// accumulators go to part[blockIdx.x * kGreenAcc ...].
// C: the configuration word, uint32_t when every configuration fits in 32 bits (halves the
// mask, flip and parity work), else uint64_t.
template <typename C> __device__ __forceinline__ int parity_of(C x);
template <> __device__ __forceinline__ int parity_of<uint32_t>(uint32_t x) { return __popc(x) & 1; }
template <> __device__ __forceinline__ int parity_of<uint64_t>(uint64_t x) { return __popcll(x) & 1; }

template <typename T, bool GC, typename C>
__global__ void __launch_bounds__(kGreenThreads) green_kernel(int64_t dim, const uint64_t *__restrict__ list_1,
                                                              const uint32_t *__restrict__ l21,
                                                              const uint32_t *__restrict__ l22, int lo_bits,
                                                              uint64_t lo_mask,
                                                              const GreenBatch<kGreenAcc / GreenWidth<T>::w> batch,
                                                              const T *__restrict__ v, SumOut so) {
  constexpr int NB = kGreenAcc / GreenWidth<T>::w;
  double acc[kGreenAcc];
#pragma unroll
  for (int q = 0; q < kGreenAcc; q++) acc[q] = 0.0;
  const C lmask = (C)lo_mask;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < dim; r += (int64_t)gridDim.x * blockDim.x) {
    const C c = GC ? (C)r : (C)__ldg(list_1 + r);
    const T x = v[r];
#pragma unroll
    for (int k = 0; k < NB; k++) {
      const GreenTerm &t = batch.t[k];
      bool hit = (c & (C)t.cm) == (C)t.cv;
      int64_t j = r;
      if (hit && t.flip) {
        const C tg = c ^ (C)t.flip;
        if (GC) {
          j = (int64_t)tg;
        } else {
          const uint32_t a = __ldg(l21 + (tg & lmask));
          const uint32_t b = __ldg(l22 + (tg >> lo_bits));
          hit = a != 0u && b != 0u;
          j = (int64_t)a + (int64_t)b - 3;
        }
      }
      if (hit) {
        const double sg = parity_of<C>(c & (C)t.sm) ? -t.coef : t.coef;
        green_acc<T>(acc, k, sg, (j == r) ? x : v[j], x);
      }
    }
  }
  grid_sum<kGreenAcc>(acc, so);
}

// Canonical sectors.  HPhi's rows come in blocks that share the upper half of the configuration,
// and a block's lower halves are those of its class (SectorBlock).  An entry's upper half is one
// answer (condition, sign, source block) for a whole block, its lower half one answer per class
// and position; a warp takes a piece of a block.
__device__ __forceinline__ double ldg_vec(const double *p) { return __ldg(p); }
__device__ __forceinline__ cplx ldg_vec(const cplx *p) {
  const double2 z = __ldg(reinterpret_cast<const double2 *>(p));
  return cplx{z.x, z.y};
}
struct GreenHalf {
  uint32_t cml, cvl, fl, sl, cmh, cvh, fh, sh;  // condition, value, flip and sign masks of the halves
};
template <int NB> struct GreenHalfBatch { GreenHalf t[NB]; };
constexpr uint32_t kGreenNone = 0x7FFFFFFFu;

// Off-diagonal entries, lower half: tab[k][u] = source position | sign << 31 of lower half low[u]
// under entry k of the batch, kGreenNone where the condition fails or the sector ends.
template <int NB>
__global__ void __launch_bounds__(kGreenThreads) green_table_kernel(int nlow, const uint32_t *__restrict__ low,
                                                                    const uint32_t *__restrict__ l21,
                                                                    const GreenHalfBatch<NB> batch,
                                                                    uint32_t *__restrict__ tab) {
  const GreenHalf &e = batch.t[blockIdx.y];
  for (int u = blockIdx.x * kGreenThreads + threadIdx.x; u < nlow; u += gridDim.x * kGreenThreads) {
    const uint32_t ia = low[u];
    uint32_t r = kGreenNone;
    if ((ia & e.cml) == e.cvl) {
      const uint32_t a = __ldg(l21 + (ia ^ e.fl));
      if (a) r = (a - 2u) | ((uint32_t)__popc(ia & e.sl) << 31);
    }
    tab[(size_t)blockIdx.y * nlow + u] = r;
  }
}

// Off-diagonal entries: sums of conj(v[source]) v[row].  An entry costs a row one coalesced table
// word and one source element (the masks, two lookups and a parity before: 191 us per 16
// entries of all rows of the 14-site half-filled Hubbard sector, 177 us now), and only in
// blocks whose upper half it matches.
template <typename T>
__global__ void __launch_bounds__(kGreenThreads, 2) green_block_kernel(const SectorBlock *__restrict__ pieces, int npieces,
                                                                       int nlow, const uint32_t *__restrict__ tab,
                                                                       const uint32_t *__restrict__ l22,
                                                                       const GreenHalfBatch<kGreenAcc / GreenWidth<T>::w> batch,
                                                                       const T *__restrict__ v, SumOut so) {
  constexpr int NB = kGreenAcc / GreenWidth<T>::w;
  constexpr int U = 2, KB = sizeof(T) == 8 ? 8 : 4;  // rows per lane and entries in flight
  const int lane = threadIdx.x & 31, nwarps = (int)(gridDim.x * kGreenThreads) >> 5;
  double acc[kGreenAcc];
#pragma unroll
  for (int q = 0; q < kGreenAcc; q++) acc[q] = 0.0;
  for (int t = (int)(blockIdx.x * kGreenThreads + threadIdx.x) >> 5; t < npieces; t += nwarps) {
    const uint4 pc = __ldg(reinterpret_cast<const uint4 *>(pieces) + t);
    const uint32_t ib = pc.x;
    const int n = (int)pc.w;
    uint32_t hb[NB], on = 0, neg = 0;
#pragma unroll
    for (int k = 0; k < NB; k++) {
      const GreenHalf &e = batch.t[k];
      hb[k] = (ib & e.cmh) == e.cvh ? __ldg(l22 + (ib ^ e.fh)) : 0u;  // first row of the source block + 1
      on |= (hb[k] != 0u ? 1u : 0u) << k;
      neg |= ((uint32_t)__popc(ib & e.sh) & 1u) << k;
    }
    const T *vp = v + pc.y;
    const uint32_t *tp = tab + pc.z;
    for (int a0 = lane; a0 < n; a0 += 32 * U) {
      T x[U];
#pragma unroll
      for (int q = 0; q < U; q++) x[q] = a0 + 32 * q < n ? vp[a0 + 32 * q] : VT<T>::zero();
#pragma unroll
      for (int k0 = 0; k0 < NB; k0 += KB) {  // KB entries at a time: their table words, then their sources
        if (!((on >> k0) & ((1u << KB) - 1u))) continue;
        uint32_t w[KB][U];
        T y[KB][U];
#pragma unroll
        for (int k = 0; k < KB; k++)
#pragma unroll
          for (int q = 0; q < U; q++)
            w[k][q] = (((on >> (k0 + k)) & 1u) && a0 + 32 * q < n) ? __ldg(tp + (size_t)(k0 + k) * nlow + a0 + 32 * q) : kGreenNone;
#pragma unroll
        for (int k = 0; k < KB; k++)
#pragma unroll
          for (int q = 0; q < U; q++) {
            y[k][q] = VT<T>::zero();
            if ((w[k][q] & kGreenNone) != kGreenNone) y[k][q] = ldg_vec(v + (hb[k0 + k] - 1u + (w[k][q] & kGreenNone)));
          }
#pragma unroll
        for (int k = 0; k < KB; k++)
#pragma unroll
          for (int q = 0; q < U; q++)
            if ((w[k][q] & kGreenNone) != kGreenNone)
              green_acc<T>(acc, k0 + k, ((w[k][q] >> 31) ^ (neg >> (k0 + k))) & 1u ? -1.0 : 1.0, y[k][q], x[q]);
      }
    }
  }
  grid_sum<kGreenAcc>(acc, so);
}

// Diagonal entries (no flip) are sums of |v|^2 over the rows they match.  Their lower halves are
// few (the density-density functions of 28 modes: 106 patterns for 406 entries), so the rows are
// summed per pattern and piece, and each entry then adds the pieces whose upper half it matches.
constexpr int kGreenDiag = 16;
template <typename T, bool SIGN>
__global__ void __launch_bounds__(kGreenThreads, 3) green_diag_kernel(const SectorBlock *__restrict__ pieces, int npieces,
                                                                      const uint32_t *__restrict__ low,
                                                                      const GreenHalfBatch<kGreenDiag> batch, int nb,
                                                                      const T *__restrict__ v, double *__restrict__ sums) {
  const int lane = threadIdx.x & 31, nwarps = (int)(gridDim.x * kGreenThreads) >> 5;
  for (int t = (int)(blockIdx.x * kGreenThreads + threadIdx.x) >> 5; t < npieces; t += nwarps) {
    const uint4 pc = __ldg(reinterpret_cast<const uint4 *>(pieces) + t);
    double acc[kGreenDiag];
#pragma unroll
    for (int q = 0; q < kGreenDiag; q++) acc[q] = 0.0;
#pragma unroll 2
    for (int a = lane; a < (int)pc.w; a += 32) {
      const uint32_t ia = __ldg(low + pc.z + a);
      const double w = VT<T>::abs2(v[pc.y + a]);
#pragma unroll
      for (int k = 0; k < kGreenDiag; k++) {
        const GreenHalf &e = batch.t[k];
        double x = w;
        if (SIGN && (__popc(ia & e.sl) & 1)) x = -w;
        if ((ia & e.cml) == e.cvl) acc[k] += x;
      }
    }
#pragma unroll
    for (int k = 0; k < kGreenDiag; k++) {
      if (k >= nb) break;
      for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_down_sync(0xFFFFFFFFu, acc[k], o);
      if (lane == 0) sums[(size_t)k * npieces + t] = acc[k];
    }
  }
}

// nkeep: patterns held at once (pattern p in place p % nkeep).
// out[e] = sum of pattern pat[e]'s pieces with (ib & cmh) == cvh, signed by the parity of ib & sh.
struct GreenUpper {
  uint32_t cmh, cvh, sh, pat;
};
__global__ void __launch_bounds__(kGreenThreads) green_diag_sum_kernel(const SectorBlock *__restrict__ pieces, int npieces,
                                                                       uint32_t nkeep, const GreenUpper *__restrict__ ent,
                                                                       const double *__restrict__ sums,
                                                                       double *__restrict__ out) {
  const GreenUpper e = ent[blockIdx.x];
  const double *s = sums + (size_t)(e.pat % nkeep) * npieces;
  double v[1] = {0.0};
  for (int t = threadIdx.x; t < npieces; t += kGreenThreads) {
    const uint32_t ib = __ldg(&pieces[t].ib);
    if ((ib & e.cmh) == e.cvh) v[0] += (__popc(ib & e.sh) & 1) ? -s[t] : s[t];
  }
  block_sum<1>(v);
  if (threadIdx.x == 0) out[blockIdx.x] = v[0];
}

// A workspace of the call: the records of a pass and all entries' sums.
struct GreenSpace {
  double *p = nullptr;
  ~GreenSpace() { cudaFree(p); }
};

// Unit entries (coefficient 1) at `nz`, one after another in batches; out: (re, im) per entry.
template <typename T>
int green_batches(Sector *s, const T *d_v, const std::vector<GreenTerm> &nz, std::vector<double> *out) {
  constexpr int W = GreenWidth<T>::w, NB = kGreenAcc / W;
  // the block kernels read whole complex elements; a vector at another address takes the row kernel
  // (as does a sector whose pieces there is no memory for)
  bool blocks = !s->gc && s->lo_bits <= 31 && s->hi_bits <= 31 && whole_elements(W == 2 ? kComplex128 : kReal64, d_v);
  std::string err;
  if (blocks && sector_pieces(s, &err) != 0) {
    cudaGetLastError();
    blocks = false;
  }
  const uint64_t lo_mask = s->ihfbit - 1;
  auto halves = [&](const GreenTerm &t) {
    const int b = s->lo_bits;
    return GreenHalf{(uint32_t)(t.cm & lo_mask), (uint32_t)(t.cv & lo_mask), (uint32_t)(t.flip & lo_mask),
                     (uint32_t)(t.sm & lo_mask), (uint32_t)(t.cm >> b), (uint32_t)(t.cv >> b), (uint32_t)(t.flip >> b),
                     (uint32_t)(t.sm >> b)};
  };
  const GreenHalf none{0, 1, 0, 0, 0, 1, 0, 0};  // matches nothing
  std::vector<int> off, dg;                      // diagonal entries have kernels of their own
  for (int e = 0; e < (int)nz.size(); e++) (blocks && nz[e].flip == 0 ? dg : off).push_back(e);
  std::vector<GreenHalf> pats;
  std::vector<GreenUpper> upper;
  std::map<std::array<uint32_t, 3>, uint32_t> pat_of;
  std::vector<std::pair<uint32_t, int>> by_pat;  // diagonal entries by pattern
  for (int e : dg) {
    const GreenHalf h = halves(nz[e]);
    const auto it = pat_of.emplace(std::array<uint32_t, 3>{h.cml, h.cvl, h.sl}, (uint32_t)pats.size());
    if (it.second) pats.push_back(h);
    by_pat.push_back({it.first->second, e});
  }
  std::sort(by_pat.begin(), by_pat.end());
  for (size_t q = 0; q < dg.size(); q++) {
    const GreenHalf h = halves(nz[by_pat[q].second]);
    dg[q] = by_pat[q].second;
    upper.push_back(GreenUpper{h.cmh, h.cvh, h.sh, by_pat[q].first});
  }
  // off-diagonal entries that move the upper half alike share their source blocks: one batch reads
  // each of them from L2 once and then from L1 (the pieces come class by class for the same reason)
  if (blocks)
    std::stable_sort(off.begin(), off.end(), [&](int x, int y) {
      const GreenHalf p = halves(nz[x]), q = halves(nz[y]);
      return std::array<uint32_t, 3>{p.fh, p.cmh, p.cvh} < std::array<uint32_t, 3>{q.fh, q.cmh, q.cvh};
    });
  const size_t noff = (off.size() + NB - 1) / NB;
  const int grid = blocks ? std::min(s->num_sms * 3, (s->npieces + 7) / 8) : s->red_blocks;
  const int grid_off = blocks ? std::min(grid, s->num_sms * 2) : grid;
  // one workspace: upper halves, a pass's table, the entries' sums, a pass's records and pieces' sums
  const size_t nrec = (size_t)grid * kGreenAcc, nout = noff * kGreenAcc + dg.size();
  const size_t ntab = blocks && noff ? (sizeof(uint32_t) * (size_t)NB * s->nlow + 15) / 16 * 2 : 0;
  // pieces' sums of as many patterns as 128 MB hold, whole passes; of one pass where that is too much
  size_t nkeep = std::max<size_t>(1, ((size_t)1 << 24) / std::max(1, s->npieces) / kGreenDiag) * kGreenDiag;
  const size_t nup = (sizeof(GreenUpper) * upper.size()) / sizeof(double);
  auto bytes = [&]() {
    const size_t nsum = std::min(pats.size(), nkeep) * (size_t)s->npieces;
    return sizeof(double) * std::max<size_t>(1, nrec + nout + nout % 2 + ntab + nup + nsum);
  };
  GreenSpace ws;
  if (cudaMalloc(&ws.p, bytes()) != cudaSuccess) {
    cudaGetLastError();
    nkeep = kGreenDiag;
    if (cudaMalloc(&ws.p, bytes()) != cudaSuccess) {
      set_error("Green's functions: device allocation failed");
      return -1;
    }
  }
  GreenUpper *d_up = reinterpret_cast<GreenUpper *>(ws.p);  // 16-byte units first
  uint32_t *d_tab = reinterpret_cast<uint32_t *>(ws.p + nup);
  double *d_out = ws.p + nup + ntab, *d_rec = d_out + nout + nout % 2, *d_sum = d_rec + nrec;
  for (size_t b = 0; b < noff; b++) {
    const int n0 = (int)b * NB, n = std::min<int>(NB, (int)off.size() - n0);
    const SumOut so = sum_out(d_rec, 0, grid_off, s->d_done, d_out + b * kGreenAcc);
    if (blocks) {
      GreenHalfBatch<NB> batch;
      for (int k = 0; k < NB; k++) batch.t[k] = k < n ? halves(nz[off[n0 + k]]) : none;
      const dim3 tg((unsigned)std::min((s->nlow + kGreenThreads - 1) / kGreenThreads, s->num_sms), n);
      green_table_kernel<NB><<<tg, kGreenThreads, 0, s->stream>>>(s->nlow, s->d_low, s->d_list_2_1, batch, d_tab);
      green_block_kernel<T><<<grid_off, kGreenThreads, 0, s->stream>>>(s->d_pieces, s->npieces, s->nlow, d_tab, s->d_list_2_2,
                                                                   batch, d_v, so);
      continue;
    }
    GreenBatch<NB> batch;
    for (int k = 0; k < NB; k++) batch.t[k] = k < n ? nz[off[n0 + k]] : GreenTerm{0, 1, 0, 0, 0.0, 0.0};
#define HPHI_GREEN_LAUNCH(GCV, CW)                                                                          \
  green_kernel<T, GCV, CW><<<grid, kGreenThreads, 0, s->stream>>>(s->dim, s->d_list_1, s->d_list_2_1,       \
                                                                  s->d_list_2_2, s->lo_bits, lo_mask, batch, \
                                                                  d_v, so)
    const bool narrow = s->model.nbits <= 32;
    if (s->gc) {
      if (narrow) HPHI_GREEN_LAUNCH(true, uint32_t);
      else HPHI_GREEN_LAUNCH(true, uint64_t);
    } else {
      HPHI_GREEN_LAUNCH(false, uint64_t);
    }
#undef HPHI_GREEN_LAUNCH
  }
  bool ok = true;
  if (!dg.empty()) {
    ok = cudaMemcpyAsync(d_up, upper.data(), sizeof(GreenUpper) * upper.size(), cudaMemcpyHostToDevice, s->stream) == cudaSuccess;
    size_t q0 = 0;
    for (size_t p0 = 0; p0 < pats.size(); p0 += kGreenDiag) {
      const int n = (int)std::min<size_t>(kGreenDiag, pats.size() - p0);
      GreenHalfBatch<kGreenDiag> batch;
      for (int k = 0; k < kGreenDiag; k++) batch.t[k] = k < n ? pats[p0 + k] : none;
      bool sign = false;  // sign masks outside the condition
      for (int k = 0; k < n; k++) sign = sign || batch.t[k].sl != 0;
      double *at = d_sum + (p0 % nkeep) * s->npieces;
      if (sign)
        green_diag_kernel<T, true><<<grid, kGreenThreads, 0, s->stream>>>(s->d_pieces, s->npieces, s->d_low, batch, n, d_v, at);
      else
        green_diag_kernel<T, false><<<grid, kGreenThreads, 0, s->stream>>>(s->d_pieces, s->npieces, s->d_low, batch, n, d_v, at);
      if ((p0 + kGreenDiag) % nkeep != 0 && p0 + kGreenDiag < pats.size()) continue;
      size_t q1 = q0;  // the entries of these patterns
      while (q1 < dg.size() && by_pat[q1].first < p0 + n) q1++;
      green_diag_sum_kernel<<<(unsigned)(q1 - q0), kGreenThreads, 0, s->stream>>>(
          s->d_pieces, s->npieces, (uint32_t)nkeep, d_up + q0, d_sum, d_out + noff * kGreenAcc + q0);
      q0 = q1;
    }
  }
  std::vector<double> h(nout);
  if (!ok || cudaGetLastError() != cudaSuccess ||
      cudaMemcpyAsync(h.data(), d_out, sizeof(double) * nout, cudaMemcpyDeviceToHost, s->stream) != cudaSuccess ||
      cudaStreamSynchronize(s->stream) != cudaSuccess) {
    set_error("Green's function kernels failed");
    return -1;
  }
  out->assign(2 * nz.size(), 0.0);
  for (size_t q = 0; q < off.size(); q++) {
    const double *rec = h.data() + (q / NB) * kGreenAcc + W * (q % NB);
    (*out)[2 * off[q]] = rec[0];
    (*out)[2 * off[q] + 1] = W == 2 ? rec[1] : 0.0;
  }
  for (size_t q = 0; q < dg.size(); q++) (*out)[2 * dg[q]] = h[noff * kGreenAcc + q];
  return 0;
}

__global__ void imag_check_kernel(int64_t n, const cplx *__restrict__ v, double *__restrict__ re,
                                  int *__restrict__ complex_flag) {
  bool nz = false;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const cplx z = v[i];
    re[i] = z.x;
    nz = nz || z.y != 0.0;
  }
  if (__any_sync(0xffffffffu, nz) && (threadIdx.x & 31) == 0) *complex_flag = 1;
}

}  // namespace

int green_stage_host_vector(Sector *s, const double *h_v_1based, void **d_vec, VecType *vt) {
  const int64_t n = s->dim;
  cplx *dc = nullptr;
  double *dr = nullptr;
  int *flag = nullptr;
  if (cudaMalloc(&dc, sizeof(cplx) * (size_t)n) != cudaSuccess || cudaMalloc(&dr, sizeof(double) * (size_t)n) != cudaSuccess ||
      cudaMalloc(&flag, sizeof(int)) != cudaSuccess) {
    cudaFree(dc);
    cudaFree(dr);
    set_error("Green's functions: device allocation failed");
    return -1;
  }
  int h_flag = 0;
  bool ok = cudaMemsetAsync(flag, 0, sizeof(int), s->stream) == cudaSuccess &&
            cudaMemcpyAsync(dc, h_v_1based + 2, sizeof(cplx) * (size_t)n, cudaMemcpyHostToDevice, s->stream) == cudaSuccess;
  if (ok) {
    imag_check_kernel<<<s->red_blocks, 256, 0, s->stream>>>(n, dc, dr, flag);
    ok = cudaGetLastError() == cudaSuccess &&
         cudaMemcpyAsync(&h_flag, flag, sizeof(int), cudaMemcpyDeviceToHost, s->stream) == cudaSuccess &&
         cudaStreamSynchronize(s->stream) == cudaSuccess;
  }
  cudaFree(flag);
  if (!ok) {
    cudaFree(dc);
    cudaFree(dr);
    set_error("Green's functions: staging the vector failed");
    return -1;
  }
  if (h_flag) {  // complex: keep the complex copy
    cudaFree(dr);
    *d_vec = dc;
    *vt = kComplex128;
  } else {       // real: the real parts, gathered by the same pass
    cudaFree(dc);
    *d_vec = dr;
    *vt = kReal64;
  }
  return 0;
}

// The requested entries as multiples of few unit ones.  Sign bits inside the condition mask have
// fixed values and go into the factor; then equal masks are one entry, and the adjoint of an
// entry (the same masks, the condition after the flip) is its complex conjugate.  All one-body
// functions of N sites need half as many passes, as do density-density ones.
int green_expect(Sector *s, VecType vt, const void *d_v, const std::vector<GreenTerm> &terms,
                 std::vector<double> *out) {
  out->assign(2 * terms.size(), 0.0);
  struct Use {
    int e, unit;
    double f;
    bool conj;
  };
  std::vector<Use> uses;
  std::vector<GreenTerm> unit;
  std::map<std::array<uint64_t, 4>, int> at;
  for (size_t e = 0; e < terms.size(); e++) {
    GreenTerm t = terms[e];
    if (t.coef == 0.0) continue;
    const double f = (__builtin_popcountll(t.cv & t.sm) & 1) ? -t.coef : t.coef;
    t.sm &= ~t.cm;
    t.coef = 1.0;
    bool conj = false;
    int u = -1;
    const auto it = at.find({t.cm, t.cv, t.flip, t.sm});
    if (it != at.end()) {
      u = it->second;
    } else if (t.flip && (t.flip & ~t.cm) == 0) {
      const auto adj = at.find({t.cm, t.cv ^ t.flip, t.flip, t.sm});
      if (adj != at.end()) {
        u = adj->second;
        conj = true;
      }
    }
    if (u < 0) {
      u = (int)unit.size();
      at[{t.cm, t.cv, t.flip, t.sm}] = u;
      unit.push_back(t);
    }
    uses.push_back(Use{(int)e, u, f, conj});
  }
  if (unit.empty()) return 0;
  if (cudaSetDevice(s->device) != cudaSuccess) {
    set_error("cudaSetDevice failed");
    return -1;
  }
  std::vector<double> val;
  const int rc = vt == kReal64 ? green_batches<double>(s, (const double *)d_v, unit, &val)
                               : green_batches<cplx>(s, (const cplx *)d_v, unit, &val);
  if (rc != 0) return -1;
  for (const Use &u : uses) {
    (*out)[2 * u.e] = u.f * val[2 * u.unit];
    (*out)[2 * u.e + 1] = (u.conj ? -u.f : u.f) * val[2 * u.unit + 1];
  }
  return 0;
}

}  // namespace hphi
