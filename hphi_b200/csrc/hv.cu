// Matrix-free H*v, general path: every off-diagonal term in gather form.
//
// Replaces mltply (src/mltply.c:56-132) and the term passes it dispatches to
// (mltplyHubbard / mltplyHubbardGC, src/mltplyHubbard.c:150-528; mltplyHalfSpin /
// mltplyHalfSpinGC, src/mltplySpin.c:192-703).  The reference makes one full pass over
// the vector per term and scatters v0[off(j)] += c * v1[j]; here each output row is
// owned by one thread, which walks the compiled terms once, tests the row's
// configuration against each term's pattern, and gathers the matching source element:
//   s = c ^ flip,  row(s) = list_2_1[s & (ihfbit-1)] + list_2_2[s >> lo_bits] - 3,
//   sign = (-1)^popcount(c & sign_mask)            (GetOffComp / SgnBit, src/bitcalc.c).
// Output rows are written exactly once, so there are no races and no atomics, and the
// fused <v1|H|v1> of the reference (X->Large.prdct) comes from a block reduction of
// conj(v1[r]) * (H v1)[r].
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/hphi_b200.h"
#include "device_util.cuh"
#include "engine.hpp"
#include "hv_blocks.hpp"
#include "hv_gc.hpp"
#include "hv_hubbard.hpp"
#include "hv_product.hpp"
#include "hv_rowblock.hpp"
#include "split.cuh"

namespace hphi {
namespace {

constexpr int kHvThreads = 256;
constexpr int kSmemTermMax = 1024;  // 48 KiB of BitTerm

// Eight blocks per SM for real vectors (32 registers): the grid is 8 blocks per SM, and at 40
// registers a second wave took the 24-site chain's H*v from 146 to 187 us.
template <typename T, bool GC, bool SMEM>
__global__ void __launch_bounds__(kHvThreads, sizeof(T) == 8 ? 8 : 4) hv_general_kernel(
    int64_t dim, const uint64_t *__restrict__ list_1, const uint32_t *__restrict__ l21,
    const uint32_t *__restrict__ l22, int lo_bits, uint64_t lo_mask, SplitView split,
    const BitTerm *__restrict__ gterms, int nterms, const double *__restrict__ diag, const T *__restrict__ v1,
    T *__restrict__ v0, const double *__restrict__ coef, SumOut so) {
  const double acc = coef[0], scale = coef[1];
  extern __shared__ BitTerm sterms[];
  const BitTerm *terms = gterms;
  if (SMEM) {
    for (int k = threadIdx.x; k < nterms; k += blockDim.x) sterms[k] = gterms[k];
    __syncthreads();
    terms = sterms;
  }
  double pr[2] = {0.0, 0.0};
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < dim; r += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t c = GC ? (uint64_t)r : list_1[r];
    const T x = v1[r];
    T y = VT<T>::scale(diag[r], x);
    if (split.lo_ptr) y = split_terms<T, GC>(split, c, r, lo_bits, lo_mask, l22, [&](int64_t j) { return v1[j]; }, y);
    for (int k = 0; k < nterms; k++) {
      const BitTerm t = terms[k];
      if ((c & t.cm) != t.cv) continue;
      const uint64_t src = c ^ t.flip;
      int64_t j;
      if (GC) {
        j = (int64_t)src;
      } else {
        const uint32_t a = l21[src & lo_mask];
        const uint32_t b = l22[src >> lo_bits];
        if (a == 0u || b == 0u) continue;
        j = (int64_t)a + (int64_t)b - 3;
      }
      const double sg = (__popcll(c & t.sm) & 1) ? -t.re : t.re;
      const double sgi = (__popcll(c & t.sm) & 1) ? -t.im : t.im;
      y = VT<T>::add(y, VT<T>::cmul_re_im(sg, sgi, v1[j]));
    }
    pr[0] += VT<T>::conj_mul_re(x, y);
    pr[1] += VT<T>::conj_mul_im(x, y);
    y = VT<T>::scale(scale, y);
    v0[r] = (acc == 0.0) ? y : VT<T>::add(VT<T>::scale(acc, v0[r]), y);
  }
  grid_sum<2>(pr, so);
}

template <typename T, bool GC>
void launch_general(Sector *s, const T *v1, T *v0, const double *coef, const SumOut &so) {
  const int grid = s->red_blocks;
  const uint64_t lo_mask = s->ihfbit - 1;
  const SplitView sv = split_view(s->split);
  if (s->split.ngen <= kSmemTermMax) {
    const size_t smem = sizeof(BitTerm) * (size_t)s->split.ngen;
    hv_general_kernel<T, GC, true><<<grid, kHvThreads, smem, s->stream>>>(
        s->dim, s->d_list_1, s->d_list_2_1, s->d_list_2_2, s->lo_bits, lo_mask, sv, s->split.gen, s->split.ngen,
        s->d_diag, v1, v0, coef, so);
  } else {
    hv_general_kernel<T, GC, false><<<grid, kHvThreads, 0, s->stream>>>(
        s->dim, s->d_list_1, s->d_list_2_1, s->d_list_2_2, s->lo_bits, lo_mask, sv, s->split.gen, s->split.ngen,
        s->d_diag, v1, v0, coef, so);
  }
}

// B vectors at once (independent samples of one sector, vector b at v + b * stride): the
// configuration, diagonal, split-plan entries, list lookups and signs of a row are worked out once
// and applied to all B.  Per vector the arithmetic and its order are the general kernel's, so every
// output equals a separate launch bit for bit.  Coefficients (acc, scale) of vector b at coef + b *
// cstride.  No sums: the callers' next sweep over the vectors has them.
template <typename T, int B>
struct Blk {
  T v[B];
};

template <typename T, int B>
struct BlkOps {
  static __device__ __forceinline__ Blk<T, B> add(Blk<T, B> a, const Blk<T, B> &b) {
#pragma unroll
    for (int q = 0; q < B; q++) a.v[q] = VT<T>::add(a.v[q], b.v[q]);
    return a;
  }
  static __device__ __forceinline__ Blk<T, B> cmul_re_im(double re, double im, const Blk<T, B> &x) {
    Blk<T, B> r;
#pragma unroll
    for (int q = 0; q < B; q++) r.v[q] = VT<T>::cmul_re_im(re, im, x.v[q]);
    return r;
  }
};

template <typename T, bool GC, bool SMEM, int B>
__global__ void __launch_bounds__(kHvThreads) hv_block_kernel(
    int64_t dim, int64_t stride, const uint64_t *__restrict__ list_1, const uint32_t *__restrict__ l21,
    const uint32_t *__restrict__ l22, int lo_bits, uint64_t lo_mask, SplitView split,
    const BitTerm *__restrict__ gterms, int nterms, const double *__restrict__ diag, const T *__restrict__ v1,
    T *__restrict__ v0, const double *__restrict__ coef, int cstride) {
  extern __shared__ BitTerm sterms[];
  const BitTerm *terms = gterms;
  if (SMEM) {
    for (int k = threadIdx.x; k < nterms; k += blockDim.x) sterms[k] = gterms[k];
    __syncthreads();
    terms = sterms;
  }
  auto load = [&](int64_t j) {
    Blk<T, B> z;
#pragma unroll
    for (int q = 0; q < B; q++) z.v[q] = v1[q * stride + j];
    return z;
  };
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < dim; r += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t c = GC ? (uint64_t)r : list_1[r];
    const Blk<T, B> x = load(r);
    const double dg = diag[r];
    Blk<T, B> y;
#pragma unroll
    for (int q = 0; q < B; q++) y.v[q] = VT<T>::scale(dg, x.v[q]);
    if (split.lo_ptr) {
      // split_terms with the block accumulator (same entries, same order)
      const uint32_t ia = (uint32_t)(c & lo_mask);
      const uint64_t ib = c >> lo_bits;
      const int64_t base = GC ? (int64_t)(c & ~lo_mask) : (int64_t)__ldg(l22 + ib) - 3;
      const uint32_t nl = __ldg(split.lo_ptr + ia);
      const uint32_t *le = split.lo_ent + ia;
      for (uint32_t e = 0; e < nl; e++, le += split.lo_stride) {
        const uint32_t v = __ldg(le);
        const uint32_t tgt = v & ((1u << kSplitTargetBits) - 1u);
        const uint32_t k = v >> kSplitTargetBits;
        const int64_t j = GC ? (base | (int64_t)tgt) : base + (int64_t)tgt;
        const double2 cf = __ldg(reinterpret_cast<const double2 *>(split.coef) + k);
        y = BlkOps<T, B>::add(y, BlkOps<T, B>::cmul_re_im(cf.x, cf.y, load(j)));
      }
      const uint32_t h0 = __ldg(split.hi_ptr + ib), h1 = __ldg(split.hi_ptr + ib + 1);
      for (uint32_t e = h0; e < h1; e++) {
        const HiEnt h = split.hi_ent[e];
        const int64_t j = GC ? (int64_t)((uint64_t)r ^ (uint64_t)h.delta) : r + h.delta;
        const double2 cf = __ldg(reinterpret_cast<const double2 *>(split.coef) + h.k);
        y = BlkOps<T, B>::add(y, BlkOps<T, B>::cmul_re_im(cf.x, cf.y, load(j)));
      }
    }
    for (int k = 0; k < nterms; k++) {
      const BitTerm t = terms[k];
      if ((c & t.cm) != t.cv) continue;
      const uint64_t src = c ^ t.flip;
      int64_t j;
      if (GC) {
        j = (int64_t)src;
      } else {
        const uint32_t a = l21[src & lo_mask];
        const uint32_t b = l22[src >> lo_bits];
        if (a == 0u || b == 0u) continue;
        j = (int64_t)a + (int64_t)b - 3;
      }
      const double sg = (__popcll(c & t.sm) & 1) ? -t.re : t.re;
      const double sgi = (__popcll(c & t.sm) & 1) ? -t.im : t.im;
      y = BlkOps<T, B>::add(y, BlkOps<T, B>::cmul_re_im(sg, sgi, load(j)));
    }
#pragma unroll
    for (int q = 0; q < B; q++) {
      const double acc = coef[q * cstride], scale = coef[q * cstride + 1];
      const T yq = VT<T>::scale(scale, y.v[q]);
      T *o = v0 + q * stride + r;
      *o = (acc == 0.0) ? yq : VT<T>::add(VT<T>::scale(acc, *o), yq);
    }
  }
}

template <typename T, bool GC, int B>
void launch_block(Sector *s, int64_t stride, const T *v1, T *v0, const double *coef, int cstride) {
  const int grid = s->red_blocks;
  const uint64_t lo_mask = s->ihfbit - 1;
  const SplitView sv = split_view(s->split);
  if (s->split.ngen <= kSmemTermMax) {
    const size_t smem = sizeof(BitTerm) * (size_t)s->split.ngen;
    hv_block_kernel<T, GC, true, B><<<grid, kHvThreads, smem, s->stream>>>(
        s->dim, stride, s->d_list_1, s->d_list_2_1, s->d_list_2_2, s->lo_bits, lo_mask, sv, s->split.gen,
        s->split.ngen, s->d_diag, v1, v0, coef, cstride);
  } else {
    hv_block_kernel<T, GC, false, B><<<grid, kHvThreads, 0, s->stream>>>(
        s->dim, stride, s->d_list_1, s->d_list_2_1, s->d_list_2_2, s->lo_bits, lo_mask, sv, s->split.gen,
        s->split.ngen, s->d_diag, v1, v0, coef, cstride);
  }
}

template <typename T, bool GC>
void launch_block_n(Sector *s, int nb, int64_t stride, const T *v1, T *v0, const double *coef, int cstride) {
  switch (nb) {
    case 1: launch_block<T, GC, 1>(s, stride, v1, v0, coef, cstride); break;
    case 2: launch_block<T, GC, 2>(s, stride, v1, v0, coef, cstride); break;
    case 3: launch_block<T, GC, 3>(s, stride, v1, v0, coef, cstride); break;
    case 4: launch_block<T, GC, 4>(s, stride, v1, v0, coef, cstride); break;
    case 5: launch_block<T, GC, 5>(s, stride, v1, v0, coef, cstride); break;
    case 6: launch_block<T, GC, 6>(s, stride, v1, v0, coef, cstride); break;
    case 7: launch_block<T, GC, 7>(s, stride, v1, v0, coef, cstride); break;
    default: launch_block<T, GC, 8>(s, stride, v1, v0, coef, cstride); break;
  }
}

}  // namespace

bool hv_block_applies(const Sector *s, VecType vt) {
  return !s->prod && !s->hub && !rb_applies(s, vt) && !(vt == kReal64 && s->model.complex_terms);
}

bool tpq_lockstep(const Sector *s, VecType vt) {
  if (!hv_block_applies(s, vt)) return false;
  const bool tiles = gc_applies(s, vt);
  if (s->model.num_ave == 1 && (tiles || bk_applies(s))) return false;
  return !tiles || s->dim < ((int64_t)1 << 24);
}

int hv_block_native(Sector *s, VecType vt, int nb, int64_t stride, const void *d_v1, void *d_v0,
                    const double *d_coef, int cstride) {
  if (nb < 1 || nb > kHvBlockMax || !hv_block_applies(s, vt)) {
    set_error("hv_block_native: block products need HPhi's row order and 1..8 vectors");
    return -1;
  }
  if (vt == kReal64) {
    if (s->gc) launch_block_n<double, true>(s, nb, stride, (const double *)d_v1, (double *)d_v0, d_coef, cstride);
    else launch_block_n<double, false>(s, nb, stride, (const double *)d_v1, (double *)d_v0, d_coef, cstride);
  } else {
    if (s->gc) launch_block_n<cplx, true>(s, nb, stride, (const cplx *)d_v1, (cplx *)d_v0, d_coef, cstride);
    else launch_block_n<cplx, false>(s, nb, stride, (const cplx *)d_v1, (cplx *)d_v0, d_coef, cstride);
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error(std::string("block hv launch failed: ") + cudaGetErrorString(e));
    return -1;
  }
  return 0;
}

HvRoute hv_route(const Sector *s, VecType vt, const void *d_v1) {
  const bool whole = whole_elements(vt, d_v1);
  if (whole && gc_applies(s, vt)) return kRouteTile;
  if (rb_applies(s, vt) && (whole || rb_own_rows(s, vt))) return kRouteRowBlock;
  if (whole && bk_applies(s)) return kRouteBlock;
  return kRouteGeneral;
}

HvPlan hv_plan(const Sector *s, VecType vt) {
  if (s->prod) {
    const int row = prod_row_words(s);
    return row ? HvPlan{HPHI_HV_TWO_PASS, 2, row} : HvPlan{HPHI_HV_ONE_PASS, 2, 0};
  }
  if (s->hub) return HvPlan{HPHI_HV_HUBBARD_BLOCK, 3, 0};
  switch (hv_route(s, vt, nullptr)) {
    case kRouteTile: return HvPlan{HPHI_HV_TILE, gc_passes(s, vt), 0};
    case kRouteRowBlock: return HvPlan{HPHI_HV_ROWBLOCK, 2, bk_row_pass(s) ? 1 : 0};
    case kRouteBlock: return HvPlan{HPHI_HV_BLOCK, 1, bk_shape(s)};
    case kRouteGeneral: break;
  }
  return HvPlan{HPHI_HV_GENERAL, 1, 0};
}

int hv_launch_scratch(Sector *s, VecType vt, const void *d_v1, void *d_v0, const double *d_coef, double *d_out,
                      double *d_part, const LanczosTail *lt) {
  if (vt == kReal64 && s->model.complex_terms) {
    set_error("H has complex coefficients: real vectors are not allowed");
    return -1;
  }
  switch (hv_route(s, vt, d_v1)) {
    case kRouteTile: return gc_hv_launch(s, vt, d_v1, d_v0, d_coef, d_out, d_part, lt);
    case kRouteRowBlock: return rb_hv_launch_scratch(s, vt, d_v1, d_v0, d_coef, d_out, d_part, lt);
    case kRouteBlock: return bk_hv_launch(s, vt, d_v1, d_v0, d_coef, d_out, d_part, lt);
    case kRouteGeneral: break;
  }
  const SumOut so = sum_out(d_part, 0, s->red_blocks, s->d_done, d_out, 0, lt);
  if (vt == kReal64) {
    if (s->gc) launch_general<double, true>(s, (const double *)d_v1, (double *)d_v0, d_coef, so);
    else launch_general<double, false>(s, (const double *)d_v1, (double *)d_v0, d_coef, so);
  } else {
    if (s->gc) launch_general<cplx, true>(s, (const cplx *)d_v1, (cplx *)d_v0, d_coef, so);
    else launch_general<cplx, false>(s, (const cplx *)d_v1, (cplx *)d_v0, d_coef, so);
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error(std::string("hv launch failed: ") + cudaGetErrorString(e));
    return -1;
  }
  return 0;
}

int hv_launch(Sector *s, VecType vt, const void *d_v1, void *d_v0, const double *d_coef, double *d_out,
              const LanczosTail *lt) {
  const HvRoute route = hv_route(s, vt, d_v1);
  double *part = route == kRouteTile ? gc_part(s) : route == kRouteRowBlock ? rb_part(s) : s->d_red;
  return hv_launch_scratch(s, vt, d_v1, d_v0, d_coef, d_out, part, lt);
}

size_t hv_scratch_doubles(const Sector *s, VecType vt) {
  if (s->prod) return prod_scratch_doubles(s, vt);
  if (s->hub) return hub_scratch_doubles(s);
  size_t n = 2 * (size_t)s->red_blocks;  // the general kernel, which an unaligned vector takes
  if (gc_applies(s, vt)) n = std::max(n, gc_scratch_doubles(s, vt));
  if (rb_applies(s, vt)) n = std::max(n, rb_scratch_doubles(s));
  if (bk_applies(s)) n = std::max(n, bk_scratch_doubles(s));
  return n;
}

int hv_native_scratch(Sector *s, VecType vt, const void *d_v1, void *d_v0, const double *d_coef, double *d_out,
                      double *d_part, int *d_counter) {
  if (s->prod) return prod_hv_launch_scratch(s, vt, d_v1, d_v0, d_coef, d_out, d_part, d_counter);
  if (s->hub) return hub_hv_launch_scratch(s, vt, d_v1, d_v0, d_coef, d_out, d_part, d_counter);
  return hv_launch_scratch(s, vt, d_v1, d_v0, d_coef, d_out, d_part, nullptr);
}

bool has_native_order(const Sector *s) { return s->hub != nullptr || s->prod != nullptr; }

int hv_native(Sector *s, VecType vt, const void *d_v1, void *d_v0, const double *d_coef, double *d_out,
              bool acc_read, const LanczosTail *lt) {
  if (s->prod) return prod_hv_launch(s, vt, d_v1, d_v0, d_coef, d_out, lt);
  if (s->hub) {
    if (hub_hv_launch(s, vt, d_v1, d_v0, d_coef, d_out, acc_read) != 0) return -1;
    return lt ? lanczos_scalars(s, 0, lt->k, lt->st, lt->alpha, lt->beta) : 0;
  }
  return hv_launch(s, vt, d_v1, d_v0, d_coef, d_out, lt);
}

int to_native(Sector *s, VecType vt, const void *in, void *out) {
  if (s->prod) return prod_permute(s, vt, in, out, true);
  if (s->hub) return hub_permute(s, vt, in, out, true);
  const size_t esz = (vt == kReal64) ? sizeof(double) : sizeof(cplx);
  if (in != out && cudaMemcpyAsync(out, in, esz * (size_t)s->dim, cudaMemcpyDeviceToDevice, s->stream) != cudaSuccess) {
    set_error("to_native: copy failed");
    return -1;
  }
  return 0;
}

int from_native(Sector *s, VecType vt, const void *in, void *out) {
  if (s->prod) return prod_permute(s, vt, in, out, false);
  if (s->hub) return hub_permute(s, vt, in, out, false);
  const size_t esz = (vt == kReal64) ? sizeof(double) : sizeof(cplx);
  if (in != out && cudaMemcpyAsync(out, in, esz * (size_t)s->dim, cudaMemcpyDeviceToDevice, s->stream) != cudaSuccess) {
    set_error("from_native: copy failed");
    return -1;
  }
  return 0;
}

int native_observables(Sector *s, VecType vt, const void *v, double *d_out) {
  if (s->prod) return prod_observables(s, vt, v, d_out);
  if (s->hub) return hub_observables(s, vt, v, d_out);
  return vec_diag_observables(s, vt, v, d_out);
}

}  // namespace hphi
