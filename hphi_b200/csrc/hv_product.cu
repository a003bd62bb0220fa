// Product-layout kernel for canonical Hubbard Hamiltonians.
//
// Applies when every off-diagonal term is a spin-conserving single hop c+_{i s} c_{j s}
// (Trans terms, src/mltplyHubbard.c:174-209, element routine CisAjt,
// src/mltplyHubbardCore.c:305-347), Nsite <= 16 and both spin counts are fixed; diagonal
// terms of any kind are allowed (src/diagonalcalc.c).
//
// Native vector order.  The sector of HPhi (Nup up and Ndown down electrons) is the set
// of pairs (u, d) of N-bit occupations with popcount Nup and Ndown.  The native order
// stores it as a dense matrix
//   pos = rank(u) * C(N, Ndown) + rank(d),
// ranks among N-bit numbers of equal popcount in increasing order, in the species-first
// fermion basis (all up modes before all down modes).  That basis differs from HPhi's
// interleaved one (bit 2i + s) by the diagonal sign
//   sigma(c) = (-1)^#{(down at i, up at j) : i < j},
// applied by the boundary permutation; in it a hop's sign only counts occupied modes of its
// own species strictly between its two sites, so it is a property of u (up hops) or d
// (down hops) alone:
//   (H v)[u, d] = D(u, d) v[u, d] + sum_{down hops} c(d) v[u, d'] + sum_{up hops} c(u) v[u', d].
//
// Two passes: a row pass (diagonal + down hops: every row is a gather inside itself) and a column
// pass (up hops: whole source rows), for real and complex vectors and any coefficients that fall
// into at most kMaxGroups values up to sign.  The row pass stages rows in shared memory (a complex
// row as its two planes) and reads them through an edge-coloured gather table per coefficient:
// within each slot of a warp, the 16 lanes of a half-warp hit 16 different shared-memory bank
// pairs, so every 8-byte gather takes the minimum two wavefronts; entries are 16-bit word indices
// with the hop's sign in bit 15, eight per lane in one 16-byte load, and empty slots point at zero
// words placed one per bank.  The column pass walks the matrix in column chunks (all rows of chunk
// 0, then chunk 1, ...) so the source rows of the chunk being processed stay in L2 while every row
// gathers its ~N/2 up-hop sources.  Both passes take their work by static striding and keep
// per-CTA partial sums of <v1|H v1>; the last CTA of the column pass adds them up in order.
//
// One pass (no down hops, more coefficients than groups, or HPHI_B200_PROD=single): persistent
// CTAs take whole rows u from an atomic dispenser; down hops are gathers inside the staged row
// driven by an ELL table ell_dn[slot][d] (source rank, coefficient index), up hops coalesced reads
// of the source rows; each row's <v1|H v1> is reduced in the CTA and summed over rows afterwards.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <string>
#include <type_traits>
#include <vector>

#include "device_util.cuh"
#include "engine.hpp"
#include "gather_table.hpp"
#include "host_parallel.hpp"
#include "hv_product.hpp"
#include "tma.cuh"

namespace hphi {
namespace {

constexpr int kProdThreads = 512;
constexpr int kMaxUpWidth = 128;          // up hops of one row, staged in shared memory
constexpr uint32_t kEllNone = 0xFFFFFFFFu;

struct ProdArgs {
  int N, Uc, Dc;               // sites, rows (up configurations), columns (down configurations)
  int wd, wu;                  // ELL widths
  const uint16_t *rank;        // [2^N] position of an up configuration (its rank)
  const uint16_t *pos_dn;      // [2^N] position of a down configuration
  const uint16_t *unrank_up;   // [Uc]
  const uint16_t *unrank_dn;   // [Dc]
  const uint32_t *ell_dn;      // [wd][Dc]: source rank | coefficient index << 16
  const uint32_t *ell_up;      // [Uc][wu]
  const uint8_t *cnt_dn;       // [Dc] valid entries of each ELL column
  const uint8_t *wmax_dn;      // [ceil(Dc / 32)] largest count in each aligned block of 32 columns
  const double *utab;          // [17] u0 * k for k = 0..16 (cross_mode 0)
  const double2 *cf_dn, *cf_up;
  const double *du, *dd;       // diagonal terms of one species, by rank
  const double *usite;         // on-site U per site (cross_mode 1)
  double u0;                   // uniform on-site U (cross_mode 0)
  int cross_mode;              // 0: u0 * popc(u & d); 1: per-site U; 2: read dfull
  const double *dfull;         // [Uc * Dc] diagonal in native order (cross_mode 2)
  const int *order;            // [Uc] processing order of the rows
};

template <typename T> __device__ __forceinline__ T ldg_v(const T *p);
template <> __device__ __forceinline__ double ldg_v<double>(const double *p) { return __ldg(p); }
template <> __device__ __forceinline__ cplx ldg_v<cplx>(const cplx *p) {
  const double2 v = __ldg(reinterpret_cast<const double2 *>(p));
  return cplx{v.x, v.y};
}

__device__ __forceinline__ int next_row(int *counter) {
  __shared__ int s_row;
  __syncthreads();
  if (threadIdx.x == 0) s_row = atomicAdd(counter, 1);
  __syncthreads();
  return s_row;
}

// The last CTA to leave resets the dispenser for the next launch.
__device__ __forceinline__ void retire(int *counter) {
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(counter + 1, 1) == (int)gridDim.x - 1) {
      counter[0] = 0;
      counter[1] = 0;
      __threadfence();
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kProdThreads, 2) prod_hv_kernel(ProdArgs a, const T *__restrict__ v1,
                                                                    T *__restrict__ v0,
                                                                    const double *__restrict__ coef,
                                                                    double *__restrict__ part, int *counter) {
  extern __shared__ unsigned char smem_raw[];
  T *row = reinterpret_cast<T *>(smem_raw);
  __shared__ uint32_t s_src[kMaxUpWidth];
  __shared__ double2 s_cf[kMaxUpWidth];
  __shared__ int s_nu;
  const double acc = coef[0], scale = coef[1];
  const int Dc = a.Dc;
  for (;;) {
    const int k_row = next_row(counter);
    if (k_row >= a.Uc) break;
    const int ua = a.order[k_row];
    const T *src = v1 + (int64_t)ua * Dc;
    for (int i = threadIdx.x; i < Dc; i += blockDim.x) row[i] = src[i];
    if (threadIdx.x == 0) {
      int n = 0;
      for (; n < a.wu; n++)
        if (a.ell_up[(int64_t)ua * a.wu + n] == kEllNone) break;
      s_nu = n;
    }
    for (int s = threadIdx.x; s < a.wu; s += blockDim.x) {
      const uint32_t e = a.ell_up[(int64_t)ua * a.wu + s];
      if (e != kEllNone) {
        s_src[s] = e & 0xFFFFu;
        s_cf[s] = a.cf_up[e >> 16];
      }
    }
    __syncthreads();
    const int nu = s_nu;
    const uint32_t u = a.unrank_up[ua];
    const double du = a.du[ua];
    double pr[2] = {0.0, 0.0};
    T *dst = v0 + (int64_t)ua * Dc;
    constexpr int CPT = 2;  // columns per thread per iteration
    for (int base = 0; base < Dc; base += CPT * (int)blockDim.x) {
      int da[CPT];
      bool ok[CPT];
      T y[CPT], x[CPT];
      int cnt[CPT], wmax = 0;
#pragma unroll
      for (int c = 0; c < CPT; c++) {
        const int d0 = base + c * (int)blockDim.x + (int)threadIdx.x;
        ok[c] = d0 < Dc;
        da[c] = ok[c] ? d0 : Dc - 1;
        x[c] = row[da[c]];
        double D;
        if (a.cross_mode == 2) {
          D = __ldg(a.dfull + (int64_t)ua * Dc + da[c]);
        } else {
          D = du + __ldg(a.dd + da[c]);
          const uint32_t ud = u & (uint32_t)__ldg(a.unrank_dn + da[c]);
          if (a.cross_mode == 0) D += __ldg(a.utab + __popc(ud));
          else for (uint32_t m = ud; m; m &= m - 1) D += __ldg(a.usite + (__ffs(m) - 1));
        }
        y[c] = VT<T>::scale(D, x[c]);
        cnt[c] = __ldg(a.cnt_dn + da[c]);
        // a warp's columns are the aligned block [base + c*blockDim + 32w, ... + 32)
        wmax = max(wmax, (int)__ldg(a.wmax_dn + ((base + c * (int)blockDim.x + (int)(threadIdx.x & ~31u)) >> 5)));
      }
      for (int s = 0; s < wmax; s += 4) {
        uint32_t e[CPT][4];
#pragma unroll
        for (int c = 0; c < CPT; c++)
#pragma unroll
          for (int k = 0; k < 4; k++)
            e[c][k] = (s + k < cnt[c]) ? __ldg(a.ell_dn + (int64_t)(s + k) * Dc + da[c]) : kEllNone;
#pragma unroll
        for (int c = 0; c < CPT; c++)
#pragma unroll
          for (int k = 0; k < 4; k++)
            if (e[c][k] != kEllNone) {
              const double2 cf = __ldg(a.cf_dn + (e[c][k] >> 16));
              y[c] = VT<T>::add(y[c], VT<T>::cmul_re_im(cf.x, cf.y, row[e[c][k] & 0xFFFFu]));
            }
      }
      constexpr int kS = (sizeof(T) > 8) ? 2 : 4;  // up hops per batch (registers: complex holds twice as much)
      for (int s = 0; s < nu; s += kS) {
        T v[kS][CPT];
#pragma unroll
        for (int k = 0; k < kS; k++) {
          const T *p = v1 + (int64_t)s_src[(s + k < nu) ? s + k : s] * Dc;
#pragma unroll
          for (int c = 0; c < CPT; c++) v[k][c] = (s + k < nu) ? ldg_v<T>(p + da[c]) : VT<T>::zero();
        }
#pragma unroll
        for (int k = 0; k < kS; k++)
          if (s + k < nu) {
            const double2 cf = s_cf[s + k];
#pragma unroll
            for (int c = 0; c < CPT; c++) y[c] = VT<T>::add(y[c], VT<T>::cmul_re_im(cf.x, cf.y, v[k][c]));
          }
      }
#pragma unroll
      for (int c = 0; c < CPT; c++)
        if (ok[c]) {
          pr[0] += VT<T>::conj_mul_re(x[c], y[c]);
          pr[1] += VT<T>::conj_mul_im(x[c], y[c]);
          const T yy = VT<T>::scale(scale, y[c]);
          dst[da[c]] = (acc == 0.0) ? yy : VT<T>::add(VT<T>::scale(acc, dst[da[c]]), yy);
        }
    }
    block_sum<2>(pr);
    if (threadIdx.x == 0) {
      part[2 * (int64_t)ua] = pr[0];
      part[2 * (int64_t)ua + 1] = pr[1];
    }
  }
  retire(counter);
}

__device__ __forceinline__ double flip_sign(double x, uint32_t sg) {
  return __hiloint2double(__double2hiint(x) ^ (int)sg, __double2loint(x));
}

constexpr int kMaxGroups = 8;     // coefficients of one species, up to sign (two-pass kernels)
constexpr int kUpThreads = 256;   // column pass: 8 warps per CTA
constexpr int kUpMinBlocks = 3;   // CTAs per SM (at most 85 registers)
constexpr int kUpChunk = 128;     // doubles of a row per warp task (4 per lane)
constexpr int kUpBatch = 4;       // up hops per batch: 64 bytes per lane and hop pair in flight

// Hops of one species are grouped by coefficient up to sign; the row pass walks one gather
// table per group and multiplies each group's signed sum once, so no coefficient is looked up
// per element.
struct TwoPassArgs {
  int npad;                    // Dc rounded up to a multiple of 32
  int ng;                      // groups of down hops
  const uint4 *gat;            // per warp of 32 columns its groups' sets of 8 slots: [32 lanes] 8 entries word | sign << 15
  const uint4 *whead;          // per warp: first set, slots of groups 0-3 and 4-7 (8 bits each)
  const double2 *cf_dn;        // [ng] coefficients
  const uint8_t *nus;          // [Uc] up hops of each row
  int wu2;                     // words per row of up_ent
  const uint32_t *up_ent;      // [Uc][wu2] one group: two hops per word, rank | sign << 15 (16 bits each);
                               // several: one hop per word, rank | (2 * group + sign) << 16
  const double2 *cf_up;        // [up groups] coefficients
  int ngu;
};

// Row pass shapes by row length: P planes of STRIDE words (a row and 16 zero words) per CTA.
// A plane is a real row or the real or imaginary part of a complex one; every table entry is
// decoded once for all P planes.  Long rows leave room for two planes and one CTA per SM;
// shorter ones take four planes and as many CTAs as shared memory holds, which hides the
// staging of one CTA behind the gathers of the others.
template <int STRIDE> struct RowShape;
template <> struct RowShape<12896> { static constexpr int P = 2, threads = 1024, ctas = 1; };  // Dc <= 12,880 (N = 16)
template <> struct RowShape<6560> { static constexpr int P = 2, threads = 512, ctas = 2; };    // 6,435 (N = 15)
template <> struct RowShape<3456> { static constexpr int P = 4, threads = 512, ctas = 2; };    // 3,432 (N = 14)
template <> struct RowShape<1744> { static constexpr int P = 4, threads = 256, ctas = 4; };    // 1,716 (N = 13)
template <> struct RowShape<960> { static constexpr int P = 4, threads = 256, ctas = 4; };     // 924 (N = 12)

// Row pass: v0[u, :] = acc * v0[u, :] + scale * (D + down hops) v1[u, :] for the rows of P
// planes at a time; part[blockIdx] = sum over the CTA's rows of conj(v1) (D + down) v1.  Real
// rows are staged by bulk asynchronous copies completing on an mbarrier (per-thread cp.async
// when they are not 16-byte aligned), complex ones are split into their parts on the way; a
// bounded wait that gives up makes the CTA's partial sum NaN.  Bound by the L1 data pipe: each
// element reads ~20 operands of 8 bytes from shared memory.
// ONSITE: the cross-species diagonal is u0 * popcount(u & d) (cross_mode 0).
template <int STRIDE, bool CPLX, bool ONSITE>
__global__ void __launch_bounds__(RowShape<STRIDE>::threads, RowShape<STRIDE>::ctas)
prod_row_kernel(ProdArgs a, TwoPassArgs b, const double *__restrict__ v1, double *__restrict__ v0,
                const double *__restrict__ coef, double *__restrict__ part) {
  constexpr int P = RowShape<STRIDE>::P, NT = RowShape<STRIDE>::threads;
  constexpr int R = CPLX ? P / 2 : P;   // rows per task
  constexpr int W = CPLX ? 2 : 1;       // planes per row
  extern __shared__ __align__(128) double planes[];
  __shared__ uint64_t bar;
  const double acc = coef[0], scale = coef[1];
  const int Dc = a.Dc, Uc = a.Uc, tid = threadIdx.x, lane = tid & 31;
  __shared__ double2 s_c[kMaxGroups];
  if (tid < b.ng) s_c[tid] = b.cf_dn[tid];
  double pr = 0.0, pi = 0.0;
  const bool bulk = !CPLX && (Dc % 2 == 0) && ((uintptr_t)v1 % 16 == 0);
  if (tid == 0) mbar_init(&bar, 1);
  mbar_fence_init();
  for (int k = tid; k < 16 * P; k += NT)  // zero words after each plane (one per bank pair), never overwritten
    planes[(k >> 4) * STRIDE + Dc + (k & 15)] = 0.0;
  uint32_t phase = 0;
  bool ok = true;
  for (int u0 = R * blockIdx.x; u0 < Uc; u0 += R * gridDim.x) {
    const int nr = min(R, Uc - u0);  // rows past the last one repeat it and are not stored
    __syncthreads();                 // the previous planes are no longer read
    if (bulk) {
      if (tid == 0) {
        mbar_arrive_expect_tx(&bar, (uint32_t)(R * Dc * 8));
#pragma unroll
        for (int q = 0; q < R; q++)
          bulk_g2s(planes + q * STRIDE, v1 + (int64_t)(u0 + min(q, nr - 1)) * Dc, (uint32_t)(Dc * 8), &bar);
      }
      // the next rows toward L2 while these are processed (a hint, no completion)
      const int un = u0 + R * gridDim.x;
      if (tid < R && un + tid < Uc) {
        const double *pf = v1 + (int64_t)(un + tid) * Dc;
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(pf), "r"((uint32_t)(Dc * 8)) : "memory");
      }
      const bool got = mbar_wait(&bar, phase);
      phase ^= 1;
      if (__syncthreads_or(!got)) {
        ok = false;
        mbar_wait(&bar, phase ^ 1);  // copies still in flight land before the CTA leaves (bounded)
        break;
      }
    } else if (CPLX) {
#pragma unroll
      for (int q = 0; q < R; q++) {
        const double2 *s = reinterpret_cast<const double2 *>(v1) + (int64_t)(u0 + min(q, nr - 1)) * Dc;
#pragma unroll 4
        for (int i = tid; i < Dc; i += NT) {
          const double2 z = __ldg(s + i);
          planes[(2 * q) * STRIDE + i] = z.x;
          planes[(2 * q + 1) * STRIDE + i] = z.y;
        }
      }
      __syncthreads();
    } else {
#pragma unroll
      for (int q = 0; q < R; q++) {
        const double *s = v1 + (int64_t)(u0 + min(q, nr - 1)) * Dc;
        const uint32_t dst = smem_u32(planes + q * STRIDE);
        for (int i = tid; i < Dc; i += NT)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst + 8 * i), "l"(s + i) : "memory");
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
      asm volatile("cp.async.wait_all;\n" ::: "memory");
      __syncthreads();
    }
    uint32_t uc[R];
    double du[R];
#pragma unroll
    for (int q = 0; q < R; q++) {
      uc[q] = a.unrank_up[u0 + min(q, nr - 1)];
      du[q] = a.du[u0 + min(q, nr - 1)];
    }
    const char *rb = reinterpret_cast<const char *>(planes);
    for (int p = tid; p < b.npad; p += NT) {
      // per-column diagonal parts, the old v0 and the first set of slots, loaded before the gathers
      const int pc = (p < Dc) ? p : Dc - 1;
      const uint4 head = __ldg(b.whead + (p >> 5));  // the same for the warp's 32 columns
      const uint4 *gp = b.gat + (int64_t)head.x * 32 + lane;
      uint4 e = __ldg(gp);
      const double ddp = (!ONSITE && a.cross_mode == 2) ? 0.0 : __ldg(a.dd + pc);
      const uint32_t cdp = __ldg(a.unrank_dn + pc);
      double *o = v0 + ((int64_t)u0 * Dc + pc) * W;
      double y[P], old[P];
#pragma unroll
      for (int q = 0; q < P; q++) y[q] = old[q] = 0.0;
      if (acc != 0.0) {
#pragma unroll
        for (int r = 0; r < R; r++) {
          if constexpr (CPLX) {
            const double2 z = __ldcs(reinterpret_cast<const double2 *>(o + (int64_t)min(r, nr - 1) * Dc * W));
            old[2 * r] = z.x;
            old[2 * r + 1] = z.y;
          } else {
            old[r] = __ldcs(o + (int64_t)min(r, nr - 1) * Dc * W);
          }
        }
      }
      // two 16-bit entries: word index (15 bits) | sign << 15, the sign as a factor +-1; slots at
      // or beyond the warp's count hold a zero word, so only whole half sets are skipped
      for (int g = 0; g < b.ng; g++) {
        const int ns = (int)(((g < 4 ? head.y : head.z) >> (8 * (g & 3))) & 255u);
        double s[P];
#pragma unroll
        for (int q = 0; q < P; q++) s[q] = 0.0;
        auto gather2 = [&](uint32_t r) {
          const double *x0 = reinterpret_cast<const double *>(rb + ((r << 3) & 0x3FFF8u));
          const double *x1 = reinterpret_cast<const double *>(rb + ((r >> 13) & 0x3FFF8u));
          const double f0 = __hiloint2double((int)(((r << 16) & 0x80000000u) | 0x3FF00000u), 0);
          const double f1 = __hiloint2double((int)((r & 0x80000000u) | 0x3FF00000u), 0);
#pragma unroll
          for (int q = 0; q < P; q++) s[q] = fma(f0, x0[q * STRIDE], s[q]);
#pragma unroll
          for (int q = 0; q < P; q++) s[q] = fma(f1, x1[q * STRIDE], s[q]);
        };
        for (int k = 0; k < ns; k += 8) {
          const uint4 c = e;
          gp += 32;
          e = __ldg(gp);  // the next set (of the next group; one set past the last is allocated)
          gather2(c.x);
          gather2(c.y);
          if (k + 4 < ns) {
            gather2(c.z);
            gather2(c.w);
          }
        }
        const double2 c = s_c[g];
#pragma unroll
        for (int r = 0; r < R; r++) {
          if constexpr (CPLX) {
            y[2 * r] += c.x * s[2 * r] - c.y * s[2 * r + 1];
            y[2 * r + 1] += c.x * s[2 * r + 1] + c.y * s[2 * r];
          } else {
            y[r] = fma(c.x, s[r], y[r]);
          }
        }
      }
      if (p < Dc) {
#pragma unroll
        for (int r = 0; r < R; r++) {
          if (r >= nr) break;
          double D;
          const uint32_t ud = uc[r] & cdp;
          if (ONSITE) {
            // popcount as a double without a conversion: 2^52 + k, less 2^52
            D = fma(a.u0, __hiloint2double(0x43300000, __popc(ud)) - 4503599627370496.0, du[r] + ddp);
          } else if (a.cross_mode == 2) {
            D = __ldg(a.dfull + (int64_t)(u0 + r) * Dc + p);
          } else {
            D = du[r] + ddp;
            for (uint32_t m = ud; m; m &= m - 1) D += __ldg(a.usite + (__ffs(m) - 1));
          }
          double *orow = o + r * (int64_t)Dc * W;
          if constexpr (CPLX) {
            const double xr = planes[(2 * r) * STRIDE + p], xi = planes[(2 * r + 1) * STRIDE + p];
            const double yr = D * xr + y[2 * r], yi = D * xi + y[2 * r + 1];
            __stcs(reinterpret_cast<double2 *>(orow),
                   acc == 0.0 ? make_double2(scale * yr, scale * yi)
                              : make_double2(acc * old[2 * r] + scale * yr, acc * old[2 * r + 1] + scale * yi));
            pr += xr * yr + xi * yi;
            pi += xr * yi - xi * yr;
          } else {
            const double x = planes[r * STRIDE + p], yy = D * x + y[r];
            __stcs(orow, (acc == 0.0) ? scale * yy : acc * old[r] + scale * yy);
            pr += x * yy;
          }
        }
      }
    }
  }
  const double nan = __longlong_as_double(0x7FF8000000000000ll);
  double v[2] = {ok ? pr : nan, ok ? pi : nan};
  block_sum<2>(v);
  if (tid == 0) {
    part[2 * blockIdx.x] = v[0];
    part[2 * blockIdx.x + 1] = v[1];
  }
}

// Column pass: v0[u, chunk] += scale * sum_up c * v1[u', chunk].  A task is one row u and 128
// doubles of it (128 real columns or 64 complex ones); V doubles per load: lane l reads doubles
// 2l, 2l + 1 and 64 + 2l, 65 + 2l as two 16-byte loads (V = 2), or l, l + 32, ... one by one
// where a row may start on an odd double (V = 1).  Tasks run chunk-major (every row of chunk 0,
// then chunk 1, ...) by static striding over the warps of a grid that is resident at once, so
// the 1 KB pieces of v1 the rows gather stay in L2.  Each lane holds hop entries of the row and
// the warp broadcasts them by shuffles (no shared memory, no CTA barrier).  MULTI: several up
// coefficients, each entry naming its own (read from shared memory at one address per warp);
// else one real coefficient and signs.  The sum includes the row pass's records.  Bound by the
// L1 data pipe: ~17 operands of 8 bytes per double.
// TAYLOR: every finished element y of v0 also goes into a Taylor sum, sum += c * y (complex
// vectors), which saves the sum's own pass over y.
struct TaylorSum {
  double2 *sum;
  double2 c;
};

template <int V, bool CPLX, bool MULTI, bool TAYLOR>
__global__ void __launch_bounds__(kUpThreads, kUpMinBlocks) prod_col_kernel(ProdArgs a, TwoPassArgs b,
                                                                          const double *__restrict__ v1,
                                                                          double *__restrict__ v0,
                                                                          const double *__restrict__ coef, SumOut so,
                                                                          TaylorSum ts) {
  static_assert(V == 2 || !CPLX, "complex rows are whole 16-byte units");
  constexpr int NL = 4 / V;  // loads per lane and source row
  __shared__ double2 s_cf[2 * kMaxGroups];
  const int lane = threadIdx.x & 31;
  const int warp = (int)((blockIdx.x * (unsigned)kUpThreads + threadIdx.x) >> 5);
  const int nwarps = (int)(gridDim.x * (unsigned)kUpThreads) >> 5;
  const int ncol = a.Dc * (CPLX ? 2 : 1), Uc = a.Uc;
  const int nchunk = (ncol + kUpChunk - 1) / kUpChunk;
  const int64_t ntask = (int64_t)nchunk * Uc;
  if (MULTI) {
    if (threadIdx.x < 2 * b.ngu) {
      const double2 c = b.cf_up[threadIdx.x >> 1];
      s_cf[threadIdx.x] = (threadIdx.x & 1) ? make_double2(-c.x, -c.y) : c;
    }
    __syncthreads();
  }
  const double scale = coef[1], tup = (MULTI || b.ngu == 0) ? 1.0 : b.cf_up[0].x;
  double pr = 0.0, pi = 0.0;
  // the row's hop count and packed entries of the next task are loaded one task ahead
  int64_t task = warp;
  int nu_n = 0;
  uint32_t my_n = 0u, my2_n = 0u;
  auto fetch = [&](int64_t t) {
    if (t < ntask) {
      const int un = (int)(t % Uc);
      nu_n = b.nus[un];
      const uint32_t *e = b.up_ent + (int64_t)un * b.wu2;
      my_n = ((MULTI ? 1 : 2) * lane < nu_n) ? __ldg(e + lane) : 0u;
      if (MULTI) my2_n = (lane + 32 < nu_n) ? __ldg(e + lane + 32) : 0u;
    }
  };
  fetch(task);
  const uint64_t rowb = (uint64_t)ncol * sizeof(double);
  for (; task < ntask; task += nwarps) {
    const int c = (int)(task / Uc), u = (int)(task - (int64_t)c * Uc);
    const int nu = nu_n;
    const uint32_t my = my_n, my2 = my2_n;
    fetch(task + nwarps);
    const int d = c * kUpChunk + V * lane;
    const char *base[NL];
    bool ok[NL];
#pragma unroll
    for (int j = 0; j < NL; j++) {
      ok[j] = d + j * 32 * V < ncol;  // V = 2: ncol is even, pairs are whole
      // lanes past the last column read column 0 and discard what they summed
      base[j] = reinterpret_cast<const char *>(v1 + (ok[j] ? d + j * 32 * V : 0));
    }
    double h[4] = {0.0, 0.0, 0.0, 0.0};
    auto load = [&](uint32_t rank, double (&x)[4]) {
      const uint64_t off = (uint64_t)rank * rowb;
#pragma unroll
      for (int j = 0; j < NL; j++) {
        if constexpr (V == 2) {
          const double2 z = __ldg(reinterpret_cast<const double2 *>(base[j] + off));
          x[2 * j] = z.x;
          x[2 * j + 1] = z.y;
        } else {
          x[j] = __ldg(reinterpret_cast<const double *>(base[j] + off));
        }
      }
    };
    auto entry = [&](int k) -> uint32_t {
      if constexpr (MULTI) return __shfl_sync(0xFFFFFFFFu, k < 32 ? my : my2, k & 31);
      const uint32_t word = __shfl_sync(0xFFFFFFFFu, my, (k >> 1) & 31);
      return (k & 1) ? (word >> 16) : (word & 0xFFFFu);
    };
    auto rank_of = [&](uint32_t e) { return MULTI ? (e & 0xFFFFu) : (e & 0x7FFFu); };
    auto add = [&](uint32_t e, const double (&x)[4]) {
      if constexpr (MULTI) {
        const double2 cc = s_cf[e >> 16];
        if constexpr (CPLX) {
#pragma unroll
          for (int j = 0; j < 4; j += 2) {
            h[j] = fma(cc.x, x[j], fma(-cc.y, x[j + 1], h[j]));
            h[j + 1] = fma(cc.x, x[j + 1], fma(cc.y, x[j], h[j + 1]));
          }
        } else {
#pragma unroll
          for (int j = 0; j < 4; j++) h[j] = fma(cc.x, x[j], h[j]);
        }
      } else {
        const uint32_t sg = (e & 0x8000u) << 16;
#pragma unroll
        for (int j = 0; j < 4; j++) h[j] += flip_sign(x[j], sg);
      }
    };
    int k = 0;
    for (; k + kUpBatch <= nu; k += kUpBatch) {
      double x[kUpBatch][4];
      uint32_t e[kUpBatch];
      if constexpr (MULTI) {
#pragma unroll
        for (int q = 0; q < kUpBatch; q++) e[q] = entry(k + q);
      } else {
#pragma unroll
        for (int q = 0; q < kUpBatch; q += 2) {
          const uint32_t word = __shfl_sync(0xFFFFFFFFu, my, ((k + q) >> 1) & 31);
          e[q] = word & 0xFFFFu;
          e[q + 1] = word >> 16;
        }
      }
#pragma unroll
      for (int q = 0; q < kUpBatch; q++) load(rank_of(e[q]), x[q]);
#pragma unroll
      for (int q = 0; q < kUpBatch; q++) add(e[q], x[q]);
    }
    for (; k < nu; k++) {
      const uint32_t e = entry(k);
      double x[4];
      load(rank_of(e), x);
      add(e, x);
    }
    const double *xp = v1 + (int64_t)u * ncol + d;
    double *yp = v0 + (int64_t)u * ncol + d;
    // v0 is streamed (read and written once): evict-first, so it does not push the chunk of
    // v1 that the following rows gather from out of L2
#pragma unroll
    for (int j = 0; j < NL; j++) {
      if (!ok[j]) continue;
      if constexpr (V == 2) {
        const double h0 = tup * h[2 * j], h1 = tup * h[2 * j + 1];
        const double2 xv = __ldg(reinterpret_cast<const double2 *>(xp + 64 * j));
        const double2 yv = __ldcs(reinterpret_cast<const double2 *>(yp + 64 * j));
        pr += xv.x * h0 + xv.y * h1;
        if (CPLX) pi += xv.x * h1 - xv.y * h0;
        const double2 yn = make_double2(yv.x + scale * h0, yv.y + scale * h1);
        __stcs(reinterpret_cast<double2 *>(yp + 64 * j), yn);
        if constexpr (TAYLOR) {
          double2 *tp = ts.sum + (((int64_t)u * ncol + d) >> 1) + 32 * j;
          double2 t = __ldcs(tp);
          t.x += ts.c.x * yn.x - ts.c.y * yn.y;
          t.y += ts.c.x * yn.y + ts.c.y * yn.x;
          __stcs(tp, t);
        }
      } else {
        const double h0 = tup * h[j];
        pr += __ldg(xp + 32 * j) * h0;
        __stcs(yp + 32 * j, __ldcs(yp + 32 * j) + scale * h0);
      }
    }
  }
  double v[2] = {pr, pi};
  grid_sum<2>(v, so);
}

__device__ __forceinline__ uint32_t compress_species(uint64_t c, int s, int N) {
  uint32_t x = 0;
  for (int i = 0; i < N; i++) x |= (uint32_t)((c >> (2 * i + s)) & 1ull) << i;
  return x;
}

// A function of the configuration in HPhi's row order (the diagonal) to native order.
__global__ void prod_permute_diag_kernel(int64_t dim, int N, int Dc, const uint64_t *__restrict__ list_1,
                                         const uint16_t *__restrict__ rank, const uint16_t *__restrict__ pos_dn,
                                         const double *__restrict__ in, double *__restrict__ out) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < dim; r += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t c = list_1[r];
    const int64_t pos = (int64_t)rank[compress_species(c, 0, N)] * Dc + pos_dn[compress_species(c, 1, N)];
    out[pos] = in[r];
  }
}

// Sign sigma(c) from the two species' words: (-1)^#{down at i, up at j : i < j}; bit j of the
// running xor of d, shifted up by one, is the parity of the downs below j.
__device__ __forceinline__ uint32_t species_parity16(uint32_t u, uint32_t d) {
  d ^= d << 1;
  d ^= d << 2;
  d ^= d << 4;
  d ^= d << 8;
  return (uint32_t)__popc(u & (d << 1)) & 1u;
}
__host__ __device__ __forceinline__ uint32_t compress_even(uint32_t x) {  // bit 2i -> bit i
  x &= 0x55555555u;
  x = (x | (x >> 1)) & 0x33333333u;
  x = (x | (x >> 2)) & 0x0F0F0F0Fu;
  x = (x | (x >> 4)) & 0x00FF00FFu;
  return (x | (x >> 8)) & 0xFFFFu;
}
__host__ __device__ __forceinline__ uint32_t spread_even(uint32_t x) {  // bit i -> bit 2i, x < 2^16
  x = (x | (x << 8)) & 0x00FF00FFu;
  x = (x | (x << 4)) & 0x0F0F0F0Fu;
  x = (x | (x << 2)) & 0x33333333u;
  return (x | (x << 1)) & 0x55555555u;
}
template <typename T> __device__ __forceinline__ T signed_v(const T &x, uint32_t par);
template <> __device__ __forceinline__ double signed_v<double>(const double &x, uint32_t par) { return par ? -x : x; }
template <> __device__ __forceinline__ cplx signed_v<cplx>(const cplx &x, uint32_t par) {
  return par ? cplx{-x.x, -x.y} : x;
}

// The two orders' permutations are bound by the L2 sectors of their scattered side (32 bytes
// moved for each 8- or 16-byte element), so both run in an order in which every sector's other
// elements are wanted soon: all rows of one group of up configurations that share their upper
// sites (7 MB of the 4x4 half-filled sector), then the next group.  The row's words come from
// a few bit steps instead of one step per site.  4x4 lattice with 6 + 6 electrons, real:
// to native 693 -> 318, from native 1083 -> 368 us.

constexpr int kPermThreads = 256;
constexpr int kPermBatch = 4;    // elements in flight per thread
// Mean rows per HPhi block (piece) below which a thread takes a row.  us per call, blocks and rows, to
// native | from native, with the wait of the call in each: 12 sites with 3 + 3 electrons (27 rows) 13.0 /
// 12.5 | 14.9 / 12.6; 15 with 4 + 4 (115) 19.9 / 18.5 | 24.0 / 18.2; 14 with 5 + 5 (278, 4 M rows) 25.7 / 25.3 |
// 30.1 / 27.0; 14 half filled (719, 12 M) 57 / 89 | 57 / 64; 4x4 with 6 + 6 (64 M) 233 / 594 | 259 / 274.
// (Down configurations in rank order; the long blocks' gain is in the change to native order.)
constexpr int kPermShort = 32;

// HPhi order -> native: a CTA per up configuration u.  HPhi's row of (u, d) is
// list_2_1[lower half] + list_2_2[upper half] - 3; with u fixed each term depends on the downs
// of one half only, so the two lookups become 2^(downs of the half) entries in shared memory.
template <typename T>
__global__ void __launch_bounds__(kPermThreads) prod_to_native_kernel(int N, int Uc, int Dc,
                                                                      const uint16_t *__restrict__ unrank_up,
                                                                      const uint16_t *__restrict__ unrank_dn,
                                                                      const uint32_t *__restrict__ l21,
                                                                      const uint32_t *__restrict__ l22,
                                                                      const T *__restrict__ in, T *__restrict__ out) {
  __shared__ uint32_t s_lo[256], s_hi[256];  // at most 8 downs of each half (N <= 16)
  const int nlo = N / 2, nhi = N - nlo;      // HPhi's lower half: N bits, (N + 1) / 2 ups and N / 2 downs
  const uint32_t mask = (uint32_t)((1ull << N) - 1);
  for (int ua = blockIdx.x; ua < Uc; ua += gridDim.x) {
    const uint32_t u = unrank_up[ua], cu = spread_even(u);
    __syncthreads();  // the previous row's tables are no longer read
    if (threadIdx.x < (1u << nlo)) s_lo[threadIdx.x] = __ldg(l21 + ((cu | (spread_even(threadIdx.x) << 1)) & mask));
    if (threadIdx.x < (1u << nhi)) {
      const uint64_t c = (uint64_t)cu | ((uint64_t)spread_even((uint32_t)threadIdx.x << nlo) << 1);
      s_hi[threadIdx.x] = __ldg(l22 + (c >> N)) - 3u;
    }
    __syncthreads();
    T *o = out + (int64_t)ua * Dc;
    for (int d0 = threadIdx.x; d0 < Dc; d0 += kPermBatch * kPermThreads) {
      T v[kPermBatch];
      uint32_t d[kPermBatch];
#pragma unroll
      for (int q = 0; q < kPermBatch; q++) {
        const int p = d0 + q * kPermThreads;
        d[q] = __ldg(unrank_dn + (p < Dc ? p : d0));
      }
#pragma unroll
      for (int q = 0; q < kPermBatch; q++) v[q] = ldg_v<T>(in + (s_lo[d[q] & ((1u << nlo) - 1)] + s_hi[d[q] >> nlo]));
#pragma unroll
      for (int q = 0; q < kPermBatch; q++) {
        const int p = d0 + q * kPermThreads;
        if (p < Dc) o[p] = signed_v<T>(v[q], species_parity16(u, d[q]));
      }
    }
  }
}

// Native -> HPhi order, a warp per piece of an HPhi block; pieces run by upper ups, then upper downs.
template <typename T>
__global__ void __launch_bounds__(kPermThreads) prod_from_native_kernel(int N, int Dc, const SectorBlock *__restrict__ tasks,
                                                                        int ntask, const uint32_t *__restrict__ low,
                                                                        const uint16_t *__restrict__ rank,
                                                                        const uint16_t *__restrict__ pos_dn,
                                                                        const T *__restrict__ in, T *__restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int nwarps = (int)(gridDim.x * kPermThreads) >> 5;
  for (int t = (int)(blockIdx.x * kPermThreads + threadIdx.x) >> 5; t < ntask; t += nwarps) {
    const uint4 w = __ldg(reinterpret_cast<const uint4 *>(tasks) + t);
    const uint64_t hi = (uint64_t)w.x << N;
    const int n = (int)w.w;
    for (int a0 = lane; a0 < n; a0 += 32 * kPermBatch) {
      T v[kPermBatch];
      uint32_t par[kPermBatch];
#pragma unroll
      for (int q = 0; q < kPermBatch; q++) {
        const int a = a0 + 32 * q;
        const uint32_t c32 = (uint32_t)hi | __ldg(low + w.z + (a < n ? a : a0));  // 2 N <= 32 bits
        const uint32_t u = compress_even(c32), d = compress_even(c32 >> 1);
        par[q] = species_parity16(u, d);
        v[q] = ldg_v<T>(in + ((int64_t)__ldg(rank + u) * Dc + __ldg(pos_dn + d)));
      }
#pragma unroll
      for (int q = 0; q < kPermBatch; q++) {
        const int a = a0 + 32 * q;
        if (a < n) out[(int64_t)w.y + a] = signed_v<T>(v[q], par[q]);
      }
    }
  }
}

// Either direction, a thread per HPhi row: sectors whose HPhi blocks are shorter than a warp
// (kPermShort), where the kernels above leave most of their lanes idle (15 sites with 3 + 3
// electrons, complex, blocks of 21 rows: a whole hphi_mltply_device 114 -> 73 us).
// Also any vector whose complex elements are not at multiples of 16 bytes (WHOLE false).
template <typename T, bool TO_NATIVE, bool WHOLE>
__global__ void __launch_bounds__(kPermThreads) prod_permute_rows_kernel(int64_t dim, int Dc,
                                                                         const uint64_t *__restrict__ list_1,
                                                                         const uint16_t *__restrict__ rank,
                                                                         const uint16_t *__restrict__ pos_dn,
                                                                         const T *__restrict__ in, T *__restrict__ out) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < dim; r += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t c = (uint32_t)__ldg(list_1 + r);  // 2 N <= 32 bits
    const uint32_t u = compress_even(c), d = compress_even(c >> 1);
    const int64_t pos = (int64_t)__ldg(rank + u) * Dc + __ldg(pos_dn + d);
    const T *from = in + (TO_NATIVE ? r : pos);
    T v;
    if constexpr (WHOLE) v = ldg_v<T>(from);
    else v = *from;
    out[TO_NATIVE ? pos : r] = signed_v<T>(v, species_parity16(u, d));
  }
}

// Diagonal observables in native order (expec_energy_flct_Hubbard, src/expec_energy_flct.c:259-330).
template <typename T>
__global__ void prod_obs_kernel(ProdArgs a, const T *__restrict__ v, SumOut so) {
  double o[6] = {0, 0, 0, 0, 0, 0};
  const int64_t n = (int64_t)a.Uc * a.Dc;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
    const int ua = (int)(p / a.Dc), da = (int)(p - (int64_t)ua * a.Dc);
    const uint32_t u = a.unrank_up[ua], d = a.unrank_dn[da];
    const double w = VT<T>::abs2(v[p]);
    const int up = __popc(u), dn = __popc(d);
    const double D = (double)__popc(u & d), Nn = (double)(up + dn), Sz = 0.5 * (double)(up - dn);
    o[0] += w * D; o[1] += w * D * D; o[2] += w * Nn; o[3] += w * Nn * Nn; o[4] += w * Sz; o[5] += w * Sz * Sz;
  }
  grid_sum<6>(o, so);
}

uint64_t binom_p(int n, int k) {
  if (k < 0 || k > n) return 0;
  uint64_t r = 1;
  for (int i = 1; i <= k; i++) r = r * (uint64_t)(n - k + i) / (uint64_t)i;
  return r;
}

int cuda_ok(cudaError_t e, const char *what) {
  if (e != cudaSuccess) {
    set_error(std::string("product kernel: ") + what + ": " + cudaGetErrorString(e));
    return -1;
  }
  return 0;
}

}  // namespace

struct ProdPlan {
  ProdArgs args{};
  std::vector<void *> allocs;
  int grid = 0;
  size_t smem[2] = {0, 0};  // real, complex
  double *part = nullptr;   // partial sums: 2 * max(Uc, grid_row + grid_col)
  int *counter = nullptr;
  bool two_pass = false;    // the two-pass kernels apply
  bool uniform = false;     // down hops of one magnitude, no complex hop
  TwoPassArgs tp{};
  int stride = 0;           // row pass shape (RowShape)
  bool multi_up = false;    // several up coefficients, or a complex one
  int grid_row[2] = {0, 0}, grid_col = 0;
  std::vector<uint16_t> rank, pos_dn, unrank_up, unrank_dn;  // host copies of the position tables
  const SectorBlock *perm = nullptr;  // pieces of HPhi's blocks for prod_from_native_kernel
  const uint32_t *perm_low = nullptr;  // the blocks' lower halves
  int nperm = 0;
};

void prod_plan_free(ProdPlan *p) {
  if (!p) return;
  for (void *q : p->allocs) cudaFree(q);
  delete p;
}

namespace {

template <typename V>
int upload(ProdPlan *p, const std::vector<V> &h, const V **d, std::string *err) {
  void *q = nullptr;
  const size_t bytes = h.empty() ? 16 : sizeof(V) * h.size();
  if (cudaMalloc(&q, bytes) != cudaSuccess) {
    *err = "product plan: device allocation failed";
    return -1;
  }
  p->allocs.push_back(q);
  if (!h.empty() && cudaMemcpy(q, h.data(), sizeof(V) * h.size(), cudaMemcpyHostToDevice) != cudaSuccess) {
    *err = "product plan: copy failed";
    return -1;
  }
  *d = (const V *)q;
  return 0;
}

struct SpeciesHop {
  int i, j;          // created, annihilated site
  double re, im;     // operator coefficient
};

// ELL of one species' hops over its configurations (by rank): per configuration the
// applicable hops as (source rank, coefficient index 2h + sign).
void build_ell(const std::vector<SpeciesHop> &hops, const std::vector<uint16_t> &unrank,
               const std::vector<uint16_t> &rank, std::vector<std::vector<uint32_t>> *rows, int *width) {
  rows->assign(unrank.size(), {});
  *width = 0;
  for (size_t r = 0; r < unrank.size(); r++) {
    const uint32_t x = unrank[r];
    for (size_t h = 0; h < hops.size(); h++) {
      const int i = hops[h].i, j = hops[h].j;
      if (!((x >> i) & 1u) || ((x >> j) & 1u)) continue;
      const uint32_t src = x ^ (1u << i) ^ (1u << j);
      const int lo = std::min(i, j), hi = std::max(i, j);
      const uint32_t between = (uint32_t)(((1ull << hi) - 1) ^ ((1ull << (lo + 1)) - 1));
      const uint32_t sign = (uint32_t)(__builtin_popcount(x & between) & 1);
      (*rows)[r].push_back((uint32_t)rank[src] | ((2u * (uint32_t)h + sign) << 16));
    }
    *width = std::max(*width, (int)(*rows)[r].size());
  }
}

std::vector<double2> coef_table(const std::vector<SpeciesHop> &hops) {
  std::vector<double2> c(2 * hops.size() + 1);
  for (size_t h = 0; h < hops.size(); h++) {
    c[2 * h] = make_double2(hops[h].re, hops[h].im);
    c[2 * h + 1] = make_double2(-hops[h].re, -hops[h].im);
  }
  return c;
}

uint64_t spread_species(uint32_t x, int s, int N) {
  uint64_t c = 0;
  for (int i = 0; i < N; i++)
    if ((x >> i) & 1u) c |= 1ull << (2 * i + s);
  return c;
}

// Positions of the down configurations for the row pass.  The row pass gives column p to
// lane p % 32 of warp p / 32, and an 8-byte gather of source column q hits the shared-memory
// bank pair q % 16; a half-warp's slot count is max(largest lane degree, largest bank-pair
// load) (the edge colouring of gather_warp), so positions decide both.  Start from the
// configurations sorted by hop count (equal lane degrees in a half-warp), then swap positions
// (within a half-warp: a bank change; across half-warps: only between equal hop counts) when
// that does not raise the summed slot counts of the half-warps it touches.  rows[r]: sources
// of configuration r (ELL entries, source in the low 16 bits).  Returns the position of each
// configuration; deterministic (fixed seed).
std::vector<int> balance_positions(const std::vector<std::vector<uint32_t>> &rows) {
  const int n = (int)rows.size();
  constexpr int G = 16;
  std::vector<int> order(n), pos(n);
  for (int r = 0; r < n; r++) order[r] = r;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return rows[a].size() > rows[b].size(); });
  for (int p = 0; p < n; p++) pos[order[p]] = p;
  const int ng = (n + G - 1) / G;
  if (n < 4 * G) return pos;
  std::vector<std::vector<int>> src(n), rdr(n);
  for (int r = 0; r < n; r++)
    for (uint32_t e : rows[r]) {
      const int q = (int)(e & 0xFFFFu);
      src[r].push_back(q);
      rdr[q].push_back(r);
    }
  std::vector<int> at(order);  // configuration at each position
  std::vector<int> load((size_t)ng * G, 0), lmax(ng, 0), D(ng, 0);
  for (int r = 0; r < n; r++) {
    const int g = pos[r] / G;
    lmax[g] = std::max(lmax[g], (int)src[r].size());
    for (int q : src[r]) load[(size_t)g * G + pos[q] % G]++;
  }
  auto eval = [&](int g) {
    int m = lmax[g];
    for (int k = 0; k < G; k++) m = std::max(m, load[(size_t)g * G + k]);
    return m;
  };
  for (int g = 0; g < ng; g++) D[g] = eval(g);
  uint64_t rng = 0x9E3779B97F4A7C15ull;
  auto next = [&]() { rng ^= rng << 13; rng ^= rng >> 7; rng ^= rng << 17; return rng; };
  std::vector<int> touched;
  std::vector<char> mark(ng, 0);
  auto touch = [&](int g) { if (!mark[g]) { mark[g] = 1; touched.push_back(g); } };
  // adds (sgn = 1) or removes (-1) a configuration's edges: its reads (in its own half-warp)
  // and the reads of it; edges to `other` are left to the other configuration's call
  auto contrib = [&](int r, int p, int sgn, int other) {
    const int g = p / G, bk = p % G;
    for (int q : src[r])
      if (q != other) load[(size_t)g * G + pos[q] % G] += sgn;
    for (int rr : rdr[r])
      if (rr != other) { const int gg = pos[rr] / G; load[(size_t)gg * G + bk] += sgn; touch(gg); }
    touch(g);
  };
  const int64_t iters = std::min<int64_t>(200 * (int64_t)n, 4000000);
  for (int64_t it = 0; it < iters; it++) {
    const int p1 = (int)(next() % n);
    int p2;
    if (next() & 1) p2 = (p1 / G) * G + (int)(next() % G);
    else p2 = (int)(next() % n);
    if (p2 >= n || p2 == p1 || src[at[p1]].size() != src[at[p2]].size()) continue;
    const int a = at[p1], b = at[p2];
    touched.clear();
    contrib(a, p1, -1, -1);
    contrib(b, p2, -1, a);
    pos[a] = p2; pos[b] = p1; at[p1] = b; at[p2] = a;
    contrib(a, p2, +1, -1);
    contrib(b, p1, +1, a);
    long before = 0, after = 0;
    std::vector<int> nd(touched.size());
    for (size_t i = 0; i < touched.size(); i++) {
      before += D[touched[i]];
      nd[i] = eval(touched[i]);
      after += nd[i];
    }
    if (after <= before) {
      for (size_t i = 0; i < touched.size(); i++) D[touched[i]] = nd[i];
    } else {
      contrib(a, p2, -1, -1);
      contrib(b, p1, -1, a);
      pos[a] = p1; pos[b] = p2; at[p1] = a; at[p2] = b;
      contrib(a, p1, +1, -1);
      contrib(b, p2, +1, a);
    }
    for (int g : touched) mark[g] = 0;
  }
  return pos;
}

}  // namespace

// The species (0 up, 1 down) and hop of a term that moves one electron; false for any other.
static bool species_hop(const BitTerm &t, SpeciesHop *h, int *species) {
  if (__builtin_popcountll(t.flip) != 2 || t.cm != t.flip) return false;
  const int p = __builtin_ctzll(t.flip), q = 63 - __builtin_clzll(t.flip);
  if ((p & 1) != (q & 1)) return false;
  if (t.cv != (1ull << p) && t.cv != (1ull << q)) return false;
  const int created = __builtin_ctzll(t.cv), annihilated = (created == p) ? q : p;
  const double sg = (__builtin_popcountll(t.cv & t.sm) & 1) ? -1.0 : 1.0;
  *h = SpeciesHop{created >> 1, annihilated >> 1, sg * t.re, sg * t.im};
  *species = p & 1;
  return true;
}

// Groups hops by coefficient up to sign: at time index k hop h has the coefficient
// gsign[h] * cf[k * groups + gid[h]] (static H: one index).  seq[k][h]: coefficients; hops share
// a group when their whole sequences agree up to one sign.
struct HopGroups {
  int n = 0;
  std::vector<int> gid, gsign;
  std::vector<double2> cf;
};
static bool coef_groups(const std::vector<std::vector<double2>> &seq, HopGroups *G) {
  const size_t nk = seq.size(), nh = seq[0].size();
  std::vector<size_t> rep;
  for (size_t h = 0; h < nh; h++) {
    int sign = 0;
    size_t g = 0;
    for (; g < rep.size() && sign == 0; g++)
      for (int sg : {1, -1}) {
        bool same = true;
        for (size_t k = 0; k < nk && same; k++)
          same = seq[k][h].x == sg * seq[k][rep[g]].x && seq[k][h].y == sg * seq[k][rep[g]].y;
        if (same) { sign = sg; break; }
      }
    if (sign == 0) {
      if (rep.size() == (size_t)kMaxGroups) return false;
      rep.push_back(h);
      sign = 1;
      g = rep.size();
    }
    G->gid.push_back((int)g - 1);
    G->gsign.push_back(sign);
  }
  G->n = (int)rep.size();
  for (size_t k = 0; k < nk; k++)
    for (size_t r : rep) G->cf.push_back(seq[k][r]);
  return true;
}
static std::vector<std::vector<double2>> static_seq(const std::vector<SpeciesHop> &hops) {
  std::vector<std::vector<double2>> q(1);
  for (const SpeciesHop &h : hops) q[0].push_back(make_double2(h.re, h.im));
  return q;
}

template <typename F>
static void with_row_kernel(int stride, bool cplx_v, bool onsite, F f) {
#define HPHI_ROW(S)                                                                                                     \
  case S:                                                                                                               \
    if (onsite) cplx_v ? f(prod_row_kernel<S, true, true>, RowShape<S>{}) : f(prod_row_kernel<S, false, true>, RowShape<S>{});  \
    else cplx_v ? f(prod_row_kernel<S, true, false>, RowShape<S>{}) : f(prod_row_kernel<S, false, false>, RowShape<S>{});       \
    break;
  switch (stride) {
    HPHI_ROW(960) HPHI_ROW(1744) HPHI_ROW(3456) HPHI_ROW(6560) HPHI_ROW(12896)
  }
#undef HPHI_ROW
}

// Tables and launch shapes of the two-pass kernels.  rows_*: per configuration its hops as
// source | (2 * hop + sign) << 16.  Leaves p->two_pass false, and the plan as it was, where a gather
// table does not apply; -1 where there is no memory for the tables.
static int two_pass_build(Sector *s, ProdPlan *p, const std::vector<std::vector<uint32_t>> &rows_dn,
                          const std::vector<std::vector<uint32_t>> &rows_up, const HopGroups (&G)[2], std::string *err) {
  const int Uc = p->args.Uc, Dc = p->args.Dc;
  TwoPassArgs &b = p->tp;
  b.npad = (Dc + 31) / 32 * 32;
  b.ng = G[1].n;
  const int nw = b.npad / 32;
  std::vector<std::vector<uint32_t>> ptr(b.ng), ents(b.ng);
  for (int g = 0; g < b.ng; g++) {
    ptr[g].push_back(0);
    for (int r = 0; r < b.npad; r++) {
      for (uint32_t e : r < Dc ? rows_dn[r] : std::vector<uint32_t>()) {
        const uint32_t h = (e >> 16) >> 1, sign = (e >> 16) & 1u;
        if (G[1].gid[h] == g) ents[g].push_back((e & 0xFFFFu) | ((sign ^ (G[1].gsign[h] < 0 ? 1u : 0u)) << 16));
      }
      ptr[g].push_back((uint32_t)ents[g].size());
    }
  }
  std::vector<std::vector<uint16_t>> code((size_t)nw * b.ng);
  std::vector<int> slots((size_t)nw * b.ng);
  size_t n_ent = 0;
  for (const auto &e : ents) n_ent += e.size();
  host_parallel(nw, 0.1 * (double)n_ent, [&](int64_t w) {
    for (int g = 0; g < b.ng; g++)
      slots[w * b.ng + g] = gather_warp(&ptr[g][32 * w], ents[g].data(), Dc, &code[w * b.ng + g]);
  });
  std::vector<uint4> gat, whead(nw);
  for (int w = 0; w < nw; w++) {
    uint64_t cnt = 0;
    whead[w].x = (uint32_t)(gat.size() / 32);
    for (int g = 0; g < b.ng; g++) {
      const int ns = slots[(size_t)w * b.ng + g];
      if (ns > 255) return 0;  // counts are packed in 8 bits
      cnt |= (uint64_t)ns << (8 * g);
      for (int j = 0; j < ns; j += 8)
        for (int lane = 0; lane < 32; lane++) {
          const GatherSet q = gather_set(code[(size_t)w * b.ng + g], j, lane);
          gat.push_back(make_uint4(q.w[0], q.w[1], q.w[2], q.w[3]));
        }
    }
    whead[w].y = (uint32_t)cnt;
    whead[w].z = (uint32_t)(cnt >> 32);
    whead[w].w = 0;
  }
  gat.resize(gat.size() + 32, make_uint4(0, 0, 0, 0));  // read ahead, never used
  b.ngu = G[0].n;
  p->multi_up = b.ngu > 1 || Uc > 32768;
  for (const double2 &c : G[0].cf) p->multi_up = p->multi_up || c.y != 0.0;
  size_t wu = 1;
  std::vector<uint8_t> nus(Uc, 0);
  for (int r = 0; r < Uc; r++) {
    nus[r] = (uint8_t)rows_up[r].size();
    wu = std::max(wu, rows_up[r].size());
  }
  b.wu2 = p->multi_up ? (int)wu : (int)(wu + 1) / 2;
  std::vector<uint32_t> ent((size_t)Uc * b.wu2, 0u);
  for (int r = 0; r < Uc; r++)
    for (size_t k = 0; k < rows_up[r].size(); k++) {
      const uint32_t e = rows_up[r][k], h = (e >> 16) >> 1, src = e & 0xFFFFu;
      const uint32_t sign = ((e >> 16) & 1u) ^ (G[0].gsign[h] < 0 ? 1u : 0u);
      uint32_t *row = &ent[(size_t)r * b.wu2];
      if (p->multi_up) row[k] = src | ((2u * (uint32_t)G[0].gid[h] + sign) << 16);
      else row[k / 2] |= (src | (sign << 15)) << (16 * (k % 2));
    }
  if (upload(p, gat, &b.gat, err) || upload(p, whead, &b.whead, err) || upload(p, G[1].cf, &b.cf_dn, err) ||
      upload(p, nus, &b.nus, err) || upload(p, ent, &b.up_ent, err) || upload(p, G[0].cf, &b.cf_up, err))
    return -1;
  for (int st : {960, 1744, 3456, 6560, 12896})
    if (Dc + 16 <= st) {
      p->stride = st;
      break;
    }
  for (int cv = 0; cv < 2; cv++) {
    int rc = 0;
    with_row_kernel(p->stride, cv == 1, p->args.cross_mode == 0, [&](auto kernel, auto shape) {
      using S = decltype(shape);
      const size_t smem = sizeof(double) * (size_t)S::P * p->stride;
      int per_sm = 0;
      if (raise_smem_limit((const void *)kernel, smem) != cudaSuccess ||
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, S::threads, smem) != cudaSuccess || per_sm < 1)
        rc = -1;
      const int rows = cv ? S::P / 2 : S::P;
      p->grid_row[cv] = std::max(1, std::min((Uc + rows - 1) / rows, per_sm * s->num_sms));
    });
    if (rc != 0) return -1;
  }
  int col = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&col, prod_col_kernel<2, true, true, false>, kUpThreads, 0);
  const int64_t ntask = (int64_t)Uc * ((2 * Dc + kUpChunk - 1) / kUpChunk);
  p->grid_col = (int)std::max<int64_t>(1, std::min<int64_t>(std::max(1, col) * s->num_sms, (ntask + 7) / 8));
  const int nrec = std::max(p->grid_row[0], p->grid_row[1]) + p->grid_col;
  if (nrec > Uc || !p->part) {
    double *part = nullptr;
    if (cudaMalloc(&part, sizeof(double) * 2 * (size_t)nrec) != cudaSuccess) return -1;
    if (p->part) p->allocs.erase(std::find(p->allocs.begin(), p->allocs.end(), (void *)p->part));
    cudaFree(p->part);
    p->part = part;
    p->allocs.push_back(p->part);
  }
  p->two_pass = true;
  return 0;
}

// Pieces of HPhi's blocks, by upper ups, then upper downs.
static int perm_tasks_build(Sector *s, ProdPlan *p, std::string *err) {
  std::vector<SectorBlock> blk, tasks;
  std::vector<uint32_t> low;
  if (sector_blocks(s, &blk, &low, err) != 0) return -1;
  // the upper half's even bits are ups when N (the lower half's bits) is even, else downs
  const uint32_t up_bits = (p->args.N % 2 == 0) ? 0x5555u : 0xAAAAu;
  // the blocks at their places (upper ups, upper downs)
  std::vector<uint32_t> at((size_t)1 << 16, 0u);
  for (size_t b = 0; b < blk.size(); b++) {
    const uint32_t x = compress_even(blk[b].ib), y = compress_even(blk[b].ib >> 1);
    const uint32_t up = up_bits & 1u ? x : y, dn = up_bits & 1u ? y : x;
    at[(up << 8) | dn] = (uint32_t)b + 1;
  }
  tasks.reserve(blk.size() + s->dim / kBlockPiece + 1);
  for (uint32_t q : at) {
    if (q == 0) continue;
    const SectorBlock &b = blk[q - 1];
    for (uint32_t a = 0; a < b.n; a += kBlockPiece)
      tasks.push_back(SectorBlock{b.ib, b.row0 + a, b.low0 + a, std::min<uint32_t>(kBlockPiece, b.n - a)});
  }
  if (upload(p, tasks, &p->perm, err) || upload(p, low, &p->perm_low, err)) return -1;
  p->nperm = (int)tasks.size();
  return 0;
}

int prod_plan_build(Sector *s, std::string *err) {
  const Model &m = s->model;
  s->prod = nullptr;
  if (m.calc_model != kHubbard || s->gc || m.nsite > 16 || m.nsite < 1) return 0;
  const int N = m.nsite;
  std::vector<SpeciesHop> hops[2];
  for (const BitTerm &t : m.offdiag) {
    SpeciesHop h;
    int sp;
    if (!species_hop(t, &h, &sp)) return 0;
    hops[sp].push_back(h);
  }
  if (hops[0].size() > 16000 || hops[1].size() > 16000) return 0;
  const int Uc = (int)binom_p(N, m.nup), Dc = (int)binom_p(N, m.ndown);
  if (Uc < 1 || Dc < 1 || Uc > 65535 || Dc > 65535 || (int64_t)Uc * Dc != s->dim) return 0;
  const size_t smem_r = sizeof(double) * (size_t)Dc, smem_c = sizeof(cplx) * (size_t)Dc;
  if (smem_c + 4096 > 227 * 1024) return 0;
  const int nx = 1 << N;
  std::vector<uint16_t> rank(nx), unrank_up, unrank_dn;
  {
    std::vector<int> fill(N + 1, 0);
    for (int x = 0; x < nx; x++) {
      const int k = __builtin_popcount(x);
      rank[x] = (uint16_t)fill[k]++;
      if (k == m.nup) unrank_up.push_back((uint16_t)x);
      if (k == m.ndown) unrank_dn.push_back((uint16_t)x);
    }
  }
  std::vector<std::vector<uint32_t>> rows_dn, rows_up;
  int wd = 0, wu = 0;
  build_ell(hops[1], unrank_dn, rank, &rows_dn, &wd);
  build_ell(hops[0], unrank_up, rank, &rows_up, &wu);
  // Two-pass kernels: few enough coefficients per species (up to sign), the planes of a row in
  // shared memory.  HPHI_B200_PROD=single keeps the one-pass kernel.
  HopGroups G[2];
  bool two_pass_ok;
  {
    const char *pe = getenv("HPHI_B200_PROD");
    two_pass_ok = !(pe && std::string(pe) == "single") && !hops[1].empty() && Dc + 16 <= 12896 && wd <= 255 &&
                  wu <= 64 && coef_groups(static_seq(hops[1]), &G[1]) && coef_groups(static_seq(hops[0]), &G[0]);
  }
  bool uniform_hops = two_pass_ok && G[1].n == 1;  // down hops of one magnitude, no complex hop
  for (const HopGroups &g : G)
    for (const double2 &c : g.cf) uniform_hops = uniform_hops && c.y == 0.0;
  // Down configurations take the positions balanced for the row pass's gather table
  // (balance_positions) where there is one magnitude; HPHI_B200_BALANCE=0 keeps rank order.
  // Up configurations keep their rank.  Complex or several hops keep rank order: the search
  // takes the build of 14 sites from 8 to 160 ms, and eight H*v with the changes of order
  // took 3290 us with its positions and 3170 in rank order (14-site ring with a flux).
  std::vector<uint16_t> pos_dn(rank);
  {
    const char *bal = getenv("HPHI_B200_BALANCE");
    if (two_pass_ok && uniform_hops && !(bal && std::string(bal) == "0")) {
      const std::vector<int> pos = balance_positions(rows_dn);
      std::vector<uint16_t> un(Dc);
      for (int r = 0; r < Dc; r++) un[pos[r]] = unrank_dn[r];
      unrank_dn.swap(un);
      for (int p = 0; p < Dc; p++) pos_dn[unrank_dn[p]] = (uint16_t)p;
      build_ell(hops[1], unrank_dn, pos_dn, &rows_dn, &wd);
    }
  }
  if (wu > kMaxUpWidth || wd > 255) return 0;
  std::vector<uint32_t> ell_dn((size_t)std::max(wd, 1) * Dc, kEllNone), ell_up((size_t)Uc * std::max(wu, 1), kEllNone);
  std::vector<uint8_t> cnt_dn(Dc), wmax_dn((Dc + 31) / 32, 0);
  for (int r = 0; r < Dc; r++) {
    for (size_t k = 0; k < rows_dn[r].size(); k++) ell_dn[k * (size_t)Dc + r] = rows_dn[r][k];
    cnt_dn[r] = (uint8_t)rows_dn[r].size();
    wmax_dn[r >> 5] = std::max<uint8_t>(wmax_dn[r >> 5], cnt_dn[r]);
  }
  for (int r = 0; r < Uc; r++)
    for (size_t k = 0; k < rows_up[r].size(); k++) ell_up[(size_t)r * std::max(wu, 1) + k] = rows_up[r][k];
  // diagonal: per-species parts, on-site cross terms, or the full diagonal
  const uint64_t even = 0x5555555555555555ull, odd = even << 1;
  std::vector<double> du(Uc, 0.0), dd(Dc, 0.0), usite(N, 0.0);
  bool general_cross = false;
  std::vector<DiagTerm> up_t, dn_t;
  for (const DiagTerm &t : m.diag) {
    if ((t.cm & odd) == 0) up_t.push_back(t);
    else if ((t.cm & even) == 0) dn_t.push_back(t);
    else {
      const int i = __builtin_ctzll(t.cm) >> 1;
      const uint64_t site = 3ull << (2 * i);
      if (t.cm == site && t.cv == site) usite[i] += t.v;
      else general_cross = true;
    }
  }
  for (int r = 0; r < Uc; r++) {
    const uint64_t c = spread_species(unrank_up[r], 0, N);
    for (const DiagTerm &t : up_t)
      if ((c & t.cm) == t.cv) du[r] += t.v;
  }
  for (int r = 0; r < Dc; r++) {
    const uint64_t c = spread_species(unrank_dn[r], 1, N);
    for (const DiagTerm &t : dn_t)
      if ((c & t.cm) == t.cv) dd[r] += t.v;
  }
  // Row processing order.  Up hops read whole source rows; rows processed close together in
  // time share sources in L2 when the order follows the hop graph.  Default: Cuthill-McKee
  // (breadth-first from a minimum-degree row, neighbours by increasing degree);
  // HPHI_B200_ROW_ORDER=natural keeps the rank order.
  std::vector<int> order(Uc);
  {
    const char *ro = getenv("HPHI_B200_ROW_ORDER");
    if (ro && std::string(ro) == "natural") {
      for (int r = 0; r < Uc; r++) order[r] = r;
    } else {
      std::vector<char> seen(Uc, 0);
      int n = 0;
      while (n < Uc) {
        int start = -1;
        for (int r = 0; r < Uc; r++)
          if (!seen[r] && (start < 0 || rows_up[r].size() < rows_up[start].size())) start = r;
        size_t head = n;
        order[n++] = start;
        seen[start] = 1;
        while (head < (size_t)n) {
          const int r = order[head++];
          std::vector<int> nb;
          for (uint32_t e : rows_up[r]) {
            const int q = (int)(e & 0xFFFFu);
            if (!seen[q]) { seen[q] = 1; nb.push_back(q); }
          }
          std::stable_sort(nb.begin(), nb.end(), [&](int x, int y) { return rows_up[x].size() < rows_up[y].size(); });
          for (int q : nb) order[n++] = q;
        }
      }
    }
  }
  ProdPlan *p = new ProdPlan();
  ProdArgs &a = p->args;
  a.N = N;
  a.Uc = Uc;
  a.Dc = Dc;
  a.wd = wd;
  a.wu = wu;
  bool uniform = true;
  for (int i = 1; i < N; i++) uniform = uniform && (usite[i] == usite[0]);
  a.cross_mode = general_cross ? 2 : (uniform ? 0 : 1);
  a.u0 = usite[0];
  std::vector<double> utab(17);
  for (int k = 0; k <= 16; k++) utab[k] = a.u0 * (double)k;
  auto fail = [&]() { prod_plan_free(p); return -1; };
  if (upload(p, rank, &a.rank, err) || upload(p, pos_dn, &a.pos_dn, err) || upload(p, unrank_up, &a.unrank_up, err) ||
      upload(p, unrank_dn, &a.unrank_dn, err) || upload(p, ell_dn, &a.ell_dn, err) ||
      upload(p, ell_up, &a.ell_up, err) || upload(p, coef_table(hops[1]), &a.cf_dn, err) ||
      upload(p, coef_table(hops[0]), &a.cf_up, err) || upload(p, du, &a.du, err) || upload(p, dd, &a.dd, err) ||
      upload(p, usite, &a.usite, err) || upload(p, order, &a.order, err) || upload(p, cnt_dn, &a.cnt_dn, err) ||
      upload(p, wmax_dn, &a.wmax_dn, err) || upload(p, utab, &a.utab, err))
    return fail();
  if (a.cross_mode == 2) {
    void *q = nullptr;
    if (cudaMalloc(&q, sizeof(double) * (size_t)s->dim) != cudaSuccess) {
      *err = "product plan: device allocation failed";
      return fail();
    }
    p->allocs.push_back(q);
    const unsigned nb = (unsigned)std::min<int64_t>((s->dim + 255) / 256, (int64_t)s->num_sms * 16);
    prod_permute_diag_kernel<<<nb, 256, 0, s->stream>>>(s->dim, N, Dc, s->d_list_1, a.rank, a.pos_dn, s->d_diag, (double *)q);
    if (cudaStreamSynchronize(s->stream) != cudaSuccess) {
      *err = "product plan: diagonal permutation failed";
      return fail();
    }
    a.dfull = (const double *)q;
  }
  if (cudaMalloc(&p->part, sizeof(double) * 2 * (size_t)Uc) != cudaSuccess ||
      cudaMalloc(&p->counter, 2 * sizeof(int)) != cudaSuccess) {
    *err = "product plan: device allocation failed";
    return fail();
  }
  p->allocs.push_back(p->part);
  p->allocs.push_back(p->counter);
  if (cudaMemset(p->counter, 0, 2 * sizeof(int)) != cudaSuccess) {
    *err = "product plan: clear failed";
    return fail();
  }
  p->smem[0] = smem_r;
  p->smem[1] = smem_c;
  if (raise_smem_limit((const void *)prod_hv_kernel<double>, smem_r) != cudaSuccess ||
      raise_smem_limit((const void *)prod_hv_kernel<cplx>, smem_c) != cudaSuccess) {
    *err = "product plan: shared-memory attribute rejected";
    return fail();
  }
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, prod_hv_kernel<double>, kProdThreads, smem_r);
  p->grid = std::max(1, std::min(Uc, std::max(1, per_sm) * s->num_sms));
  p->uniform = uniform_hops;
  // without them the one-pass kernel remains
  if (two_pass_ok && two_pass_build(s, p, rows_dn, rows_up, G, err) != 0) cudaGetLastError();
  p->rank.swap(rank);
  p->pos_dn.swap(pos_dn);
  p->unrank_up.swap(unrank_up);
  p->unrank_dn.swap(unrank_dn);
  if (perm_tasks_build(s, p, err) != 0) cudaGetLastError();  // a thread per row then
  s->prod = p;
  return 0;
}

// The kernel number that hphi_info reports: 3 for hops of one real magnitude per species.
bool prod_two_pass(const Sector *s) { return s->prod && s->prod->two_pass && s->prod->uniform; }

int prod_row_words(const Sector *s) { return s->prod->two_pass ? s->prod->stride : 0; }

size_t prod_scratch_doubles(const Sector *s, VecType vt) {
  const ProdPlan *p = s->prod;
  // the two-pass kernels keep one partial sum per CTA of each pass, the one-pass kernel one per
  // row; callers with a fixed scratch (hphi_mltply_device_noalloc) are told of the latter for every
  // input but real vectors under uniform hops, so the sectors they refuse stay the same
  const size_t two = p->two_pass ? 2 * (size_t)(p->grid_row[vt == kReal64 ? 0 : 1] + p->grid_col) : 0;
  if (p->two_pass && p->uniform && vt == kReal64) return two;
  return std::max(two, 2 * (size_t)p->args.Uc);
}

namespace {
// Row pass then column pass; partial sums at d_part (grid_row + grid_col records of 2).
void two_pass_launch(Sector *s, const ProdPlan *p, bool cv, const double *v1, double *v0, const double *d_coef,
                     double *d_out, double *d_part, const LanczosTail *lt, const TaylorSum &ts = TaylorSum{}) {
  const int gr = p->grid_row[cv], gc = p->grid_col;
  with_row_kernel(p->stride, cv, p->args.cross_mode == 0, [&](auto kernel, auto shape) {
    using S = decltype(shape);
    kernel<<<gr, S::threads, sizeof(double) * (size_t)S::P * p->stride, s->stream>>>(p->args, p->tp, v1, v0, d_coef, d_part);
  });
  const SumOut so = sum_out(d_part, gr, gr + gc, s->d_done, d_out, 0, lt);
  // 16-byte loads where every row starts on a 16-byte boundary
  const bool v2 = cv || ((p->args.Dc % 2 == 0) && ((((uintptr_t)v1) | ((uintptr_t)v0)) % 16 == 0));
#define HPHI_COL_T(V, C, M, T) \
  prod_col_kernel<V, C, M, T><<<gc, kUpThreads, 0, s->stream>>>(p->args, p->tp, v1, v0, d_coef, so, ts)
#define HPHI_COL(V, C, M) HPHI_COL_T(V, C, M, false)
  if (cv && ts.sum) {
    if (p->multi_up) HPHI_COL_T(2, true, true, true);
    else HPHI_COL_T(2, true, false, true);
  } else if (cv) {
    if (p->multi_up) HPHI_COL(2, true, true);
    else HPHI_COL(2, true, false);
  } else if (v2) {
    if (p->multi_up) HPHI_COL(2, false, true);
    else HPHI_COL(2, false, false);
  } else {
    if (p->multi_up) HPHI_COL(1, false, true);
    else HPHI_COL(1, false, false);
  }
#undef HPHI_COL
#undef HPHI_COL_T
}

int prod_launch(Sector *s, VecType vt, const void *d_v1, void *d_v0, const double *d_coef, double *d_out, double *d_part,
                int *d_counter, const LanczosTail *lt, bool one_pass = false) {
  ProdPlan *p = s->prod;
  if (vt == kReal64 && s->model.complex_terms) {
    set_error("H has complex coefficients: real vectors are not allowed");
    return -1;
  }
  if (!whole_elements(vt, d_v1) || !whole_elements(vt, d_v0)) {
    if (p->args.wu > 0) {  // the source rows of up hops are read in whole elements
      set_error("complex vectors in native order must start at a multiple of 16 bytes");
      return -1;
    }
    one_pass = true;
  }
  if (p->two_pass && !one_pass) {
    two_pass_launch(s, p, vt != kReal64, (const double *)d_v1, (double *)d_v0, d_coef, d_out, d_part, lt);
    return cuda_ok(cudaGetLastError(), "launch");
  }
  if (vt == kReal64)
    prod_hv_kernel<double><<<p->grid, kProdThreads, p->smem[0], s->stream>>>(
        p->args, (const double *)d_v1, (double *)d_v0, d_coef, d_part, d_counter);
  else
    prod_hv_kernel<cplx><<<p->grid, kProdThreads, p->smem[1], s->stream>>>(p->args, (const cplx *)d_v1,
                                                                           (cplx *)d_v0, d_coef, d_part, d_counter);
  finalize_partials_kernel<2><<<1, 256, 0, s->stream>>>(d_part, p->args.Uc, d_out);
  if (cuda_ok(cudaGetLastError(), "launch") != 0) return -1;
  return lt ? lanczos_scalars(s, 0, lt->k, lt->st, lt->alpha, lt->beta) : 0;
}
}  // namespace

int prod_hv_launch_scratch(Sector *s, VecType vt, const void *d_v1, void *d_v0, const double *d_coef, double *d_out,
                           double *d_part, int *d_counter) {
  const bool one_pass = !s->prod->two_pass || !whole_elements(vt, d_v1) || !whole_elements(vt, d_v0);
  if (one_pass && cudaMemsetAsync(d_counter, 0, 2 * sizeof(int), s->stream) != cudaSuccess) {
    set_error("product kernel: clearing the row counter failed");
    return -1;
  }
  return prod_launch(s, vt, d_v1, d_v0, d_coef, d_out, d_part, d_counter, nullptr);
}

int prod_hv_launch(Sector *s, VecType vt, const void *d_v1, void *d_v0, const double *d_coef, double *d_out,
                   const LanczosTail *lt) {
  return prod_launch(s, vt, d_v1, d_v0, d_coef, d_out, s->prod->part, s->prod->counter, lt);
}

// By the one-pass kernel: <v1|H v1> of complex vectors as the sum of its per-row sums.  All there
// is of that sum's imaginary part is its rounding, so a call that hands both parts to its caller
// keeps the order of the additions.
int prod_hv_launch_rows(Sector *s, VecType vt, const void *d_v1, void *d_v0, const double *d_coef, double *d_out) {
  return prod_launch(s, vt, d_v1, d_v0, d_coef, d_out, s->prod->part, s->prod->counter, nullptr, true);
}

// Time evolution: H(t) = the static terms plus those of a time index.  The plan holds the hops
// of all indices once and a coefficient per group and index; its positions and diagonal are the
// static plan's, so vectors, permutations and observables are those of s->prod.  *out stays
// null where the two-pass kernels do not apply (terms other than hops, more coefficient groups
// than kMaxGroups).
int prod_te_plan_build(Sector *s, const std::vector<BitTerm> &terms, const std::vector<std::vector<double2>> &coefs,
                       ProdPlan **out, std::string *err) {
  *out = nullptr;
  const ProdPlan *base = s->prod;
  if (!base || coefs.empty() || base->args.Dc + 16 > 12896) return 0;
  std::vector<SpeciesHop> hops[2];
  std::vector<std::vector<double2>> seq[2];
  for (auto &q : seq) q.resize(coefs.size());
  for (size_t t = 0; t < terms.size(); t++) {
    SpeciesHop h;
    int sp;
    BitTerm unit = terms[t];  // the term's sign alone
    unit.re = 1.0;
    unit.im = 0.0;
    if (!species_hop(unit, &h, &sp)) return 0;
    hops[sp].push_back(h);
    for (size_t k = 0; k < coefs.size(); k++)
      seq[sp][k].push_back(make_double2(h.re * coefs[k][t].x, h.re * coefs[k][t].y));
  }
  if (hops[1].empty() || hops[0].size() > 16000 || hops[1].size() > 16000) return 0;
  HopGroups G[2];
  if (!coef_groups(seq[0], &G[0]) || !coef_groups(seq[1], &G[1])) return 0;
  std::vector<std::vector<uint32_t>> rows_dn, rows_up;
  int wd = 0, wu = 0;
  build_ell(hops[1], base->unrank_dn, base->pos_dn, &rows_dn, &wd);
  build_ell(hops[0], base->unrank_up, base->rank, &rows_up, &wu);
  if (wd > 255 || wu > 64) return 0;
  ProdPlan *p = new ProdPlan();
  p->args = base->args;
  if (two_pass_build(s, p, rows_dn, rows_up, G, err) != 0) cudaGetLastError();
  if (!p->two_pass) {
    prod_plan_free(p);
    return 0;
  }
  *out = p;
  return 0;
}

int prod_te_launch(Sector *s, const ProdPlan *te, int index, const void *d_v1, void *d_v0, const double *d_coef,
                   double *d_out, void *d_sum, double c_re, double c_im) {
  ProdPlan p;  // the tables of this index's coefficients
  p.args = te->args;
  p.tp = te->tp;
  p.tp.cf_dn += (size_t)index * te->tp.ng;
  p.tp.cf_up += (size_t)index * te->tp.ngu;
  p.stride = te->stride;
  p.multi_up = te->multi_up;
  p.grid_row[1] = te->grid_row[1];
  p.grid_col = te->grid_col;
  two_pass_launch(s, &p, true, (const double *)d_v1, (double *)d_v0, d_coef, d_out, te->part, nullptr,
                  TaylorSum{(double2 *)d_sum, make_double2(c_re, c_im)});
  return cuda_ok(cudaGetLastError(), "launch");
}

int prod_permute(Sector *s, VecType vt, const void *in, void *out, bool to_native) {
  const ProdPlan *p = s->prod;
  const ProdArgs &a = p->args;
  const bool whole = whole_elements(vt, in);
  if (p->nperm == 0 || s->dim < (int64_t)kPermShort * p->nperm || !whole) {
    const unsigned nb = (unsigned)std::min<int64_t>((s->dim + kPermThreads - 1) / kPermThreads, (int64_t)s->num_sms * 16);
    auto rows = [&](auto *x, auto *y, auto w) {
      using T = std::remove_reference_t<decltype(*y)>;
      constexpr bool W = decltype(w)::value;
      if (to_native)
        prod_permute_rows_kernel<T, true, W><<<nb, kPermThreads, 0, s->stream>>>(s->dim, a.Dc, s->d_list_1, a.rank, a.pos_dn, x, y);
      else
        prod_permute_rows_kernel<T, false, W><<<nb, kPermThreads, 0, s->stream>>>(s->dim, a.Dc, s->d_list_1, a.rank, a.pos_dn, x, y);
    };
    if (vt == kReal64) rows((const double *)in, (double *)out, std::true_type{});
    else if (whole) rows((const cplx *)in, (cplx *)out, std::true_type{});
    else rows((const cplx *)in, (cplx *)out, std::false_type{});
    return cuda_ok(cudaGetLastError(), "permute");
  }
  if (to_native) {
    const unsigned nb = (unsigned)std::min(a.Uc, s->num_sms * 8);
    if (vt == kReal64)
      prod_to_native_kernel<double><<<nb, kPermThreads, 0, s->stream>>>(
          a.N, a.Uc, a.Dc, a.unrank_up, a.unrank_dn, s->d_list_2_1, s->d_list_2_2, (const double *)in, (double *)out);
    else
      prod_to_native_kernel<cplx><<<nb, kPermThreads, 0, s->stream>>>(
          a.N, a.Uc, a.Dc, a.unrank_up, a.unrank_dn, s->d_list_2_1, s->d_list_2_2, (const cplx *)in, (cplx *)out);
  } else {
    const unsigned nb = (unsigned)std::min((p->nperm + 7) / 8, s->num_sms * 8);
    if (vt == kReal64)
      prod_from_native_kernel<double><<<nb, kPermThreads, 0, s->stream>>>(a.N, a.Dc, p->perm, p->nperm, p->perm_low, a.rank,
                                                                          a.pos_dn, (const double *)in, (double *)out);
    else
      prod_from_native_kernel<cplx><<<nb, kPermThreads, 0, s->stream>>>(a.N, a.Dc, p->perm, p->nperm, p->perm_low, a.rank,
                                                                        a.pos_dn, (const cplx *)in, (cplx *)out);
  }
  return cuda_ok(cudaGetLastError(), "permute");
}

int prod_observables(Sector *s, VecType vt, const void *v, double *d_out) {
  ProdPlan *p = s->prod;
  const int nb = s->red_blocks;
  const SumOut so = sum_out(s->d_red, 0, nb, s->d_done, d_out);
  if (vt == kReal64)
    prod_obs_kernel<double><<<nb, 256, 0, s->stream>>>(p->args, (const double *)v, so);
  else
    prod_obs_kernel<cplx><<<nb, 256, 0, s->stream>>>(p->args, (const cplx *)v, so);
  return cuda_ok(cudaGetLastError(), "observables");
}

}  // namespace hphi
