// Block kernel: one-pass H*v for canonical sectors in HPhi's row order (Spin, general spin,
// Kondo, HubbardNConserved), whose vectors fit in L2 or which have no row-block plan.
//
// HPhi's rows come in blocks that share the upper half of the configuration (sector_blocks); the
// blocks whose lower halves are the same, in the same order, form a class.  Of a term's masks
//   in the lower half:  the term moves a row within its block, the same way in every block of the
//                       class: a gather table per class, decoded once for all blocks of a task;
//   in the upper half:  it moves a whole block, position for position: one row shift per block;
//   in both:            it acts on the blocks whose upper half matches; its source position
//                       follows from the lower half (a table per class and flipped bit).
// A task is P planes of one class: P blocks of a real vector, or the real and imaginary parts of
// P / 2 blocks of a complex one.  The planes are staged in shared memory, where the lower-half
// terms are edge-coloured gathers (gather_warp: no bank conflicts, 16-bit entries); upper
// and crossing terms are listed per block when the plan is made (source block and coefficient)
// and read v1 in (nearly) consecutive pieces from L2.  The general kernel (hv.cu) spends three
// scattered L1 requests per matrix element (entry, coefficient, source) and is bound by them;
// here an element is one shared-memory word or one coalesced load.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdint>
#include <map>
#include <string>
#include <vector>

#include "block_tables.hpp"
#include "device_util.cuh"
#include "engine.hpp"
#include "hv_blocks.hpp"
#include "plan_upload.hpp"
#include "tma.cuh"

namespace hphi {
namespace {

template <int ID> struct BkShape {
  static constexpr int stride = kBkShapeDefs[ID].stride, P = kBkShapeDefs[ID].P, Q = kBkShapeDefs[ID].Q,
                       U = kBkShapeDefs[ID].U, threads = kBkShapeDefs[ID].threads, ctas = kBkShapeDefs[ID].ctas;
};

struct BkArgs {
  int ncls, ng, nlist;     // nlist: BlockTables
  const BkClass *cls;
  const uint32_t *b_row0;  // per block, by class: its first row
  const uint2 *b_list;     // its first record, and numbers of upper (low half) and crossing terms
  const BkRec *rec;
  const double *rec_im;    // imaginary parts of the records' coefficients (nullptr: none)
  const uint4 *gat;
  const uint2 *head;
  const double2 *cf;       // [ng]
  const uint16_t *tab;     // source position | sign << 15 of each position, kBkNone: not matched
};

template <typename T> struct BkVal;
template <> struct BkVal<double> {
  static constexpr int W = 1;
  static __device__ __forceinline__ double ld(const double *p) { return __ldg(p); }
  static __device__ __forceinline__ double get(const double *pl, int stride) { return pl[0]; }
};
template <> struct BkVal<cplx> {
  static constexpr int W = 2;
  static __device__ __forceinline__ cplx ld(const cplx *p) {
    const double2 z = __ldg(reinterpret_cast<const double2 *>(p));
    return cplx{z.x, z.y};
  }
  static __device__ __forceinline__ cplx get(const double *pl, int stride) { return cplx{pl[0], pl[stride]}; }
};

// IM: some listed coefficient has an imaginary part (complex vectors only).
template <int ID, typename T, bool IM>
__global__ void __launch_bounds__(BkShape<ID>::threads, BkShape<ID>::ctas)
bk_kernel(BkArgs a, const BkTask *__restrict__ tasks, int ntask, const double *__restrict__ diag,
          const T *__restrict__ v1, T *__restrict__ v0, const double *__restrict__ coef, SumOut so) {
  // launched while the kernel before it ends (launch_chained): everything below waits for that one
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  const double acc = coef[0], scale = coef[1];
  using S = BkShape<ID>;
  constexpr int STRIDE = S::stride, P = S::P, Q = S::Q, NT = S::threads;
  constexpr int W = BkVal<T>::W, R = P / W;  // R blocks per task
  constexpr uint32_t U = S::U;               // listed terms in flight per block and position
  extern __shared__ __align__(16) double planes[];
  BkRec *s_rec = reinterpret_cast<BkRec *>(planes + P * STRIDE);   // [R][nlist]
  double *s_im = reinterpret_cast<double *>(s_rec + R * a.nlist);  // [R][nlist] (IM)
  __shared__ double2 s_c[kBkGroups];
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid < a.ng) s_c[tid] = a.cf[tid];
  double pr[2] = {0.0, 0.0};
  for (int t = blockIdx.x; t < ntask; t += gridDim.x) {
    // block r of the task: its first row, lists and vector (planes past the last repeat it)
    uint32_t row0[R], nh[R], nx[R], hmin = ~0u, hmax = 0, xmax = 0;
    const uint4 tk = __ldg(reinterpret_cast<const uint4 *>(tasks) + t);
    const int nr = (R == 2 && tk.z != ~0u) ? 2 : 1;
    uint32_t blk[R];
    blk[0] = tk.y;
    if (R == 2) blk[R - 1] = nr == 2 ? tk.z : tk.y;
    const BkClass C = a.cls[tk.x];
    const int n = C.n, npad = (int)(tk.w >> 16), end = min(n, npad);  // npad: whole warps
    __syncthreads();  // the previous task's planes and lists are no longer read
#pragma unroll
    for (int r = 0; r < R; r++) {
      row0[r] = __ldg(a.b_row0 + blk[r]);
      const uint2 li = __ldg(a.b_list + blk[r]);
      nh[r] = li.y & 0xFFFFu;
      nx[r] = li.y >> 16;
      hmin = min(hmin, nh[r]);
      hmax = max(hmax, nh[r]);
      xmax = max(xmax, nx[r]);
      if constexpr (W == 1) {
        const uint32_t to = smem_u32(planes + r * STRIDE);
        for (int i = tid; i < n; i += NT)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(to + 8 * i), "l"(v1 + row0[r] + i) : "memory");
      } else {
        for (int i = tid; i < n; i += NT) {
          const cplx z = BkVal<T>::ld(v1 + row0[r] + i);
          planes[2 * r * STRIDE + i] = z.x;
          planes[(2 * r + 1) * STRIDE + i] = z.y;
        }
      }
      for (int k = tid; k < (int)(nh[r] + nx[r]); k += NT) {
        *(reinterpret_cast<uint4 *>(s_rec + r * a.nlist) + k) = __ldg(reinterpret_cast<const uint4 *>(a.rec + li.x) + k);
        if (IM) s_im[r * a.nlist + k] = __ldg(a.rec_im + li.x + k);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    for (int k = tid; k < 16 * P; k += NT) planes[(k >> 4) * STRIDE + n + (k & 15)] = 0.0;  // the empty slots' words
    const uint2 *headp = a.head + C.head;
    const uint4 *gatp = a.gat + C.gat + lane;
    const uint16_t *tabp = a.tab;
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    const char *rb = reinterpret_cast<const char *>(planes);
    // A position's loads (slots, diagonal, old v0, the first upper-half terms) are issued before
    // the gathers, and later ones several at a time: waits for L2 are what this loop is made of.
    for (int p0 = (int)(tk.w & 0xFFFFu) + tid; p0 < npad; p0 += Q * NT) {
      int p[Q];
      bool in[Q];
      uint2 head[Q];
      uint4 e4[Q];
      double dg[Q][R], y[Q][P];
      T old[Q][R], z[U][R][Q];
#pragma unroll
      for (int q = 0; q < Q; q++) {
        p[q] = p0 + q * NT;
        in[q] = p[q] < end;
        head[q] = make_uint2(0u, 0u);
        e4[q] = make_uint4(0u, 0u, 0u, 0u);
        if (p[q] < npad) {  // the same for the warp
          head[q] = __ldg(headp + (p[q] >> 5));
          e4[q] = __ldg(gatp + (int64_t)(p[q] >> 5) * C.sets * 32);
        }
#pragma unroll
        for (int r = 0; r < R; r++) {
          dg[q][r] = 0.0;
          old[q][r] = VT<T>::zero();
          if (in[q]) {
            dg[q][r] = __ldg(diag + row0[r] + p[q]);
            if (acc != 0.0) old[q][r] = v0[(int64_t)row0[r] + p[q]];
          }
        }
#pragma unroll
        for (int k = 0; k < P; k++) y[q][k] = 0.0;
      }
      // the loads of terms e .. e + U; TAIL: some may be past a block's list
      auto hi_load = [&](uint32_t e, bool tail) {
#pragma unroll
        for (uint32_t u = 0; u < U; u++)
#pragma unroll
          for (int r = 0; r < R; r++) {
            if (tail && e + u >= nh[r]) continue;
            const T *at = v1 + (s_rec[r * a.nlist + e + u].row + (uint32_t)p0);
#pragma unroll
            for (int q = 0; q < Q; q++)
              if (in[q]) z[u][r][q] = BkVal<T>::ld(at + q * NT);
          }
      };
      auto add = [&](int q, int r, double cr, double ci, const T &x) {
        if constexpr (W == 2) {
          y[q][2 * r] = fma(cr, x.x, y[q][2 * r]);
          y[q][2 * r + 1] = fma(cr, x.y, y[q][2 * r + 1]);
          if (IM) {
            y[q][2 * r] = fma(-ci, x.y, y[q][2 * r]);
            y[q][2 * r + 1] = fma(ci, x.x, y[q][2 * r + 1]);
          }
        } else {
          y[q][r] = fma(cr, x, y[q][r]);
        }
      };
      auto im_of = [&](int r, uint32_t e) { return IM ? s_im[r * a.nlist + e] : 0.0; };
      auto hi_add = [&](uint32_t e, bool tail) {
#pragma unroll
        for (uint32_t u = 0; u < U; u++)
#pragma unroll
          for (int r = 0; r < R; r++) {
            if (tail && e + u >= nh[r]) continue;
            const double c = s_rec[r * a.nlist + e + u].re, ci = im_of(r, e + u);
#pragma unroll
            for (int q = 0; q < Q; q++)
              if (in[q]) add(q, r, c, ci, z[u][r][q]);
          }
      };
      const bool tail0 = U > hmin;
      hi_load(0, tail0);
#pragma unroll
      for (int q = 0; q < Q; q++) {
        if (p[q] >= npad) break;
        const uint4 *gp = gatp + (int64_t)(p[q] >> 5) * C.sets * 32;
        uint4 e = e4[q];
        for (int k = 0; k < a.ng; k++) {
          const int ns = (int)(((k < 4 ? head[q].x : head[q].y) >> (8 * (k & 3))) & 255u);
          double s[P];
#pragma unroll
          for (int c = 0; c < P; c++) s[c] = 0.0;
          auto gather2 = [&](uint32_t h) {  // two entries: word | sign << 15, the sign as a factor +-1
            const double *x0 = reinterpret_cast<const double *>(rb + ((h << 3) & 0x3FFF8u));
            const double *x1 = reinterpret_cast<const double *>(rb + ((h >> 13) & 0x3FFF8u));
            const double f0 = __hiloint2double((int)(((h << 16) & 0x80000000u) | 0x3FF00000u), 0);
            const double f1 = __hiloint2double((int)((h & 0x80000000u) | 0x3FF00000u), 0);
#pragma unroll
            for (int c = 0; c < P; c++) s[c] = fma(f0, x0[c * STRIDE], s[c]);
#pragma unroll
            for (int c = 0; c < P; c++) s[c] = fma(f1, x1[c * STRIDE], s[c]);
          };
          for (int j = 0; j < ns; j += 8) {
            const uint4 w = e;
            gp += 32;
            e = __ldg(gp);  // the next set (one past a warp's last is allocated)
            gather2(w.x);
            gather2(w.y);
            if (j + 4 < ns) {
              gather2(w.z);
              gather2(w.w);
            }
          }
          const double2 c = s_c[k];
#pragma unroll
          for (int r = 0; r < R; r++) {
            if constexpr (W == 2) {
              y[q][2 * r] += c.x * s[2 * r] - c.y * s[2 * r + 1];
              y[q][2 * r + 1] += c.x * s[2 * r + 1] + c.y * s[2 * r];
            } else {
              y[q][r] = fma(c.x, s[r], y[q][r]);
            }
          }
        }
      }
      // upper-half terms: the task's blocks side by side
      hi_add(0, tail0);
      uint32_t e = U;
      for (; e + U <= hmin; e += U) {
        hi_load(e, false);
        hi_add(e, false);
      }
      for (; e < hmax; e += U) {
        hi_load(e, true);
        hi_add(e, true);
      }
      // crossing terms: the source positions from the table, then the elements
      for (uint32_t i = 0; i < xmax; i += U) {
        uint32_t tb[U][R][Q];
#pragma unroll
        for (uint32_t u = 0; u < U; u++)
#pragma unroll
          for (int r = 0; r < R; r++) {
            const uint16_t *at = tabp + s_rec[r * a.nlist + nh[r] + i + u].tab + p0;
#pragma unroll
            for (int q = 0; q < Q; q++) tb[u][r][q] = (i + u < nx[r] && in[q]) ? __ldg(at + q * NT) : kBkNone;
          }
#pragma unroll
        for (uint32_t u = 0; u < U; u++)
#pragma unroll
          for (int r = 0; r < R; r++) {
            const T *at = v1 + s_rec[r * a.nlist + nh[r] + i + u].row;
#pragma unroll
            for (int q = 0; q < Q; q++)
              if ((tb[u][r][q] & 0x7FFFu) != kBkNone) z[u][r][q] = BkVal<T>::ld(at + (tb[u][r][q] & 0x7FFFu));
          }
#pragma unroll
        for (uint32_t u = 0; u < U; u++)
#pragma unroll
          for (int r = 0; r < R; r++) {
            const double c = s_rec[r * a.nlist + nh[r] + i + u].re, ci = im_of(r, nh[r] + i + u);
#pragma unroll
            for (int q = 0; q < Q; q++)
              if ((tb[u][r][q] & 0x7FFFu) != kBkNone) {
                const int sg = (int)((tb[u][r][q] & 0x8000u) << 16);
                add(q, r, __hiloint2double(__double2hiint(c) ^ sg, __double2loint(c)),
                    __hiloint2double(__double2hiint(ci) ^ sg, __double2loint(ci)), z[u][r][q]);
              }
          }
      }
#pragma unroll
      for (int q = 0; q < Q; q++)
#pragma unroll
        for (int r = 0; r < R; r++) {
          if (!in[q] || r >= nr) continue;
          const T x = BkVal<T>::get(planes + W * r * STRIDE + p[q], STRIDE);
          T yy;
          if constexpr (W == 2) yy = cplx{y[q][2 * r], y[q][2 * r + 1]};
          else yy = y[q][r];
          yy = VT<T>::add(yy, VT<T>::scale(dg[q][r], x));
          pr[0] += VT<T>::conj_mul_re(x, yy);
          pr[1] += VT<T>::conj_mul_im(x, yy);
          const T ys = VT<T>::scale(scale, yy);
          v0[(int64_t)row0[r] + p[q]] = (acc == 0.0) ? ys : VT<T>::add(VT<T>::scale(acc, old[q][r]), ys);
        }
    }
  }
  if (so.done) {
    grid_sum<2>(pr, so);
  } else {  // the column pass sums these records with its own
    block_sum<2>(pr);
    if (tid == 0) {
      so.part[2 * blockIdx.x] = pr[0];
      so.part[2 * blockIdx.x + 1] = pr[1];
    }
  }
}

}  // namespace

struct BlockPlan {
  BkArgs args{};
  std::vector<void *> allocs;
  int shape = 0;               // BkShape
  int ntask[2] = {0, 0};       // real, complex vectors
  const BkTask *tasks[2] = {nullptr, nullptr};
  bool two_pass = false;       // lower-half and crossing terms only: the row-block plan's row pass
  bool im = false;             // complex coefficients in the lists
  size_t smem[2] = {0, 0};
  int grid[2] = {0, 0};        // resident CTAs
};

void bk_plan_free(BlockPlan *p) {
  if (!p) return;
  for (void *q : p->allocs) cudaFree(q);
  delete p;
}

namespace {

template <typename F>
void with_bk_shape(int id, F f) {
  switch (id) {
    case 0: f(std::integral_constant<int, 0>{}); break;
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    default: f(std::integral_constant<int, 7>{}); break;
  }
}

}  // namespace

// Leaves s->bk null where the plan does not apply (block_tables) or there is no memory for it: the
// general kernel remains.
void bk_plan_build(Sector *s, bool two_pass) {
  s->bk = nullptr;
  if (s->gc || !s->d_list_1 || s->lo_bits > 20 || s->hi_bits > 20 || s->model.offdiag.empty()) return;
  std::vector<SectorBlock> blk;
  std::vector<uint32_t> low, l22(s->sdim);
  std::string why;
  if (sector_blocks(s, &blk, &low, &why) != 0 ||
      cudaMemcpy(l22.data(), s->d_list_2_2, sizeof(uint32_t) * l22.size(), cudaMemcpyDeviceToHost) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  BlockTables t;
  if (!block_tables(s->model.offdiag, s->lo_bits, l22, blk, low, s->dim, two_pass, &t)) return;
  BlockPlan *p = new BlockPlan();
  BkArgs &a = p->args;
  a.ncls = (int)t.cls.size();
  a.ng = (int)t.cf.size();
  a.nlist = t.nlist;
  p->im = t.im;
  p->two_pass = two_pass;
  p->shape = t.shape;
  bool fits = true;
  with_bk_shape(p->shape, [&](auto st) {
    using S = BkShape<decltype(st)::value>;
    for (int cv = 0; cv < 2; cv++) {
      const int R = S::P / (cv ? 2 : 1);
      constexpr int ST = decltype(st)::value;
      p->smem[cv] = sizeof(double) * (size_t)S::P * S::stride + (sizeof(BkRec) + (t.im ? sizeof(double) : 0)) * a.nlist * (size_t)R;
      const void *f = !cv ? (const void *)bk_kernel<ST, double, false>
                          : t.im ? (const void *)bk_kernel<ST, cplx, true> : (const void *)bk_kernel<ST, cplx, false>;
      int per_sm = 0;
      if (p->smem[cv] > 227 * 1024 || raise_smem_limit(f, p->smem[cv]) != cudaSuccess ||
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, S::threads, p->smem[cv]) != cudaSuccess || per_sm < 1)
        fits = false;
      p->grid[cv] = std::max(1, std::min(per_sm, 10)) * s->num_sms;
    }
  });
  cudaGetLastError();
  if (!fits) {
    bk_plan_free(p);
    return;
  }
  PlanUpload up;
  up.add(t.cls, &a.cls);
  up.add(t.b_row0, &a.b_row0);
  up.add(t.b_list, &a.b_list);
  up.add(t.rec, &a.rec);
  up.add(t.gat, &a.gat);
  up.add(t.head, &a.head);
  up.add(t.cf, &a.cf);
  up.add(t.tab, &a.tab);
  if (t.im) up.add(t.rec_im, &a.rec_im);
  std::vector<BkTask> tk[2];
  for (int cv = 0; cv < 2; cv++) {
    tk[cv] = block_tasks(t, cv != 0, p->grid[cv]);
    p->ntask[cv] = (int)tk[cv].size();
    up.add(tk[cv], &p->tasks[cv]);
  }
  if (up.run(&p->allocs) != 0) {
    cudaGetLastError();
    bk_plan_free(p);
    return;
  }
  s->bk = p;
}

bool bk_applies(const Sector *s) { return s->bk && !s->bk->two_pass; }
int bk_shape(const Sector *s) { return s->bk->shape; }
bool bk_row_pass(const Sector *s) { return s->bk && s->bk->two_pass; }

int bk_grid(const Sector *s, VecType vt) {
  const int cv = vt == kReal64 ? 0 : 1;
  return std::max(1, std::min(s->bk->grid[cv], s->bk->ntask[cv]));
}

size_t bk_scratch_doubles(const Sector *s) { return 2 * (size_t)std::max(s->bk->grid[0], s->bk->grid[1]); }

int bk_hv_launch(Sector *s, VecType vt, const void *d_v1, void *d_v0, const double *d_coef, double *d_out, double *d_part,
                 const LanczosTail *lt) {
  const BlockPlan *p = s->bk;
  const int cv = vt == kReal64 ? 0 : 1, grid = bk_grid(s, vt);
  // no output: the records are left for a later launch
  const SumOut so = sum_out(d_part, 0, grid, d_out ? s->d_done : nullptr, d_out, 0, lt);
  with_bk_shape(p->shape, [&](auto st) {
    constexpr int ST = decltype(st)::value;
#define HPHI_BK(T, IM)                                                                \
  launch_chained(bk_kernel<ST, T, IM>, grid, BkShape<ST>::threads, p->smem[cv], s->stream, p->args, p->tasks[cv], \
                 p->ntask[cv], (const double *)s->d_diag, (const T *)d_v1, (T *)d_v0, d_coef, so)
    if (!cv) HPHI_BK(double, false);
    else if (p->im) HPHI_BK(cplx, true);
    else HPHI_BK(cplx, false);
#undef HPHI_BK
  });
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error(std::string("block kernel: launch failed: ") + cudaGetErrorString(e));
    return -1;
  }
  return 0;
}

}  // namespace hphi
