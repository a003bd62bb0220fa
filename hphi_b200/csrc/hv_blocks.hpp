// Block kernel for canonical sectors kept in HPhi's row order (hv_blocks.cu).
#pragma once
#include <string>

#include "engine.hpp"

namespace hphi {

struct BlockPlan;
// two_pass: the row pass of the row-block plan (lower-half and crossing terms only), else all terms.
void bk_plan_build(Sector *s, bool two_pass);
void bk_plan_free(BlockPlan *p);
bool bk_applies(const Sector *s);   // whole H*v in one launch
bool bk_row_pass(const Sector *s);  // the row-block plan's row pass
int bk_shape(const Sector *s);      // kBkShapeDefs
size_t bk_scratch_doubles(const Sector *s);
int bk_grid(const Sector *s, VecType vt);  // CTAs (records of partial sums) of a launch
// v0 = coef[0] * v0 + coef[1] * H v1, sum conj(v1) (H v1) to d_out (and lt); with d_out null the
// partial sums (bk_grid records) stay at d_part.
int bk_hv_launch(Sector *s, VecType vt, const void *d_v1, void *d_v0, const double *d_coef, double *d_out, double *d_part,
                 const LanczosTail *lt);

}  // namespace hphi
