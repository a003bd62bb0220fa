// Tile kernel for grand-canonical sectors whose rows are their configurations (hv_gc.cu).
#pragma once
#include <string>

#include "engine.hpp"

namespace hphi {

struct GcPlan;
void gc_plan_build(Sector *s);
void gc_plan_free(GcPlan *p);
bool gc_applies(const Sector *s, VecType vt);
int gc_passes(const Sector *s, VecType vt);
size_t gc_scratch_doubles(const Sector *s, VecType vt);
double *gc_part(const Sector *s);
int gc_hv_launch(Sector *s, VecType vt, const void *d_v1, void *d_v0, const double *d_coef, double *d_out,
                 double *d_part, const LanczosTail *lt);

}  // namespace hphi
