// Product-layout kernel for canonical Hubbard models (hv_product.cu).
#pragma once
#include <cstdint>
#include <string>
#include <vector>

#include "engine.hpp"

namespace hphi {

struct ProdPlan;
// Builds the plan when the model qualifies (leaves s->prod null otherwise).
int prod_plan_build(Sector *s, std::string *err);
void prod_plan_free(ProdPlan *p);
// Native-order H*v (see engine.hpp hv_native).
int prod_hv_launch(Sector *s, VecType vt, const void *d_v1, void *d_v0, const double *d_coef, double *d_out,
                   const LanczosTail *lt = nullptr);
// Same with caller-provided row partial sums (prod_scratch_doubles) and row counter (2 ints).
int prod_hv_launch_scratch(Sector *s, VecType vt, const void *d_v1, void *d_v0, const double *d_coef, double *d_out,
                           double *d_part, int *d_counter);
size_t prod_scratch_doubles(const Sector *s, VecType vt);
// Words of a row's plane in the two-pass kernels, 0 where the one-pass kernel runs.
int prod_row_words(const Sector *s);
// True when real vectors take the two-pass kernels (row pass + column pass).
bool prod_two_pass(const Sector *s);
int prod_hv_launch_rows(Sector *s, VecType vt, const void *d_v1, void *d_v0, const double *d_coef, double *d_out);
// Time evolution on the product layout (complex vectors in s->prod's native order):
// terms: off-diagonal terms by mask, coefs[k][t] the coefficient of term t at time index k.
int prod_te_plan_build(Sector *s, const std::vector<BitTerm> &terms, const std::vector<std::vector<double2>> &coefs,
                       ProdPlan **out, std::string *err);
// v0 = coef[0] * v0 + coef[1] * H(index) v1; with d_sum also d_sum += c * v0 (the result).
int prod_te_launch(Sector *s, const ProdPlan *te, int index, const void *d_v1, void *d_v0, const double *d_coef,
                   double *d_out, void *d_sum, double c_re, double c_im);
int prod_permute(Sector *s, VecType vt, const void *in, void *out, bool to_native);
int prod_observables(Sector *s, VecType vt, const void *v, double *d_out);

}  // namespace hphi
