// One step of the differentiable fit and its reverse with the branch-free
// quotient and root (flat_math.cuh), repeated with the plain ones where an
// operand left their range.
#pragma once

#include "kalman.cuh"
#include "adjoint_step.cuh"

namespace mkfg {
namespace adj {

// The material grid with the branch-free quotient and root (flat_math.cuh)
// and the range of the operands they were given.
struct FlatGrid : MatGrid {
  mutable float lo = 1.f, hi = 1.f;
  __device__ __forceinline__ explicit FlatGrid(const MatGrid& g) : MatGrid(g) {}
  __device__ __forceinline__ bool ok() const { return lo >= 0x1p-90f && hi <= 0x1p90f; }
};
__device__ __forceinline__ float ad_div(const FlatGrid&, float a, float b) {
  return flat_div_y(a, b, flat_rcp(b));
}
__device__ __forceinline__ float ad_sqrt(const FlatGrid&, float x) { return flat_sqrt(x); }
__device__ __forceinline__ void ad_see(const FlatGrid& m, float v) {
  m.lo = min_nan(m.lo, fabsf(v));
  m.hi = max_nan(m.hi, fabsf(v));
}
__device__ __forceinline__ void ad_see_top(const FlatGrid& m, float v) { m.hi = max_nan(m.hi, fabsf(v)); }
// The results of a step: dividends are not watched, but a quotient that
// overflowed is NaN, and so is some result (where a maximum could drop the
// NaN, the generated step watches its operand).
template <int N>
__device__ __forceinline__ void ad_see_all(const FlatGrid& m, const float (&v)[N]) {
#pragma unroll
  for (int e = 0; e < N; ++e) ad_see_top(m, v[e]);
}

// The step and its reverse with the plain forms, where an operand left the
// range: not inlined, on copies, so the usual path keeps its registers.
struct StepIn {
  float par[6], err[21], m[3], me[6], ta, tb, tc, k;
};
struct StepState {
  float par[6], err[21], c2;
};
struct StepBars {
  float par[6], err[21], ga, gb, gc;
};
template <bool kMat>
__device__ __noinline__ void step_fwd_plain(const StepIn* x, MatGrid mat, StepState* o) {
  if (kMat)
    barrel_step_fwd_mat(x->par, x->err, x->m, x->me, x->ta, x->tb, x->tc, x->k, mat, o->par, o->err,
                        o->c2);
  else
    barrel_step_fwd_nomat(x->par, x->err, x->m, x->me, x->ta, x->tb, x->tc, x->k, mat, o->par,
                          o->err, o->c2);
}
template <bool kMat>
__device__ __noinline__ void step_rev_plain(const StepIn* x, MatGrid mat, float g, StepBars* b) {
  StepBars o;
  if (kMat)
    barrel_step_rev_mat(x->par, x->err, x->m, x->me, x->ta, x->tb, x->tc, x->k, mat, b->par, b->err,
                        g, o.par, o.err, o.ga, o.gb, o.gc);
  else
    barrel_step_rev_nomat(x->par, x->err, x->m, x->me, x->ta, x->tb, x->tc, x->k, mat, b->par,
                          b->err, g, o.par, o.err, o.ga, o.gb, o.gc);
  *b = o;
}
__device__ __forceinline__ StepIn step_in(const float (&par)[6], const float (&err)[21],
                                          const float (&m)[3], const float (&me)[6], float ta,
                                          float tb, float tc, float k) {
  StepIn x;
#pragma unroll
  for (int e = 0; e < 6; ++e) x.par[e] = par[e];
#pragma unroll
  for (int e = 0; e < 21; ++e) x.err[e] = err[e];
#pragma unroll
  for (int e = 0; e < 3; ++e) x.m[e] = m[e];
#pragma unroll
  for (int e = 0; e < 6; ++e) x.me[e] = me[e];
  x.ta = ta;
  x.tb = tb;
  x.tc = tc;
  x.k = k;
  return x;
}

template <bool kMat>
__device__ __forceinline__ void step_fwd(const float (&par)[6], const float (&err)[21],
                                         const float (&m)[3], const float (&me)[6], float ta, float tb,
                                         float tc, float k, const MatGrid& grid, float (&opar)[6],
                                         float (&oerr)[21], float& c2) {
  const FlatGrid mat(grid);
  if (kMat)
    barrel_step_fwd_mat(par, err, m, me, ta, tb, tc, k, mat, opar, oerr, c2);
  else
    barrel_step_fwd_nomat(par, err, m, me, ta, tb, tc, k, mat, opar, oerr, c2);
  ad_see_all(mat, opar);
  ad_see_all(mat, oerr);
  ad_see_top(mat, c2);
  if (mat.ok()) return;
  const StepIn x = step_in(par, err, m, me, ta, tb, tc, k);
  StepState o;
  step_fwd_plain<kMat>(&x, grid, &o);
#pragma unroll
  for (int e = 0; e < 6; ++e) opar[e] = o.par[e];
#pragma unroll
  for (int e = 0; e < 21; ++e) oerr[e] = o.err[e];
  c2 = o.c2;
}

template <bool kMat>
__device__ __forceinline__ void step_rev(const float (&par)[6], const float (&err)[21],
                                         const float (&m)[3], const float (&me)[6], float ta, float tb,
                                         float tc, float k, const MatGrid& grid,
                                         const float (&par_bar)[6], const float (&err_bar)[21], float g,
                                         float (&pb)[6], float (&eb)[21], float& ga, float& gb,
                                         float& gc) {
  const FlatGrid mat(grid);
  if (kMat)
    barrel_step_rev_mat(par, err, m, me, ta, tb, tc, k, mat, par_bar, err_bar, g, pb, eb, ga, gb, gc);
  else
    barrel_step_rev_nomat(par, err, m, me, ta, tb, tc, k, mat, par_bar, err_bar, g, pb, eb, ga, gb, gc);
  ad_see_all(mat, pb);
  ad_see_all(mat, eb);
  ad_see_top(mat, ga);
  ad_see_top(mat, gb);
  ad_see_top(mat, gc);
  if (mat.ok()) return;
  const StepIn x = step_in(par, err, m, me, ta, tb, tc, k);
  StepBars o;
#pragma unroll
  for (int e = 0; e < 6; ++e) o.par[e] = par_bar[e];
#pragma unroll
  for (int e = 0; e < 21; ++e) o.err[e] = err_bar[e];
  step_rev_plain<kMat>(&x, grid, g, &o);
#pragma unroll
  for (int e = 0; e < 6; ++e) pb[e] = o.par[e];
#pragma unroll
  for (int e = 0; e < 21; ++e) eb[e] = o.err[e];
  ga = o.ga;
  gb = o.gb;
  gc = o.gc;
}

}  // namespace adj
}  // namespace mkfg
