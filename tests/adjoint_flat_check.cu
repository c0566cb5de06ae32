// One step of the differentiable fit and its reverse: the form with the
// branch-free arithmetic (csrc/adjoint_flat.cuh) beside the plain one, from
// given states; built and loaded by test_flat_math_gpu.py.
#include "../mkfit_b200/csrc/adjoint_flat.cuh"

using namespace mkfg;

// in[38][n]: parameters 6, covariance 21, hit 3 + 6, gradient of chi2, charge
// (as a number); bars[27][n]; out[2][58][n]: 6 + 21 + chi2, then the 27 bars
// and three alignment gradients, flat and plain.
__global__ void __launch_bounds__(128) k_adj(int n, const float* in, const float* bars,
                                             adj::MatGrid grid, float* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float par[6], err[21], m[3], me[6], pbar[6], ebar[21];
  for (int k = 0; k < 6; ++k) par[k] = in[k * n + i];
  for (int k = 0; k < 21; ++k) err[k] = in[(6 + k) * n + i];
  for (int k = 0; k < 3; ++k) m[k] = in[(27 + k) * n + i];
  for (int k = 0; k < 6; ++k) me[k] = in[(30 + k) * n + i];
  for (int k = 0; k < 6; ++k) pbar[k] = bars[k * n + i];
  for (int k = 0; k < 21; ++k) ebar[k] = bars[(6 + k) * n + i];
  const float g = in[36 * n + i], kk = in[37 * n + i] * 100.f / (-kSol * kBfield);
  const adj::StepIn x = adj::step_in(par, err, m, me, 0.f, 0.f, 1.f, kk);
  for (int form = 0; form < 2; ++form) {
    adj::StepState o;
    adj::StepBars b;
    if (form == 0) {
      adj::step_fwd<true>(par, err, m, me, 0.f, 0.f, 1.f, kk, grid, o.par, o.err, o.c2);
      adj::step_rev<true>(par, err, m, me, 0.f, 0.f, 1.f, kk, grid, pbar, ebar, g, b.par, b.err,
                                b.ga, b.gb, b.gc);
    } else {
      adj::step_fwd_plain<true>(&x, grid, &o);
      for (int k = 0; k < 6; ++k) b.par[k] = pbar[k];
      for (int k = 0; k < 21; ++k) b.err[k] = ebar[k];
      adj::step_rev_plain<true>(&x, grid, g, &b);
    }
    float* w = out + (size_t)form * 58 * n + i;
    for (int k = 0; k < 6; ++k) w[k * n] = o.par[k];
    for (int k = 0; k < 21; ++k) w[(6 + k) * n] = o.err[k];
    w[27 * n] = o.c2;
    for (int k = 0; k < 6; ++k) w[(28 + k) * n] = b.par[k];
    for (int k = 0; k < 21; ++k) w[(34 + k) * n] = b.err[k];
    w[55 * n] = b.ga;
    w[56 * n] = b.gb;
    w[57 * n] = b.gc;
  }
}
extern "C" int adjoint_flat_step(int n, const float* in, const float* bars, const float* rl,
                                 const float* xi, float* out) {
  k_adj<<<(n + 127) / 128, 128>>>(n, in, bars, adj::MatGrid{rl, xi}, out);
  return (int)cudaDeviceSynchronize();
}
