// Compares the branch-free arithmetic of csrc/flat_math.cuh, and the steps of
// the fit that use it, with the plain ones on the device; built and loaded by
// test_flat_math_gpu.py.
#include "../mkfit_b200/csrc/kalman.cuh"

using namespace mkfg;

enum { kRcp, kDiv, kSqrt, kSin, kCos, kLog, kHypot, kInvDet };

// counts[0]: values that differ, counts[1]: largest difference in ulps.
__global__ void k_check(int what, long long n, const float* a, const float* b, unsigned* counts) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    // Without inputs: every mantissa, in two exponents.
    const float x = a ? a[i] : __int_as_float(0x3f800000 + (int)i);
    const float y = b ? b[i] : 1.f;
    float got = 0.f, want = 0.f, s, c;
    FlatMath m;
    switch (what) {
      case kRcp: got = FlatMath::rcp(x); want = 1.f / x; break;
      case kDiv: got = FlatMath::div(x, y); want = x / y; break;
      case kSqrt: got = FlatMath::sqrt(x); want = sqrtf(x); break;
      case kSin: m.sincos(x, &s, &c); got = s; want = f_sin(x); break;
      case kCos: m.sincos(x, &s, &c); got = c; want = f_cos(x); break;
      case kLog: got = m.log(x); want = f_log(x); break;
      case kHypot: got = m.hypot(x, y); want = hypot_f(x, y); break;
      case kInvDet: {
        const double d = (double)x * y;
        got = m.inv_det(d);
        want = (float)(1.0 / d);
        break;
      }
    }
    if (!m.ok()) atomicOr(counts + 2, 1u);
    if (got != want) {
      atomicAdd(counts, 1u);
      atomicMax(counts + 1, (unsigned)abs(__float_as_int(got) - __float_as_int(want)));
    }
  }
}

extern "C" int flat_math_check(int what, long long n, const float* a, const float* b,
                               unsigned* counts) {
  k_check<<<1024, 256>>>(what, n, a, b, counts);
  return (int)cudaDeviceSynchronize();
}

// The range bookkeeping: ok() after seeing the given operands.
__global__ void k_seen(int n, const float* v, int wide, int* ok) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  FlatMath m;
  if (wide) m.see_wide(v[i]);
  else m.see(v[i]);
  m.see(1.f);
  ok[i] = m.ok();
}
extern "C" int flat_math_seen(int n, const float* v, int wide, int* ok) {
  k_seen<<<(n + 127) / 128, 128>>>(n, v, wide, ok);
  return (int)cudaDeviceSynchronize();
}

// A propagation (barrel: to the hit's radius, else to its z) and an update of
// the given state, flat and plain: out[2][55][n] (6 + 21 propagated, 6 + 21
// updated, chi2), back[2][n]: whether the flat form would use the plain one.
struct StepArgs {
  int n, barrel;
  unsigned pflags;
  Material mat;
  const float *par, *err, *hpos, *herr;
  const int* chg;
  float* out;
  int* back;
};
template <bool kBarrel>
__device__ void step_check(const StepArgs& a, int i) {
  float p[6], e[21], m[3], v[6];
  for (int k = 0; k < 6; ++k) p[k] = a.par[k * a.n + i];
  for (int k = 0; k < 21; ++k) e[k] = a.err[k * a.n + i];
  for (int k = 0; k < 3; ++k) m[k] = a.hpos[k * a.n + i];
  for (int k = 0; k < 6; ++k) v[k] = a.herr[k * a.n + i];
  const int chg = a.chg[i];
  const float r = hypot_f(m[0], m[1]);
  for (int form = 0; form < 2; ++form) {
    float pp[6], pe[21], up[6], ue[21], chi2;
    if (form == 0) {
      if (kBarrel) propagate_to_r_flat(p, e, chg, r, a.pflags, a.mat, false, pp, pe);
      else propagate_to_z_flat(p, e, chg, m[2], a.pflags, a.mat, false, pp, pe);
    } else {
      if (kBarrel) propagate_to_r(p, e, chg, r, a.pflags, a.mat, false, pp, pe);
      else propagate_to_z(p, e, chg, m[2], a.pflags, a.mat, false, pp, pe);
    }
    // The update from the given state, which may lie anywhere.
    if (form == 0)
      chi2 = update_flat<true, kBarrel>(p, e, m, v, up, ue);
    else
      chi2 = kBarrel ? kalman_barrel<true, true>(p, e, m, v, up, ue)
                     : kalman_endcap<true, true>(p, e, m, v, up, ue);
    float* o = a.out + (size_t)form * 55 * a.n + i;
    for (int k = 0; k < 6; ++k) o[k * a.n] = pp[k];
    for (int k = 0; k < 21; ++k) o[(6 + k) * a.n] = pe[k];
    for (int k = 0; k < 6; ++k) o[(27 + k) * a.n] = up[k];
    for (int k = 0; k < 21; ++k) o[(33 + k) * a.n] = ue[k];
    o[54 * a.n] = chi2;
  }
  FlatMath fp, fu;
  float pp[6], pe[21];
  if (kBarrel) {
    propagate_to_r_in(fp, p, e, chg, r, a.pflags, a.mat, false, pp, pe);
    kalman_barrel_in<true, true>(fu, p, e, m, v, pp, pe);
  } else {
    propagate_to_z_in(fp, p, e, chg, m[2], a.pflags, a.mat, false, pp, pe);
    kalman_endcap_in<true, true>(fu, p, e, m, v, pp, pe);
  }
  a.back[i] = !fp.ok();
  a.back[a.n + i] = !fu.ok();
}
__global__ void __launch_bounds__(128) k_step(const StepArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  if (a.barrel) step_check<true>(a, i);
  else step_check<false>(a, i);
}
extern "C" int flat_math_step(int n, int barrel, unsigned pflags, const float* rl, const float* xi,
                              const float* par, const float* err, const int* chg, const float* hpos,
                              const float* herr, float* out, int* back) {
  const StepArgs a{n, barrel, pflags, Material{rl, xi}, par, err, hpos, herr, chg, out, back};
  k_step<<<(n + 127) / 128, 128>>>(a);
  return (int)cudaDeviceSynchronize();
}
