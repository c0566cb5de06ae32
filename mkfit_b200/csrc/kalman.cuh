// Device-side Kalman-filter math for one track per CUDA thread.
//
// Semantics follow the reference CPU Matriplex path (trackreco/mkFit); each
// function names the reference routine it restates. All state lives in
// registers: parameters (x, y, z, 1/pT, phi, theta) in CCS coordinates, the
// 6x6 covariance as 21 floats (packed lower triangle, same element order as
// the reference's MatriplexSym), 6x6 Jacobians as 36-float arrays whose
// known-zero entries are folded away by the generated products.
//
// Every sum of products says which product is fused (fmaf) and which is
// rounded, and the fit's, the operator calls' and the finding's sources are
// compiled without the compiler's own contraction (build.py), so all their
// kernels give the same bits. The choice is the one the compiler had made in
// the finding's launch sequence.
#pragma once

#include <cuda_runtime.h>
#include <math_constants.h>

#include "flat_math.cuh"
#include "generated_ops.cuh"

namespace mkfg {

// Physics / math constants (Config.h:77-88, 240-245 of the reference).
constexpr float kPI = 3.14159265358979323846f;
constexpr float kTwoPI = 6.28318530717958647692f;
constexpr float kPIOver2 = kPI / 2.0f;
constexpr float kInvPI = 1.0f / kPI;
constexpr float kSol = 0.299792458f;
constexpr float kBfield = 3.8112f;
constexpr float kMagC1 = 3.8114f;
constexpr float kMagB0 = -3.94991e-06f;
constexpr float kMagB1 = 7.53701e-06f;
constexpr float kMagA = 2.43878e-11f;
constexpr int kNiter = 5;  // Config::Niter

// Material grid (Config.h:123-127): 300 z bins x 120 r bins over 300 x 120 cm.
constexpr int kMatNZ = 300;
constexpr int kMatNR = 120;
constexpr float kMatRangeZ = 300.f;
constexpr float kMatRangeR = 120.f;

// Propagation flag bits (Config.h:17-23).
constexpr unsigned kPfParamB = 0x1;
constexpr unsigned kPfMaterial = 0x2;

struct Material {
  const float* rl;  // [kMatNZ][kMatNR] radiation lengths
  const float* xi;  // [kMatNZ][kMatNR] energy-loss xi
};

__device__ __forceinline__ float sqr(float x) { return x * x; }

// Packed lower-triangle index of symmetric element (i, j).
__host__ __device__ constexpr int sidx(int i, int j) {
  return i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i;
}

// Elementary functions. The reference calls the host C library's float
// functions (sinf, cosf, logf, atan2f), which are correctly rounded for
// nearly all arguments. With MKFG_LIBM_EXACT (default) the device evaluates
// them in double precision and rounds once to float, which reproduces those
// results except in rare double-rounding cases; without it the CUDA float
// versions (<= 2 ulp) are used.
#ifndef MKFG_LIBM_EXACT
#define MKFG_LIBM_EXACT 1
#endif
__device__ __forceinline__ void f_sincos(float x, float* s, float* c) {
#if MKFG_LIBM_EXACT
  double sd, cd;
  sincos((double)x, &sd, &cd);
  *s = (float)sd;
  *c = (float)cd;
#else
  sincosf(x, s, c);
#endif
}
__device__ __forceinline__ float f_sin(float x) {
#if MKFG_LIBM_EXACT
  return (float)sin((double)x);
#else
  return sinf(x);
#endif
}
__device__ __forceinline__ float f_cos(float x) {
#if MKFG_LIBM_EXACT
  return (float)cos((double)x);
#else
  return cosf(x);
#endif
}
__device__ __forceinline__ float f_log(float x) {
#if MKFG_LIBM_EXACT
  return (float)log((double)x);
#else
  return logf(x);
#endif
}
__device__ __forceinline__ float f_atan2(float y, float x) {
#if MKFG_LIBM_EXACT
  return (float)atan2((double)y, (double)x);
#else
  return atan2f(y, x);
#endif
}

// sqrt(x*x + y*y) in float, as the reference's hipo() (Matrix.h:38).
__device__ __forceinline__ float hipo(float x, float y) { return sqrtf(fmaf(x, x, y * y)); }

// std::hypot(float, float) as evaluated by glibc: the sum of squares is
// formed in double precision and the root is rounded once to float.
__device__ __forceinline__ float hypot_f(float x, float y) {
  const double dx = x, dy = y;
  return (float)sqrt(fma(dx, dx, dy * dy));
}

// The plain form of the step's arithmetic (flat_math.cuh).
struct ExactMath {
  static constexpr bool kPlain = true;
  __device__ __forceinline__ void see(float) {}
  __device__ __forceinline__ void see_wide(float) {}
  __device__ __forceinline__ void see_top(float) {}
  __device__ __forceinline__ bool ok() const { return true; }
  __device__ __forceinline__ static float rcp(float b) { return 1.f / b; }
  __device__ __forceinline__ static float div(float a, float b) { return a / b; }
  __device__ __forceinline__ static float div_const(float a, float b, float) { return a / b; }
  __device__ __forceinline__ static float sqrt(float x) { return sqrtf(x); }
  __device__ __forceinline__ static void sincos(float x, float* s, float* c) { f_sincos(x, s, c); }
  __device__ __forceinline__ static float log(float x) { return f_log(x); }
  __device__ __forceinline__ static float hypot(float x, float y) { return hypot_f(x, y); }
  __device__ __forceinline__ static float inv_det(double det) { return (float)(1.0 / det); }
};

// Magnetic field model (Config.h:434-437).
__device__ __forceinline__ float bfield_zr(float z, float r) {
  return (fmaf(kMagB0 * z, z, kMagB1 * z) + kMagC1) * fmaf(kMagA * r, r, 1.f);
}

// Fourth-order sin/cos polynomial of the reference (Matrix.h:48-56).
__device__ __forceinline__ void sincos4(float x, float& s, float& c) {
  const float x2 = x * x;
  c = fmaf(0.04166667f * x2, x2, fmaf(-0.5f, x2, 1.f));
  s = fmaf(-0.16666667f * x, x2, x);
}

// phi into [-pi, pi) (squashPhiMPlex, mkFit/PropagationMPlex.h:8-15).
__device__ __forceinline__ float squash_phi(float phi) {
  if (phi >= kPI) phi -= kTwoPI;
  if (phi < -kPI) phi += kTwoPI;
  return phi;
}

//------------------------------------------------------------------------------
// Helix to radius r: 5 fixed iterations with arc-length derivative tracking.
// Restates helixAtRFromIterativeCCS_impl (mkFit/PropagationMPlex.icc:5-246).
// Returns the fail flag (1 when the step would approach the apex), and the
// sine of theta for the material effects.
//------------------------------------------------------------------------------
// k = charge * 100 / (-sol * B) of a unit charge in the constant field.
constexpr float kCurv1 = 100.f / (-kSol * kBfield);
constexpr float kCurvInv1 = 1.f / kCurv1;

// The curvature constant k and its inverse.
template <class F>
__device__ __forceinline__ void curvature(F& m, int chg, bool param_b, float z, float r, float& k,
                                          float& kinv) {
  if (!param_b && (chg == 1 || chg == -1)) {
    k = chg > 0 ? kCurv1 : -kCurv1;
    kinv = chg > 0 ? kCurvInv1 : -kCurvInv1;
    return;
  }
  const float bf = param_b ? bfield_zr(z, r) : kBfield;
  const float d = -kSol * bf;
  m.see(d);
  k = F::div(float(chg) * 100.f, d);
  m.see(k);
  kinv = F::rcp(k);
}

// kResidual: the 1/pT derivative of z takes ipt * dadipt - alpha, which nearly
// cancels, from the exact product (the fits) or from the rounded one (the
// finding and its operator calls).
template <bool kResidual = true, class F>
__device__ __forceinline__ int helix_to_r(F& m, const float (&in)[6], int chg, float r, bool param_b,
                                          float (&out)[6], float (&J)[36], float& sinT) {
#pragma unroll
  for (int i = 0; i < 36; ++i) J[i] = 0.f;
  int fail = 0;

  float r02 = fmaf(in[0], in[0], in[1] * in[1]);
  m.see(r02);
  float r0 = F::sqrt(r02);
  float k, kinv;
  curvature(m, chg, param_b, in[2], r0, k, kinv);

  const float xin = in[0], yin = in[1], ipt = in[3], phiin = in[4], theta = in[5];
  m.see(ipt);
  const float pt = F::rcp(ipt);

  float D = 0.f, cosa = 0.f, sina = 0.f, cosah = 0.f, sinah = 0.f, id = 0.f;
  float cosPorT, sinPorT;
  m.sincos(phiin, &sinPorT, &cosPorT);
  float pxin = cosPorT * pt;
  float pyin = sinPorT * pt;

  float dDdx = r0 > 0.f ? F::div(-xin, r0) : 0.f;
  float dDdy = r0 > 0.f ? F::div(-yin, r0) : 0.f;
  float dDdipt = 0.f;
  float dDdphi = 0.f;

  float ox = in[0], oy = in[1];
#pragma unroll
  for (int it = 0; it < kNiter; ++it) {
    if (it > 0) {
      r02 = fmaf(ox, ox, oy * oy);
      m.see(r02);
      r0 = F::sqrt(r02);
    }
    const float dot = fmaf(pxin, ox, pyin * oy);
    m.see(dot);
    const float oodotp = F::div(r0 * pt, dot);
    if (oodotp > 5.0f || oodotp < 0) {
      id = 0.0f;
      fail = 1;
    } else {
      id = (r - r0) * oodotp;
    }
    D += id;

    sincos4(id * ipt * kinv * 0.5f, sinah, cosah);
    cosa = fmaf(-2.f * sinah, sinah, 1.f);
    sina = 2.f * sinah * cosah;
    // The direction after the step.
    const float pxca = pxin * cosa, pxsa = pxin * sina;
    const float pyca = pyin * cosa, pysa = pyin * sina;
    const float pxnew = pxca - pysa, pynew = pyca + pxsa;

    // Far from the target radius (the first steps) the factor 1 / r0 of
    // every derivative term is 0: FlatMath, whose numbers are finite, skips
    // them there.
    const bool near_r = r0 > 0.f && fabsf(r - r0) < 0.0001f;
    if (it + 1 != kNiter && (F::kPlain || near_r)) {
      const float x = ox, y = oy;
      const float oor0 = near_r ? F::rcp(r0) : 0.f;
      const float dadipt = id * kinv;
      const float dadx = -x * ipt * kinv * oor0;
      const float dady = -y * ipt * kinv * oor0;
      float tmp = k * dadx;
      dDdx = fmaf(-fmaf(y * tmp, pynew, x * fmaf(tmp, pxnew, 1.f)), oor0, dDdx);
      tmp = k * dady;
      dDdy = fmaf(-fmaf(x * tmp, pxnew, y * fmaf(tmp, pynew, 1.f)), oor0, dDdy);
      tmp = dadipt * ipt;
      const float a = fmaf(-pxin, sina, fmaf(-pyin, cosa, fmaf(pxca, tmp, -(pysa * tmp)))) + pyin;
      const float b = fmaf(pxin, cosa, fmaf(-pyin, sina, fmaf(pyca, tmp, pxsa * tmp))) - pxin;
      dDdipt = fmaf(-(k * fmaf(x, a, y * b) * pt), oor0, dDdipt);
      const float u = fmaf(pxin, cosa, fmaf(pyin, sina, -pxin));
      const float v = fmaf(pyin, cosa, fmaf(pxin, sina, -pyin));
      dDdphi = fmaf(k * fmaf(x, u, -(y * v)), oor0, dDdphi);
    }

    ox = fmaf(2.f * k * sinah, fmaf(pxin, cosah, -(pyin * sinah)), ox);
    oy = fmaf(2.f * k * sinah, fmaf(pxin, sinah, pyin * cosah), oy);
    pxin = pxnew;
    pyin = pynew;
  }

  const float alpha = D * ipt * kinv;
  const float dadx = dDdx * ipt * kinv;
  const float dady = dDdy * ipt * kinv;
  const float dadipt = fmaf(ipt, dDdipt, D) * kinv;
  const float dadphi = dDdphi * ipt * kinv;

  sincos4(alpha, sina, cosa);

  // Sine and cosine of the direction's azimuth at the end, and the 1/pT terms.
  const float ca = fmaf(cosPorT, cosa, -(sinPorT * sina));
  const float sa = fmaf(cosPorT, sina, sinPorT * cosa);
  const float w = ipt * dadipt;
  const float wc = fmaf(w, cosa, -sina), ws = fmaf(w, sina, -(1.f - cosa));

  J[0 * 6 + 0] = fmaf(k * dadx * ca, pt, 1.f);
  J[0 * 6 + 1] = k * dady * ca * pt;
  J[0 * 6 + 3] = k * fmaf(cosPorT, wc, sinPorT * -ws) * pt * pt;
  J[0 * 6 + 4] = k * (fmaf(cosPorT, cosa, fmaf(cosPorT * dadphi, cosa, -(sinPorT * dadphi * sina)) - sinPorT * sina) - cosPorT) * pt;

  J[1 * 6 + 0] = k * dadx * sa * pt;
  J[1 * 6 + 1] = fmaf(k * dady * sa, pt, 1.f);
  J[1 * 6 + 3] = k * fmaf(sinPorT, wc, cosPorT * ws) * pt * pt;
  J[1 * 6 + 4] = k * (fmaf(cosPorT, sina, fmaf(sinPorT, cosa, fmaf(sinPorT * dadphi, cosa, cosPorT * dadphi * sina))) - sinPorT) * pt;

  float cosT;
  m.sincos(theta, &sinT, &cosT);
  m.see(sinT);
  const float isinT = F::rcp(sinT);

  out[0] = ox;
  out[1] = oy;
  out[2] = fmaf(k * alpha * cosT * pt, isinT, in[2]);
  out[3] = ipt;
  out[4] = in[4] + alpha;
  out[5] = theta;

  J[2 * 6 + 0] = k * cosT * dadx * pt * isinT;
  J[2 * 6 + 1] = k * cosT * dady * pt * isinT;
  J[2 * 6 + 2] = 1.f;
  const float dalpha = kResidual ? fmaf(ipt, dadipt, -alpha) : w - alpha;
  J[2 * 6 + 3] = k * cosT * dalpha * pt * pt * isinT;
  J[2 * 6 + 4] = k * dadphi * cosT * pt * isinT;
  J[2 * 6 + 5] = -k * alpha * pt * isinT * isinT;

  J[3 * 6 + 3] = 1.f;

  J[4 * 6 + 0] = dadx;
  J[4 * 6 + 1] = dady;
  J[4 * 6 + 3] = dadipt;
  J[4 * 6 + 4] = fmaf(dDdphi * ipt, kinv, 1.f);

  J[5 * 6 + 5] = 1.f;
  return fail;
}

//------------------------------------------------------------------------------
// Helix to plane z (endcap). Restates helixAtZ (mkFit/PropagationMPlex.cc:604-712).
//------------------------------------------------------------------------------
template <class F>
__device__ __forceinline__ void helix_to_z(F& m, const float (&in)[6], int chg, float zout,
                                           bool param_b, float (&out)[6], float (&J)[36],
                                           float& sinT, float& cosT) {
#pragma unroll
  for (int i = 0; i < 36; ++i) J[i] = 0.f;
  J[0 * 6 + 0] = 1.f;
  J[1 * 6 + 1] = 1.f;
  J[3 * 6 + 3] = 1.f;
  J[4 * 6 + 4] = 1.f;
  J[5 * 6 + 5] = 1.f;

  const float zin = in[2], ipt = in[3], phiin = in[4], theta = in[5];
  float k, kinv;
  curvature(m, chg, param_b, zin, param_b ? hipo(in[0], in[1]) : 0.f, k, kinv);
  m.see(ipt);
  const float pt = F::rcp(ipt);

  float cosP, sinP;
  m.sincos(phiin, &sinP, &cosP);
  m.sincos(theta, &sinT, &cosT);
  m.see(cosT);
  const float tanT = F::div(sinT, cosT);
  const float icos2T = F::rcp(cosT * cosT);
  const float pxin = cosP * pt;
  const float pyin = sinP * pt;

  const float deltaZ = zout - zin;
  const float alpha = deltaZ * tanT * ipt * kinv;

  float sinah, cosah;
  sincos4(alpha * 0.5f, sinah, cosah);
  const float cosa = fmaf(-2.f * sinah, sinah, 1.f);
  const float sina = 2.f * sinah * cosah;

  out[0] = fmaf(2.f * k * sinah, fmaf(pxin, cosah, -(pyin * sinah)), in[0]);
  out[1] = fmaf(2.f * k * sinah, fmaf(pxin, sinah, pyin * cosah), in[1]);
  out[2] = zout;
  out[3] = in[3];
  out[4] = phiin + alpha;
  out[5] = in[5];

  const float ac = fmaf(alpha, cosa, -sina), as = fmaf(-alpha, cosah, sinah);
  const float pxcaMpysa = fmaf(pxin, cosa, -(pyin * sina));
  J[0 * 6 + 2] = -tanT * ipt * pxcaMpysa;
  J[0 * 6 + 3] = k * pt * pt * fmaf(sinP * 2.f * sinah, as, cosP * ac);
  J[0 * 6 + 4] = -2 * k * pt * sinah * fmaf(cosP, sinah, sinP * cosah);
  J[0 * 6 + 5] = deltaZ * ipt * pxcaMpysa * icos2T;

  const float pycaPpxsa = fmaf(pxin, sina, pyin * cosa);
  J[1 * 6 + 2] = -tanT * ipt * pycaPpxsa;
  J[1 * 6 + 3] = k * pt * pt * fmaf(sinP, ac, -(cosP * 2.f * sinah * as));
  J[1 * 6 + 4] = 2 * k * pt * sinah * fmaf(cosP, cosah, -(sinP * sinah));
  J[1 * 6 + 5] = deltaZ * ipt * pycaPpxsa * icos2T;

  J[4 * 6 + 2] = -ipt * tanT * kinv;
  J[4 * 6 + 3] = tanT * deltaZ * kinv;
  J[4 * 6 + 5] = ipt * deltaZ * kinv * icos2T;
}

//------------------------------------------------------------------------------
// Multiple scattering + energy loss. Restates applyMaterialEffects
// (mkFit/PropagationMPlex.cc:716-767): updates C[3][3], C[4][4], C[5][5] of
// the (pre-similarity) covariance and 1/pT of the propagated parameters.
//------------------------------------------------------------------------------
// sinT, cosT: of par[5] (cosT read in the endcaps only). The operands of the
// divisions and roots are bounded by 1/pT and sinT (cosT), which are seen
// here again.
template <class F>
__device__ __forceinline__ void material_effects(F& m, float radL, float xi, float prop_sign,
                                                 bool is_barrel, float sinT, float cosT,
                                                 float (&C)[21], float (&par)[6]) {
  if (radL < 1e-13f) return;
  m.see(par[3]);
  m.see(sinT);
  const float pt = F::rcp(par[3]);
  const float p = F::div(pt, sinT);
  const float p2 = p * p;
  constexpr float mpi = 0.140f;
  constexpr float mpi2 = mpi * mpi;
  const float beta2 = F::div(p2, p2 + mpi2);
  const float beta = F::sqrt(beta2);
  const float invCos = is_barrel ? F::div(p, pt) : F::rcp(fabsf(cosT));
  radL = radL * invCos;
  if (radL < 1e-13f) return;
  const float thetaMSC = F::div(0.0136f * fmaf(0.038f, m.log(radL), 1.f), beta * p);
  C[14] = fmaf(thetaMSC * thetaMSC, radL, C[14]);  // (4,4)
  C[20] = fmaf(thetaMSC * thetaMSC, radL, C[20]);  // (5,5)
  constexpr float impi2 = 1.f / mpi2, impi = 1.f / mpi;
  const float gamma2 = F::div_const(p2 + mpi2, mpi2, impi2);
  const float gamma = F::sqrt(gamma2);
  constexpr float me = 0.0005f;
  const float wmax = F::div(2.f * me * beta2 * gamma2,
                            1.f + F::div_const(2.f * gamma * me, mpi, impi) + me * me / (mpi * mpi));
  constexpr float I = (float)(16.0e-9 * 10.75);
  constexpr float I2 = I * I, iI2 = 1.f / I2;
  // log(28.816e-9 sqrt(2.33 * 0.498) / I), each step rounded to float.
  constexpr float log_plasma = -1.7122072f;
  const float deltahalf = log_plasma + m.log(beta * gamma) - 0.5f;
  const float log_w = m.log(F::div_const(2.f * me * beta2 * gamma2 * wmax, I2, iI2));
  const float dEdx =
      beta < 1.f ? (2.f * (F::div(xi * invCos * (fmaf(0.5f, log_w, -beta2) - deltahalf), beta2))) : 0.f;
  const float dP = F::div(prop_sign * dEdx, beta);
  m.see_top(dP);
  par[3] = F::div(p, fmaxf(p + dP, 0.001f) * pt);
  C[9] += F::div(dP * dP, p2 * pt * pt);  // (3,3)
}

// Material grid lookup with the reference's bin arithmetic and range guard
// (MaterialEffects.h:8-11, mkFit/PropagationMPlex.cc:455-460).
__device__ __forceinline__ void material_lookup(const Material& m, float z, float r, float& rl, float& xi) {
  const int zb = (int)((fabsf(z) * kMatNZ) / kMatRangeZ);
  const int rb = (int)((r * kMatNR) / kMatRangeR);
  if (zb >= 0 && zb < kMatNZ && rb >= 0 && rb < kMatNR) {
    rl = __ldg(m.rl + zb * kMatNR + rb);
    xi = __ldg(m.xi + zb * kMatNR + rb);
  } else {
    rl = 0.f;
    xi = 0.f;
  }
}

//------------------------------------------------------------------------------
// Full propagation to radius r with material and covariance transport.
// Restates propagateHelixToRMPlex (mkFit/PropagationMPlex.cc:408-505).
// On failure the output is reset to the input (fix-up at :497-504).
//------------------------------------------------------------------------------
template <bool kResidual = true, class F>
__device__ __forceinline__ int propagate_to_r_in(F& m, const float (&par)[6], const float (&err)[21],
                                                 int chg, float r, unsigned pflags,
                                                 const Material& mat, bool no_mat_eff,
                                                 float (&opar)[6], float (&oerr)[21]) {
  float J[36];
  float p[6];
  float sinT;
  const int fail = helix_to_r<kResidual>(m, par, chg, r, pflags & kPfParamB, p, J, sinT);
  float C[21];
#pragma unroll
  for (int i = 0; i < 21; ++i) C[i] = err[i];
  if (pflags & kPfMaterial) {
    float rl = 0.f, xi = 0.f;
    if (!(fail || no_mat_eff)) material_lookup(mat, p[2], r, rl, xi);
    const float r0 = F::sqrt(fmaf(par[0], par[0], par[1] * par[1]));
    const float sign = (r > r0 ? 1.f : -1.f);
    material_effects(m, rl, xi, sign, true, sinT, 1.f, C, p);
  }
  p[4] = squash_phi(p[4]);
  float Co[21];
  similarity_barrel(J, C, Co);
  if (fail) {
#pragma unroll
    for (int i = 0; i < 6; ++i) opar[i] = par[i];
#pragma unroll
    for (int i = 0; i < 21; ++i) oerr[i] = err[i];
  } else {
#pragma unroll
    for (int i = 0; i < 6; ++i) opar[i] = p[i];
#pragma unroll
    for (int i = 0; i < 21; ++i) oerr[i] = Co[i];
  }
  return fail;
}

// Propagation to plane z. Restates propagateHelixToZMPlex
// (mkFit/PropagationMPlex.cc:510-601); this path has no fail flag.
template <class F>
__device__ __forceinline__ void propagate_to_z_in(F& m, const float (&par)[6], const float (&err)[21],
                                                  int chg, float z, unsigned pflags,
                                                  const Material& mat, bool no_mat_eff,
                                                  float (&opar)[6], float (&oerr)[21]) {
  float J[36];
  float p[6];
  float sinT, cosT;
  helix_to_z(m, par, chg, z, pflags & kPfParamB, p, J, sinT, cosT);
  float C[21];
#pragma unroll
  for (int i = 0; i < 21; ++i) C[i] = err[i];
  if (pflags & kPfMaterial) {
    float rl = 0.f, xi = 0.f;
    if (!no_mat_eff) material_lookup(mat, z, m.hypot(p[0], p[1]), rl, xi);
    const float sign = (fabsf(z) > fabsf(par[2]) ? 1.f : -1.f);
    material_effects(m, rl, xi, sign, false, sinT, cosT, C, p);
  }
  p[4] = squash_phi(p[4]);
  similarity_endcap(J, C, oerr);
#pragma unroll
  for (int i = 0; i < 6; ++i) opar[i] = p[i];
}

// The steps repeated with ExactMath where FlatMath's operands left their
// range (rare: a track at the beam line, 1/pT near zero, an overflow). Not
// inlined, on copies, so the usual path keeps its arrays in registers.
struct StateCopy {
  float par[6], err[21];
};
static __device__ __noinline__ int propagate_exact(StateCopy* s, bool to_r, int chg, float at,
                                            unsigned pflags, Material mat, bool no_mat_eff) {
  ExactMath m;
  float par[6], err[21];
  int fail = 0;
  if (to_r)
    fail = propagate_to_r_in(m, s->par, s->err, chg, at, pflags, mat, no_mat_eff, par, err);
  else
    propagate_to_z_in(m, s->par, s->err, chg, at, pflags, mat, no_mat_eff, par, err);
#pragma unroll
  for (int i = 0; i < 6; ++i) s->par[i] = par[i];
#pragma unroll
  for (int i = 0; i < 21; ++i) s->err[i] = err[i];
  return fail;
}

__device__ __forceinline__ int propagate_again(const float (&par)[6], const float (&err)[21], bool to_r,
                                               int chg, float at, unsigned pflags, const Material& mat,
                                               bool no_mat_eff, float (&opar)[6], float (&oerr)[21]) {
  StateCopy s;
#pragma unroll
  for (int i = 0; i < 6; ++i) s.par[i] = par[i];
#pragma unroll
  for (int i = 0; i < 21; ++i) s.err[i] = err[i];
  const int fail = propagate_exact(&s, to_r, chg, at, pflags, mat, no_mat_eff);
#pragma unroll
  for (int i = 0; i < 6; ++i) opar[i] = s.par[i];
#pragma unroll
  for (int i = 0; i < 21; ++i) oerr[i] = s.err[i];
  return fail;
}

// With ExactMath, and (the *_flat forms) with FlatMath. The fit uses the
// flat ones, the finding the plain ones: with FlatMath its propagation and
// update were 6 and 13% faster, but its chi2 6% slower, and the double
// functions' rare other rounding would turn near-ties of its decisions.
template <bool kResidual = true>
__device__ __forceinline__ int propagate_to_r(const float (&par)[6], const float (&err)[21], int chg,
                                              float r, unsigned pflags, const Material& mat,
                                              bool no_mat_eff, float (&opar)[6], float (&oerr)[21]) {
  ExactMath m;
  return propagate_to_r_in<kResidual>(m, par, err, chg, r, pflags, mat, no_mat_eff, opar, oerr);
}

__device__ __forceinline__ void propagate_to_z(const float (&par)[6], const float (&err)[21], int chg,
                                               float z, unsigned pflags, const Material& mat,
                                               bool no_mat_eff, float (&opar)[6], float (&oerr)[21]) {
  ExactMath m;
  propagate_to_z_in(m, par, err, chg, z, pflags, mat, no_mat_eff, opar, oerr);
}

__device__ __forceinline__ int propagate_to_r_flat(const float (&par)[6], const float (&err)[21],
                                                   int chg, float r, unsigned pflags,
                                                   const Material& mat, bool no_mat_eff,
                                                   float (&opar)[6], float (&oerr)[21]) {
  FlatMath m;
  int fail = propagate_to_r_in(m, par, err, chg, r, pflags, mat, no_mat_eff, opar, oerr);
  if (!m.ok())
    fail = propagate_again(par, err, true, chg, r, pflags, mat, no_mat_eff, opar, oerr);
  return fail;
}

__device__ __forceinline__ void propagate_to_z_flat(const float (&par)[6], const float (&err)[21],
                                                    int chg, float z, unsigned pflags,
                                                    const Material& mat, bool no_mat_eff,
                                                    float (&opar)[6], float (&oerr)[21]) {
  FlatMath m;
  propagate_to_z_in(m, par, err, chg, z, pflags, mat, no_mat_eff, opar, oerr);
  if (!m.ok()) propagate_again(par, err, false, chg, z, pflags, mat, no_mat_eff, opar, oerr);
}

//------------------------------------------------------------------------------
// 2x2 symmetric inverse with the determinant formed in double precision
// (CramerInverterSym<T,2,N>, Matriplex/MatriplexSym.h:422-445).
//------------------------------------------------------------------------------
template <class F>
__device__ __forceinline__ void invert_sym2(F& m, float& a0, float& a1, float& a2) {
  const double det = fma((double)a0, (double)a2, -((double)a1 * a1));
  const float s = m.inv_det(det);
  const float tmp = s * a2;
  a1 *= -s;
  a2 = s * a0;
  a0 = tmp;
}

//------------------------------------------------------------------------------
// Barrel Kalman operation: residual rotated onto the plane tangent to the
// cylinder, chi2 and/or update. Restates kalmanOperation
// (mkFit/KalmanUtilsMPlex.cc:548-681). do_update: write (opar, oerr).
//------------------------------------------------------------------------------
template <bool kChi2, bool kUpdate, class F>
__device__ __forceinline__ float kalman_barrel_in(F& m, const float (&par)[6], const float (&err)[21],
                                                  const float (&mpos)[3], const float (&merr)[6],
                                                  float (&opar)[6], float (&oerr)[21]) {
  const float r = m.hypot(mpos[0], mpos[1]);
  const float sx = mpos[0] + par[0], sy = mpos[1] + par[1];
  m.see_top(sx);
  m.see_top(sy);
  const float r00 = F::div(-sy, 2 * r);
  const float r01 = F::div(sx, 2 * r);

  const float res0 = mpos[0] - par[0], res1 = mpos[1] - par[1], res2 = mpos[2] - par[2];
  // Covariance sum in global position coordinates (upper-left 3x3).
  const float g0 = err[0] + merr[0], g1 = err[1] + merr[1], g2 = err[2] + merr[2];
  const float g3 = err[3] + merr[3], g4 = err[4] + merr[4], g5 = err[5] + merr[5];

  // Local residual and its covariance (ProjectResErr / ProjectResErrTransp).
  const float loc0 = fmaf(r00, res0, r01 * res1);
  const float loc1 = res2;
  const float t0 = fmaf(r00, g0, r01 * g1);
  const float t1 = fmaf(r00, g1, r01 * g2);
  float s0 = fmaf(t0, r00, t1 * r01);
  float s1 = fmaf(g3, r00, g4 * r01);
  float s2 = g5;
  invert_sym2(m, s0, s1, s2);

  float chi2 = 0.f;
  if (kChi2) chi2 = fmaf(2.f, s1 * loc1 * loc0, fmaf(s0 * loc0, loc0, s2 * loc1 * loc1));

  if (kUpdate) {
    // H^T G (KalmanHTG): 3x2 live block.
    const float h00 = r00 * s0, h01 = r00 * s1;
    const float h10 = r01 * s0, h11 = r01 * s1;
    const float h20 = s1, h21 = s2;
    // Gain K = C[:, 0:3] * HTG (KalmanGain): 6x2.
    float K[12];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const float ci0 = err[sidx(i, 0)], ci1 = err[sidx(i, 1)], ci2 = err[sidx(i, 2)];
      K[2 * i + 0] = fmaf(ci2, h20, fmaf(ci0, h00, ci1 * h10));
      K[2 * i + 1] = fmaf(ci2, h21, fmaf(ci0, h01, ci1 * h11));
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) opar[i] = fmaf(K[2 * i + 1], loc1, fmaf(K[2 * i], loc0, par[i]));
    opar[4] = squash_phi(opar[4]);
    // KH (KHMult): rows (K0*r00, K0*r01, K1, 0, 0, 0).
    float KH[36];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      KH[i * 6 + 0] = K[2 * i] * r00;
      KH[i * 6 + 1] = K[2 * i] * r01;
      KH[i * 6 + 2] = K[2 * i + 1];
      KH[i * 6 + 3] = 0.f;
      KH[i * 6 + 4] = 0.f;
      KH[i * 6 + 5] = 0.f;
    }
    float KHC[21];
    khc_barrel(KH, err, KHC);
#pragma unroll
    for (int i = 0; i < 21; ++i) oerr[i] = err[i] - KHC[i];
  }
  return chi2;
}

//------------------------------------------------------------------------------
// Endcap Kalman operation: xy residual, 6x2 gain. Restates
// kalmanOperationEndcap (mkFit/KalmanUtilsMPlex.cc:774-888).
//------------------------------------------------------------------------------
template <bool kChi2, bool kUpdate, class F>
__device__ __forceinline__ float kalman_endcap_in(F& m, const float (&par)[6], const float (&err)[21],
                                                  const float (&mpos)[3], const float (&merr)[6],
                                                  float (&opar)[6], float (&oerr)[21]) {
  const float res0 = mpos[0] - par[0], res1 = mpos[1] - par[1];
  float s0 = err[0] + merr[0], s1 = err[1] + merr[1], s2 = err[2] + merr[2];
  invert_sym2(m, s0, s1, s2);
  float chi2 = 0.f;
  if (kChi2) chi2 = fmaf(2.f, s1 * res1 * res0, fmaf(s0 * res0, res0, s2 * res1 * res1));
  if (kUpdate) {
    // K = C[:, 0:2] * S^-1 (KalmanGain62).
    float K[12];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const float ci0 = err[sidx(i, 0)], ci1 = err[sidx(i, 1)];
      K[2 * i + 0] = fmaf(ci0, s0, ci1 * s1);
      K[2 * i + 1] = fmaf(ci0, s1, ci1 * s2);
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) opar[i] = fmaf(K[2 * i + 1], res1, fmaf(K[2 * i], res0, par[i]));
    opar[4] = squash_phi(opar[4]);
    float KHC[21];
    khc_endcap(K, err, KHC);
#pragma unroll
    for (int i = 0; i < 21; ++i) oerr[i] = err[i] - KHC[i];
  }
  return chi2;
}

template <bool kChi2, bool kUpdate>
__device__ __forceinline__ float kalman_barrel(const float (&par)[6], const float (&err)[21],
                                               const float (&mpos)[3], const float (&merr)[6],
                                               float (&opar)[6], float (&oerr)[21]) {
  ExactMath m;
  return kalman_barrel_in<kChi2, kUpdate>(m, par, err, mpos, merr, opar, oerr);
}
template <bool kChi2, bool kUpdate>
__device__ __forceinline__ float kalman_endcap(const float (&par)[6], const float (&err)[21],
                                               const float (&mpos)[3], const float (&merr)[6],
                                               float (&opar)[6], float (&oerr)[21]) {
  ExactMath m;
  return kalman_endcap_in<kChi2, kUpdate>(m, par, err, mpos, merr, opar, oerr);
}

// The update with FlatMath, repeated with ExactMath where its operands left
// their range (see propagate_exact).
struct HitCopy {
  float pos[3], err[6];
};
template <bool kChi2>
__device__ __noinline__ float update_exact(StateCopy* s, HitCopy h, bool barrel) {
  ExactMath m;
  StateCopy o;
  const float chi2 = barrel
                         ? kalman_barrel_in<kChi2, true>(m, s->par, s->err, h.pos, h.err, o.par, o.err)
                         : kalman_endcap_in<kChi2, true>(m, s->par, s->err, h.pos, h.err, o.par, o.err);
  *s = o;
  return chi2;
}

template <bool kChi2, bool kBarrel>
__device__ __forceinline__ float update_flat(const float (&par)[6], const float (&err)[21],
                                             const float (&mpos)[3], const float (&merr)[6],
                                             float (&opar)[6], float (&oerr)[21]) {
  FlatMath m;
  float chi2 = kBarrel ? kalman_barrel_in<kChi2, true>(m, par, err, mpos, merr, opar, oerr)
                       : kalman_endcap_in<kChi2, true>(m, par, err, mpos, merr, opar, oerr);
  if (!m.ok()) {
    StateCopy s;
    HitCopy h;
#pragma unroll
    for (int i = 0; i < 6; ++i) s.par[i] = par[i];
#pragma unroll
    for (int i = 0; i < 21; ++i) s.err[i] = err[i];
#pragma unroll
    for (int i = 0; i < 3; ++i) h.pos[i] = mpos[i];
#pragma unroll
    for (int i = 0; i < 6; ++i) h.err[i] = merr[i];
    chi2 = update_exact<kChi2>(&s, h, kBarrel);
#pragma unroll
    for (int i = 0; i < 6; ++i) opar[i] = s.par[i];
#pragma unroll
    for (int i = 0; i < 21; ++i) oerr[i] = s.err[i];
  }
  return chi2;
}

}  // namespace mkfg
