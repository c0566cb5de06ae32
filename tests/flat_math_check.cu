// Compares the branch-free arithmetic of csrc/flat_math.cuh with the plain
// one on the device; built and loaded by test_flat_math_gpu.py.
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
