// Generated by gen_dft.py -- do not edit by hand.
// Forward DFT codelets (W = exp(-2*pi*i/N)) in registers.
#pragma once
#include <cuda_runtime.h>

namespace vfrb {

struct Cx {
  float re, im;
};

// v *= c + i*s
__device__ __forceinline__ void cx_mul(Cx& v, float c, float s) {
  const float re = fmaf(-v.im, s, v.re * c);
  v.im = fmaf(v.re, s, v.im * c);
  v.re = re;
}
__device__ __forceinline__ Cx cx_prod(Cx a, Cx b) {
  return Cx{fmaf(-a.im, b.im, a.re * b.re), fmaf(a.re, b.im, a.im * b.re)};
}

// packed pairs (re, im): one instruction for both where nothing crosses over
__device__ __forceinline__ float2 f2(const Cx& v) { return make_float2(v.re, v.im); }
__device__ __forceinline__ float2 f2s(float c) { return make_float2(c, c); }
__device__ __forceinline__ float2 f2subv(float2 a, float2 b) {
  unsigned long long x, y, d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(b.x), "f"(b.y));
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x), "l"(y));
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(d));
  return r;
}
__device__ __forceinline__ float2 f2add(const Cx& a, const Cx& b) { return __fadd2_rn(f2(a), f2(b)); }
__device__ __forceinline__ float2 f2sub(const Cx& a, const Cx& b) { return f2subv(f2(a), f2(b)); }

// forward DFT-4 in place: (a,b,c,d) <- X0..X3
__device__ __forceinline__ void dft4(Cx& a, Cx& b, Cx& c, Cx& d) {
  const float2 p = f2add(a, c), m = f2sub(a, c), q = f2add(b, d), n = f2sub(b, d);
  const float2 x0 = __fadd2_rn(p, q), x2 = f2subv(p, q);
  a = Cx{x0.x, x0.y};
  c = Cx{x2.x, x2.y};
  b = Cx{m.x + n.y, m.y - n.x};
  d = Cx{m.x - n.y, m.y + n.x};
}

// forward DFT-5 in place: (a,b,c,d,e) <- X0..X4.  With c1, c2 = cos(2 pi/5), cos(4
// pi/5) and s1, s2 the sines: (c1 + c2)/2 = -1/4, (c1 - c2)/2 = sqrt(5)/4, s2 = 6.180339887e-01f s1
__device__ __forceinline__ void dft5(Cx& a, Cx& b, Cx& c, Cx& d, Cx& e) {
  constexpr float h = 5.590169944e-01f, s1 = 9.510565163e-01f, rho = 6.180339887e-01f;
  const float2 t1 = f2add(b, e), t2 = f2add(c, d), t3 = f2sub(b, e), t4 = f2sub(d, c);  // t4 negated
  const float2 u = __fadd2_rn(t1, t2), m = __ffma2_rn(f2s(-0.25f), u, f2(a));
  const float2 v = f2subv(t1, t2);
  const float2 m1 = __ffma2_rn(f2s(h), v, m), m2 = __ffma2_rn(f2s(-h), v, m);
  const float2 n1 = __ffma2_rn(f2s(-rho), t4, t3), n2 = __ffma2_rn(f2s(rho), t3, t4);
  const float2 a0 = __fadd2_rn(f2(a), u);
  a = Cx{a0.x, a0.y};
  // X1 = m1 - i*s1*n1, X4 = m1 + i*s1*n1, X2 = m2 - i*s1*n2, X3 = m2 + i*s1*n2
  b = Cx{fmaf(s1, n1.y, m1.x), fmaf(-s1, n1.x, m1.y)};
  e = Cx{fmaf(-s1, n1.y, m1.x), fmaf(s1, n1.x, m1.y)};
  c = Cx{fmaf(s1, n2.y, m2.x), fmaf(-s1, n2.x, m2.y)};
  d = Cx{fmaf(-s1, n2.y, m2.x), fmaf(s1, n2.x, m2.y)};
}

// forward DFT-25 = 5 x 5; X[k1 + 5*k2] ends in v[5*k1 + k2].  The inner DFT of
// inputs Q, Q + 5, ... and its twiddles (for each Q < 5), then the outer ones:
template <int Q>
__device__ __forceinline__ void dft25_inner(Cx (&v)[25]) {
  dft5(v[Q + 0], v[Q + 5], v[Q + 10], v[Q + 15], v[Q + 20]);
  if constexpr (Q == 1) {
    cx_mul(v[6], 9.685831611e-01f, -2.486898872e-01f);  // W_25^1
    cx_mul(v[11], 8.763066800e-01f, -4.817536741e-01f);  // W_25^2
    cx_mul(v[16], 7.289686274e-01f, -6.845471059e-01f);  // W_25^3
    cx_mul(v[21], 5.358267950e-01f, -8.443279255e-01f);  // W_25^4
  }
  if constexpr (Q == 2) {
    cx_mul(v[7], 8.763066800e-01f, -4.817536741e-01f);  // W_25^2
    cx_mul(v[12], 5.358267950e-01f, -8.443279255e-01f);  // W_25^4
    cx_mul(v[17], 6.279051953e-02f, -9.980267284e-01f);  // W_25^6
    cx_mul(v[22], -4.257792916e-01f, -9.048270525e-01f);  // W_25^8
  }
  if constexpr (Q == 3) {
    cx_mul(v[8], 7.289686274e-01f, -6.845471059e-01f);  // W_25^3
    cx_mul(v[13], 6.279051953e-02f, -9.980267284e-01f);  // W_25^6
    cx_mul(v[18], -6.374239897e-01f, -7.705132428e-01f);  // W_25^9
    cx_mul(v[23], -9.921147013e-01f, -1.253332336e-01f);  // W_25^12
  }
  if constexpr (Q == 4) {
    cx_mul(v[9], 5.358267950e-01f, -8.443279255e-01f);  // W_25^4
    cx_mul(v[14], -4.257792916e-01f, -9.048270525e-01f);  // W_25^8
    cx_mul(v[19], -9.921147013e-01f, -1.253332336e-01f);  // W_25^12
    cx_mul(v[24], -6.374239897e-01f, 7.705132428e-01f);  // W_25^16
  }
}
__device__ __forceinline__ void dft25_outer(Cx (&v)[25]) {
  dft5(v[0], v[1], v[2], v[3], v[4]);
  dft5(v[5], v[6], v[7], v[8], v[9]);
  dft5(v[10], v[11], v[12], v[13], v[14]);
  dft5(v[15], v[16], v[17], v[18], v[19]);
  dft5(v[20], v[21], v[22], v[23], v[24]);
}
// output index r of dft25 lives in v[dft25_pos(r)]
__host__ __device__ constexpr int dft25_pos(int r) { return 5 * (r % 5) + r / 5; }

// forward DFT-20 = 4 x 5; X[k1 + 4*k2] ends in v[5*k1 + k2].  The inner DFT of
// inputs Q, Q + 5, ... and its twiddles (for each Q < 5), then the outer ones:
template <int Q>
__device__ __forceinline__ void dft20_inner(Cx (&v)[20]) {
  dft4(v[Q + 0], v[Q + 5], v[Q + 10], v[Q + 15]);
  if constexpr (Q == 1) {
    cx_mul(v[6], 9.510565163e-01f, -3.090169944e-01f);  // W_20^1
    cx_mul(v[11], 8.090169944e-01f, -5.877852523e-01f);  // W_20^2
    cx_mul(v[16], 5.877852523e-01f, -8.090169944e-01f);  // W_20^3
  }
  if constexpr (Q == 2) {
    cx_mul(v[7], 8.090169944e-01f, -5.877852523e-01f);  // W_20^2
    cx_mul(v[12], 3.090169944e-01f, -9.510565163e-01f);  // W_20^4
    cx_mul(v[17], -3.090169944e-01f, -9.510565163e-01f);  // W_20^6
  }
  if constexpr (Q == 3) {
    cx_mul(v[8], 5.877852523e-01f, -8.090169944e-01f);  // W_20^3
    cx_mul(v[13], -3.090169944e-01f, -9.510565163e-01f);  // W_20^6
    cx_mul(v[18], -9.510565163e-01f, -3.090169944e-01f);  // W_20^9
  }
  if constexpr (Q == 4) {
    cx_mul(v[9], 3.090169944e-01f, -9.510565163e-01f);  // W_20^4
    cx_mul(v[14], -8.090169944e-01f, -5.877852523e-01f);  // W_20^8
    cx_mul(v[19], -8.090169944e-01f, 5.877852523e-01f);  // W_20^12
  }
}
__device__ __forceinline__ void dft20_outer(Cx (&v)[20]) {
  dft5(v[0], v[1], v[2], v[3], v[4]);
  dft5(v[5], v[6], v[7], v[8], v[9]);
  dft5(v[10], v[11], v[12], v[13], v[14]);
  dft5(v[15], v[16], v[17], v[18], v[19]);
}
// output index r of dft20 lives in v[dft20_pos(r)]
__host__ __device__ constexpr int dft20_pos(int r) { return 5 * (r % 4) + r / 4; }

}  // namespace vfrb
