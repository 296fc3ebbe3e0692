#!/usr/bin/env python3
"""Build step: writes dft_codelets.cuh, the in-register DFT-4/-5/-20/-25
codelets of the channeliser's 12500-point complex FFT.

The codelets follow the textbook Cooley-Tukey split of a length N = N1*N2 DFT
(inner DFTs of length N1 over n1, twiddles W_N^(n2*k1), outer DFTs of length
N2 over n2).  All constants are cos/sin of rational multiples of 2*pi computed
here in double precision and written as float literals, which become immediate
operands; nothing is taken from a library.  Output order: the value
X[k1 + N1*k2] is left in v[N2*k1 + k2] (the caller's stores undo the
permutation at compile time).

Run:  python gen_dft.py > dft_codelets.cuh
"""
import math


def lit(x: float) -> str:
    return "0.0f" if abs(x) < 1e-300 else f"{x:.9e}f"


def w(e: int, n: int):
    a = -2.0 * math.pi * e / n
    return math.cos(a), math.sin(a)


HEADER = """// Generated by gen_dft.py -- do not edit by hand.
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
// pi/5) and s1, s2 the sines: (c1 + c2)/2 = -1/4, (c1 - c2)/2 = sqrt(5)/4, s2 = RHO s1
__device__ __forceinline__ void dft5(Cx& a, Cx& b, Cx& c, Cx& d, Cx& e) {
  constexpr float h = H5, s1 = S1, rho = RHO;
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
"""


def codelet(n1: int, n2: int) -> str:
    n = n1 * n2
    s = f"\n// forward DFT-{n} = {n1} x {n2}; X[k1 + {n1}*k2] ends in v[{n2}*k1 + k2].  The inner DFT of\n"
    s += f"// inputs Q, Q + {n2}, ... and its twiddles (for each Q < {n2}), then the outer ones:\n"
    s += "template <int Q>\n"
    s += f"__device__ __forceinline__ void dft{n}_inner(Cx (&v)[{n}]) {{\n"
    s += f"  dft{n1}({', '.join(f'v[Q + {n2 * i}]' for i in range(n1))});\n"
    for q in range(1, n2):
        s += f"  if constexpr (Q == {q}) {{\n"
        for k1 in range(1, n1):
            c, sn = w((q * k1) % n, n)
            s += f"    cx_mul(v[{n2 * k1 + q}], {lit(c)}, {lit(sn)});  // W_{n}^{(q * k1) % n}\n"
        s += "  }\n"
    s += "}\n"
    s += f"__device__ __forceinline__ void dft{n}_outer(Cx (&v)[{n}]) {{\n"
    for k1 in range(n1):
        s += f"  dft{n2}({', '.join(f'v[{n2 * k1 + q}]' for q in range(n2))});\n"
    s += "}\n"
    s += (f"// output index r of dft{n} lives in v[dft{n}_pos(r)]\n"
          f"__host__ __device__ constexpr int dft{n}_pos(int r) {{ return {n2} * (r % {n1}) + r / {n1}; }}\n")
    return s


def main():
    out = HEADER
    s1 = math.sin(2 * math.pi / 5)
    for k, v in (("H5", math.sqrt(5.0) / 4.0), ("S1", s1), ("RHO", math.sin(4 * math.pi / 5) / s1)):
        out = out.replace(f" = {k}", f" = {lit(v)}")
    print(out + codelet(5, 5) + codelet(4, 5) + "\n}  // namespace vfrb\n", end="")


if __name__ == "__main__":
    main()
