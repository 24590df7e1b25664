// Two single-precision values in one 64-bit register pair, with sm_100a's
// packed arithmetic: one instruction adds, multiplies or multiply-adds both.
// A kernel that transforms two columns per thread keeps column c's real parts
// of both in one F2 and their imaginary parts in another, so the codelets
// (engine.cuh) run unchanged on cpx<F2> with half the instructions.  The
// arithmetic units' rate is the same either way (measured: 126 packed and 110
// scalar lane operations per SM and clock); what is saved is issue slots.
// Each packed operation rounds each half as the scalar one does.
#pragma once

#include <cstring>

#include "engine.cuh"

namespace ffb {

struct F2 {
  unsigned long long v;
  F2() = default;
  FFB_HD F2(float a, float b) {
#ifdef __CUDA_ARCH__
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
#else
    const float t[2] = {a, b};
    std::memcpy(&v, t, 8);
#endif
  }
  FFB_HD explicit F2(double c) : F2((float)c, (float)c) {}
  FFB_HD void get(float &a, float &b) const {
#ifdef __CUDA_ARCH__
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
#else
    float t[2];
    std::memcpy(t, &v, 8);
    a = t[0];
    b = t[1];
#endif
  }
};

#ifdef __CUDA_ARCH__
#define FFB_F2_OP(name, ins)                                                   \
  FFB_HD F2 name(F2 a, F2 b) {                                                 \
    F2 r;                                                                      \
    asm(ins ".f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));            \
    return r;                                                                  \
  }
FFB_F2_OP(operator+, "add.rn")
FFB_F2_OP(operator-, "sub.rn")
FFB_F2_OP(operator*, "mul.rn")
#undef FFB_F2_OP
FFB_HD F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
#else
template <class F>
inline F2 f2_apply(F2 a, F2 b, F f) {
  float a0, a1, b0, b1;
  a.get(a0, a1);
  b.get(b0, b1);
  return F2(f(a0, b0), f(a1, b1));
}
inline F2 operator+(F2 a, F2 b) {
  return f2_apply(a, b, [](float x, float y) { return x + y; });
}
inline F2 operator-(F2 a, F2 b) {
  return f2_apply(a, b, [](float x, float y) { return x - y; });
}
inline F2 operator*(F2 a, F2 b) {
  return f2_apply(a, b, [](float x, float y) { return x * y; });
}
inline F2 fma2(F2 a, F2 b, F2 c) { return a * b + c; }
#endif
FFB_HD F2 operator-(F2 a) { return a * F2(-1.0); }

// The rotations and small codelets written for F2 in multiply-adds, without
// negations (a packed value has no free sign change).
template <>
struct Dft<3, F2> {
  static FFB_HD void run(cpx<F2> *v) {
    const F2 c(-0.5), s(0.86602540378443864676), ms(-0.86602540378443864676);
    const cpx<F2> t1 = v[1] + v[2], t2 = v[1] - v[2];
    const cpx<F2> m1 = mk(fma2(c, t1.x, v[0].x), fma2(c, t1.y, v[0].y));
    v[0] = v[0] + t1;
    v[1] = mk(fma2(s, t2.y, m1.x), fma2(ms, t2.x, m1.y));
    v[2] = mk(fma2(ms, t2.y, m1.x), fma2(s, t2.x, m1.y));
  }
};
template <>
struct Dft<4, F2> {
  static FFB_HD void run(cpx<F2> *v) {
    const cpx<F2> a = v[0] + v[2], b = v[0] - v[2];
    const cpx<F2> c = v[1] + v[3], e = v[1] - v[3];
    v[0] = a + c;
    v[2] = a - c;
    v[1] = mk(b.x + e.y, b.y - e.x);
    v[3] = mk(b.x - e.y, b.y + e.x);
  }
};
// a times exp(-2 pi i m / 16)
FFB_HD cpx<F2> rot16(cpx<F2> a, int m) {
  const double r2 = 0.70710678118654752440, c1 = 0.92387953251128675613, s1 = 0.38268343236508977173;
  switch (m) {
    case 1: return mk(fma2(a.x, F2(c1), a.y * F2(s1)), fma2(a.y, F2(c1), a.x * F2(-s1)));
    case 2: return mk(F2(r2) * (a.x + a.y), F2(r2) * (a.y - a.x));
    case 3: return mk(fma2(a.x, F2(s1), a.y * F2(c1)), fma2(a.y, F2(s1), a.x * F2(-c1)));
    case 4: return mk(a.y, -a.x);
    case 6: return mk(F2(r2) * (a.y - a.x), F2(-r2) * (a.x + a.y));
    case 9: return mk(fma2(a.x, F2(-c1), a.y * F2(-s1)), fma2(a.y, F2(-c1), a.x * F2(s1)));
    default: return a;
  }
}
template <>
struct Dft<16, F2> {
  static FFB_HD void run(cpx<F2> *v) {
    cpx<F2> u[16];
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
      cpx<F2> t[4] = {v[n2], v[4 + n2], v[8 + n2], v[12 + n2]};
      Dft<4, F2>::run(t);
#pragma unroll
      for (int k1 = 0; k1 < 4; ++k1) u[n2 * 4 + k1] = rot16(t[k1], n2 * k1);
    }
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
      cpx<F2> t[4] = {u[k1], u[4 + k1], u[8 + k1], u[12 + k1]};
      Dft<4, F2>::run(t);
#pragma unroll
      for (int k2 = 0; k2 < 4; ++k2) v[k1 + 4 * k2] = t[k2];
    }
  }
};

// The codelet in direction INV: the inverse is the forward one with real and
// imaginary parts exchanged on both sides (a renaming of registers).
template <int R, bool INV>
FFB_HD void dft_swapped(cpx<F2> *v) {
  if constexpr (INV) {
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = mk(v[r].y, v[r].x);
  }
  Dft<R, F2>::run(v);
  if constexpr (INV) {
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = mk(v[r].y, v[r].x);
  }
}

// a * w: one twiddle for every column the value holds
FFB_HD cpx<F2> mul_tw(cpx<F2> a, cpx<float> w) {
  const F2 wr(w.x, w.x), wi(w.y, w.y), mi(-w.y, -w.y);
  return mk(fma2(a.x, wr, a.y * mi), fma2(a.y, wr, a.x * wi));
}

// a * b, each column its own factor
FFB_HD cpx<F2> mul_each(cpx<F2> a, cpx<F2> b) {
  return mk(fma2(a.x, b.x, (-a.y) * b.y), fma2(a.y, b.x, a.x * b.y));
}

}  // namespace ffb
