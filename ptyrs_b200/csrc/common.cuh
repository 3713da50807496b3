// Shared device helpers: complex float2 arithmetic and compensated sums.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define PTYB_HD __host__ __device__ __forceinline__
#define PTYB_D __device__ __forceinline__

PTYB_HD float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
PTYB_HD float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
PTYB_HD float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// conj(a) * b
PTYB_HD float2 cmulc(float2 a, float2 b) {
  return make_float2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}
// a * b and conj(a) * b in the line transforms and around them: the products that are rounded
// and those that are fused are written out, so the result does not depend on what the compiler
// makes of the code around.
PTYB_D float2 cmul_rn(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -(a.y * b.y)), fmaf(a.x, b.y, a.y * b.x));
}
PTYB_D float2 cmulc_rn(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(a.x, b.y, -(a.y * b.x)));
}
PTYB_HD float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
// conj(a) * b with the other product of the imaginary part fused: the probe sums' form, as accurate
// as the one above, and kept apart from it for the same case's bits (fft.cuh, rotate_by).
PTYB_D float2 cmulc_rn2(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(-a.y, b.x, a.x * b.y));
}
// a + b and a − b as one packed instruction each (both components per issue slot).
PTYB_D float2 cadd2(float2 a, float2 b) {
  float2 r;
  asm("{.reg .b64 x, y, z; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; add.rn.f32x2 z, x, y; "
      "mov.b64 {%0, %1}, z;}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
PTYB_D float2 csub2(float2 a, float2 b) {
  float2 r;
  asm("{.reg .b64 x, y, z, m; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; mov.b64 m, {%6, %6}; "
      "fma.rn.f32x2 z, y, m, x; mov.b64 {%0, %1}, z;}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(-1.f));
  return r;
}
// cscale, not contracted into an addition that follows.
PTYB_D float2 cscale_rn(float2 a, float s) {
  return make_float2(__fmul_rn(a.x, s), __fmul_rn(a.y, s));
}
PTYB_HD float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
PTYB_HD float cnorm2(float2 a) { return a.x * a.x + a.y * a.y; }

// Kahan-compensated accumulation of a float: sum and running compensation.
struct Kahan {
  float s, c;
  PTYB_D void init() { s = 0.f; c = 0.f; }
  PTYB_D void add(float v) {
    float y = v - c;
    float t = s + y;
    c = (t - s) - y;
    s = t;
  }
};

struct KahanC {
  Kahan re, im;
  PTYB_D void init() { re.init(); im.init(); }
  PTYB_D void add(float2 v) { re.add(v.x); im.add(v.y); }
  PTYB_D float2 value() const { return make_float2(re.s, im.s); }
};

// Bits of a non-negative float order as the float does, so an unsigned atomicMax on them is
// a float max that gives the same result in any order.
PTYB_D void atomic_max_nonneg(float* addr, float v) {
  atomicMax(reinterpret_cast<unsigned int*>(addr), __float_as_uint(fmaxf(v, 0.f)));
}

// Warp and block reductions in double.
PTYB_D double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
PTYB_D float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// v[i0] + v[i0+1] + … + v[i1−1] in that order by one thread, eight loads ahead of the additions.
PTYB_D double ordered_sum(const double* v, int i0, int i1) {
  double s = 0.0;
  int i = i0;
  for (; i + 8 <= i1; i += 8) {
    double a[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = v[i + k];
#pragma unroll
    for (int k = 0; k < 8; ++k) s += a[k];
  }
  for (; i < i1; ++i) s += v[i];
  return s;
}
