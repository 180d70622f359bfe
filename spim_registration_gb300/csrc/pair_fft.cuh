// Register DFTs on pairs of complex numbers with the packed FP32 instructions of sm_103a.
//
// A C2 holds two complex numbers as two 64-bit register pairs, (re_a, re_b) and (im_a, im_b): the
// same step of two independent transforms.  add / mul / fma.rn.f32x2 then do two transforms'
// arithmetic in one instruction each.  The FP32 pipe's rate is the same either way (measured:
// FFMA 125 and FFMA2 128 lane operations per clock and SM), but the packed form takes half the
// issue slots, which is what bounds the FFT passes, and one 16-byte access moves both numbers.
// Every rounding is the scalar instruction's.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "dft_consts.cuh"

namespace mvd {

using f2 = unsigned long long;  // two floats in a register pair (low: first)

__device__ __forceinline__ f2 pk(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpk(f2 v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

struct C2 {
  f2 r, i;
};

__device__ __forceinline__ C2 operator+(C2 a, C2 b) { return {add2(a.r, b.r), add2(a.i, b.i)}; }
__device__ __forceinline__ C2 operator-(C2 a, C2 b) { return {sub2(a.r, b.r), sub2(a.i, b.i)}; }
// a - i b (forward) or a + i b (inverse), and the other sign
template <bool INV>
__device__ __forceinline__ C2 add_mi(C2 a, C2 b) {
  return INV ? C2{sub2(a.r, b.i), add2(a.i, b.r)} : C2{add2(a.r, b.i), sub2(a.i, b.r)};
}
template <bool INV>
__device__ __forceinline__ C2 sub_mi(C2 a, C2 b) {
  return add_mi<!INV>(a, b);
}
// a times a root given as (x, x), (y, y), (-y, -y); INV: its conjugate
template <bool INV>
__device__ __forceinline__ C2 mul_root(C2 a, f2 x, f2 y, f2 ny) {
  return {fma2(a.i, INV ? y : ny, mul2(a.r, x)), fma2(a.i, x, mul2(a.r, INV ? ny : y))};
}
// a times the per-lane pair (w.r, w.i)
__device__ __forceinline__ C2 mul_c2(C2 a, C2 w) {
  return {sub2(mul2(a.r, w.r), mul2(a.i, w.i)), fma2(a.i, w.r, mul2(a.r, w.i))};
}

__device__ __forceinline__ C2 ld_c2(const float4* p) {  // shared or global memory, 16 bytes
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  return {v.x, v.y};
}
__device__ __forceinline__ void st_c2(float4* p, C2 v) { *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v.r, v.i); }

// ---------------------------------------------------------------------------------------
// R-point DFTs in registers, natural order in and out; forward exp(-2 pi i / R)
// ---------------------------------------------------------------------------------------
template <int R, bool INV>
struct PDft;

template <bool INV>
struct PDft<1, INV> {
  __device__ __forceinline__ static void run(C2*) {}
};

template <bool INV>
struct PDft<2, INV> {
  __device__ __forceinline__ static void run(C2* v) {
    const C2 a = v[0], b = v[1];
    v[0] = a + b;
    v[1] = a - b;
  }
};

template <bool INV>
struct PDft<3, INV> {
  __device__ __forceinline__ static void run(C2* v) {
    const f2 c = pk(-0.5f, -0.5f);
    const f2 s = pk(0.86602540378443864676f, 0.86602540378443864676f);  // sin(2 pi / 3)
    const f2 ns = pk(-0.86602540378443864676f, -0.86602540378443864676f);
    const C2 a = v[1] + v[2], b = v[1] - v[2];
    const C2 t = {fma2(a.r, c, v[0].r), fma2(a.i, c, v[0].i)};
    v[0] = v[0] + a;
    v[1] = {fma2(b.i, INV ? ns : s, t.r), fma2(b.r, INV ? s : ns, t.i)};
    v[2] = {fma2(b.i, INV ? s : ns, t.r), fma2(b.r, INV ? ns : s, t.i)};
  }
};

template <bool INV>
struct PDft<4, INV> {
  __device__ __forceinline__ static void run(C2* v) {
    const C2 s0 = v[0] + v[2], d0 = v[0] - v[2], s1 = v[1] + v[3], d1 = v[1] - v[3];
    v[0] = s0 + s1;
    v[2] = s0 - s1;
    v[1] = add_mi<INV>(d0, d1);
    v[3] = sub_mi<INV>(d0, d1);
  }
};

template <bool INV>
struct PDft<5, INV> {
  __device__ __forceinline__ static void run(C2* v) {
    const f2 c1 = pk(0.30901699437494742410f, 0.30901699437494742410f);    // cos(2 pi / 5)
    const f2 c2 = pk(-0.80901699437494742410f, -0.80901699437494742410f);  // cos(4 pi / 5)
    const f2 s1 = pk(0.95105651629515357212f, 0.95105651629515357212f);    // sin(2 pi / 5)
    const f2 ns1 = pk(-0.95105651629515357212f, -0.95105651629515357212f);
    const f2 s2 = pk(0.58778525229247312917f, 0.58778525229247312917f);  // sin(4 pi / 5)
    const C2 p1 = v[1] + v[4], m1 = v[1] - v[4], p2 = v[2] + v[3], m2 = v[2] - v[3];
    const C2 x0 = v[0];
    const C2 a1 = {fma2(c2, p2.r, fma2(c1, p1.r, x0.r)), fma2(c2, p2.i, fma2(c1, p1.i, x0.i))};
    const C2 a2 = {fma2(c1, p2.r, fma2(c2, p1.r, x0.r)), fma2(c1, p2.i, fma2(c2, p1.i, x0.i))};
    const C2 b1 = {fma2(s2, m2.r, mul2(s1, m1.r)), fma2(s2, m2.i, mul2(s1, m1.i))};
    const C2 b2 = {fma2(ns1, m2.r, mul2(s2, m1.r)), fma2(ns1, m2.i, mul2(s2, m1.i))};
    v[0] = x0 + (p1 + p2);
    v[1] = add_mi<INV>(a1, b1);
    v[4] = sub_mi<INV>(a1, b1);
    v[2] = add_mi<INV>(a2, b2);
    v[3] = sub_mi<INV>(a2, b2);
  }
};

template <bool INV>
struct PDft<8, INV> {
  __device__ __forceinline__ static void run(C2* v) {
    const f2 h = pk(0.70710678118654752440f, 0.70710678118654752440f);  // sqrt(1/2)
    const f2 nh = pk(-0.70710678118654752440f, -0.70710678118654752440f);
    C2 e[4] = {v[0], v[2], v[4], v[6]};
    C2 o[4] = {v[1], v[3], v[5], v[7]};
    PDft<4, INV>::run(e);
    PDft<4, INV>::run(o);
    // o[1] h (1 -+ i) and o[3] h (-1 -+ i), the factor h folded into the last additions
    const C2 t1 = add_mi<INV>(o[1], o[1]), t3 = sub_mi<INV>(o[3], o[3]);
    v[0] = e[0] + o[0];
    v[4] = e[0] - o[0];
    v[1] = {fma2(h, t1.r, e[1].r), fma2(h, t1.i, e[1].i)};
    v[5] = {fma2(nh, t1.r, e[1].r), fma2(nh, t1.i, e[1].i)};
    v[2] = add_mi<INV>(e[2], o[2]);
    v[6] = sub_mi<INV>(e[2], o[2]);
    v[3] = {fma2(nh, t3.r, e[3].r), fma2(nh, t3.i, e[3].i)};
    v[7] = {fma2(h, t3.r, e[3].r), fma2(h, t3.i, e[3].i)};
  }
};

// R = A * B by one Cooley-Tukey split (as DftAB in fft_device.cuh)
template <int A, int B, bool INV>
struct PDftAB {
  __device__ __forceinline__ static void run(C2* v) {
    constexpr int R = A * B;
    C2 y[B][A];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
      C2 t[A];
#pragma unroll
      for (int n1 = 0; n1 < A; ++n1) t[n1] = v[B * n1 + n2];
      PDft<A, INV>::run(t);
#pragma unroll
      for (int k1 = 0; k1 < A; ++k1) {
        const int m = n2 * k1;
        if (m == 0) {
          y[n2][k1] = t[k1];
        } else if (4 * m == R) {  // -i (forward), +i (inverse)
          const f2 z = 0ull;
          y[n2][k1] = INV ? C2{sub2(z, t[k1].i), t[k1].r} : C2{t[k1].i, sub2(z, t[k1].r)};
        } else {
          const float2 w = wroot<R>(m);
          y[n2][k1] = mul_root<INV>(t[k1], pk(w.x, w.x), pk(w.y, w.y), pk(-w.y, -w.y));
        }
      }
    }
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      C2 t[B];
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) t[n2] = y[n2][k1];
      PDft<B, INV>::run(t);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = t[k2];
    }
  }
};

template <bool INV> struct PDft<6, INV> : PDftAB<2, 3, INV> {};
template <bool INV> struct PDft<9, INV> : PDftAB<3, 3, INV> {};
template <bool INV> struct PDft<10, INV> : PDftAB<2, 5, INV> {};
template <bool INV> struct PDft<12, INV> : PDftAB<4, 3, INV> {};
template <bool INV> struct PDft<15, INV> : PDftAB<3, 5, INV> {};
template <bool INV> struct PDft<16, INV> : PDftAB<4, 4, INV> {};
template <bool INV> struct PDft<18, INV> : PDftAB<2, 9, INV> {};
template <bool INV> struct PDft<20, INV> : PDftAB<4, 5, INV> {};

}  // namespace mvd
