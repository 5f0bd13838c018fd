// Short DFTs in registers, shared by the FFT passes of the cone stage.
//
// The passes are bound by instruction issue and latency before the float32 pipe
// (x pass of seven beams at 192^3: 0.32 ms of the pipe, 0.27 of memory, in 0.68).
// So complex sums take one packed instruction (add.rn.f32x2: the pipe's time of
// two, one issue slot, the same roundings), and the rotations inside 16 points
// are two multiply-adds (t x + y, t y - x with t = cot 22.5 or 1) whose common
// factor sin 22.5 or cos 45 joins the sums that follow (rms error of 16 points
// against float64 6.1e-8 -> 5.9e-8).  Cone stage, scalar / this: 64 mixed beams
// 2768 / 2615 us, 32 at 128^3 1268 / 1205, four at 160^3 424 / 396, at 201^3 1271
// / 1237, seven at 192^3 1254 / 1236.
//
// The header needs nothing but the vector types and compiles for the host too
// (tests/test_spectral_dft_cpu.py), with scalar forms of the packed instructions.
#pragma once

#include <cuda_runtime.h>

namespace ch {

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// ------------------------------------------------- compile-time cos, sin --
// Taylor series on [0, pi / 4] (terms down to 1e-20), octants by symmetry.
constexpr double ct_sin0(double x) {
  double t = x, s = x;
  for (int k = 1; k < 12; ++k) {
    t *= -x * x / (double)((2 * k) * (2 * k + 1));
    s += t;
  }
  return s;
}
constexpr double ct_cos0(double x) {
  double t = 1.0, s = 1.0;
  for (int k = 1; k < 12; ++k) {
    t *= -x * x / (double)((2 * k - 1) * (2 * k));
    s += t;
  }
  return s;
}
constexpr double CT_PI = 3.14159265358979323846;
// cos and sin of 2 pi k / n, 0 <= k (any size), n > 0
constexpr double ct_cos(int k, int n);
constexpr double ct_sin(int k, int n) {
  k %= n;
  return 2 * k > n    ? -ct_sin(n - k, n)                       // lower half plane
         : 4 * k > n  ? ct_sin(n - 2 * k, 2 * n)                // pi - x
         : 8 * k > n  ? ct_cos0(CT_PI * (double)(n - 4 * k) / (double)(2 * n))
                      : ct_sin0(2.0 * CT_PI * (double)k / (double)n);
}
constexpr double ct_cos(int k, int n) { return ct_sin(4 * (k % n) + n, 4 * n); }

// -------------------------------------------------------- packed pairs --
#ifdef __CUDA_ARCH__
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long r) {
  float2 a;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
  return a;
}
#endif
__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
#ifdef __CUDA_ARCH__
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a.x, a.y)), "l"(pack2(b.x, b.y)));
  return unpack2(r);
#else
  return make_float2(a.x + b.x, a.y + b.y);
#endif
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
#ifdef __CUDA_ARCH__
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a.x, a.y)), "l"(pack2(b.x, b.y)));
  return unpack2(r);
#else
  return make_float2(a.x - b.x, a.y - b.y);
#endif
}
__device__ __forceinline__ float2 cscale(float2 a, float k) {
#ifdef __CUDA_ARCH__
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a.x, a.y)), "l"(pack2(k, k)));
  return unpack2(r);
#else
  return make_float2(k * a.x, k * a.y);
#endif
}
// k a + b
__device__ __forceinline__ float2 cfma(float k, float2 a, float2 b) {
#ifdef __CUDA_ARCH__
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pack2(a.x, a.y)), "l"(pack2(k, k)), "l"(pack2(b.x, b.y)));
  return unpack2(r);
#else
  return make_float2(__builtin_fmaf(k, a.x, b.x), __builtin_fmaf(k, a.y, b.y));
#endif
}
// -+i (a - b)
template <bool INV>
__device__ __forceinline__ float2 turned_diff(float2 a, float2 b) {
  return INV ? make_float2(b.y - a.y, a.x - b.x) : make_float2(a.y - b.y, b.x - a.x);
}
// a -+ i b
template <bool INV>
__device__ __forceinline__ float2 add_turned(float2 a, float2 b) {
  return INV ? make_float2(a.x - b.y, a.y + b.x) : make_float2(a.x + b.y, a.y - b.x);
}

// -------------------------------------------------------------- radix 4 --
// 4-point DFT in place (forward: X1 = d02 - i d13; inverse: d02 + i d13)
template <bool INV>
__device__ __forceinline__ void dft4(float2& a0, float2& a1, float2& a2, float2& a3) {
  const float2 s02 = cadd(a0, a2), d02 = csub(a0, a2), s13 = cadd(a1, a3), d13 = csub(a1, a3);
  a0 = cadd(s02, s13);
  a1 = add_turned<INV>(d02, d13);
  a2 = csub(s02, s13);
  a3 = add_turned<!INV>(d02, d13);
}
// the last sums of a 4-point DFT whose inputs 1 and 3 are k a1 and k a3
template <bool INV>
__device__ __forceinline__ void dft4_scaled(float k, float2 s02, float2 d02, float2& a0, float2& a1, float2& a2,
                                            float2& a3) {
  const float2 s13 = cadd(a1, a3), mi = turned_diff<INV>(a1, a3);
  a0 = cfma(k, s13, s02);
  a1 = cfma(k, mi, d02);
  a2 = cfma(-k, s13, s02);
  a3 = cfma(-k, mi, d02);
}

// v exp(-+i theta) by its common factor: 22.5 and 67.5 degrees / S1, 45 / R2
// (by sin 22.5 and not by cos 22.5: their roundings to float32, -1.6e-8 and -3.1e-8, are
// the same in every butterfly, a gain that a dose passes six times and S^ three.
// With this factor the rotations' gain cancels that of the 45 degrees, 5e-11 for
// 16 points, where the other left -1.1e-8.  Error of a dose against 64 bits: 64^3
// 1.69e-7 -> 1.29e-7, 128^3 2.34 -> 1.70, 150 x 130 x 92 2.95 -> 2.67, 192^3 2.63 ->
// 2.05; the same instructions, the same times)
constexpr float DFT_S1 = 0.38268343236508977f;   // sin(pi/8) = cos(3 pi/8)
constexpr float DFT_T1 = 2.4142135623730950f;    // cot(pi/8) = tan(3 pi/8)
constexpr float DFT_R2 = 0.70710678118654752f;   // cos(pi/4)
template <bool INV>
__device__ __forceinline__ float2 lift22(float2 v) {
  return INV ? make_float2(DFT_T1 * v.x - v.y, DFT_T1 * v.y + v.x)
             : make_float2(DFT_T1 * v.x + v.y, DFT_T1 * v.y - v.x);
}
template <bool INV>
__device__ __forceinline__ float2 lift202(float2 v) {   // a half turn and 22.5
  return INV ? make_float2(v.y - DFT_T1 * v.x, -DFT_T1 * v.y - v.x)
             : make_float2(-DFT_T1 * v.x - v.y, v.x - DFT_T1 * v.y);
}
template <bool INV>
__device__ __forceinline__ float2 lift67(float2 v) {
  return INV ? make_float2(v.x - DFT_T1 * v.y, DFT_T1 * v.x + v.y)
             : make_float2(DFT_T1 * v.y + v.x, v.y - DFT_T1 * v.x);
}
template <bool INV>
__device__ __forceinline__ float2 lift45(float2 v) {
  return INV ? make_float2(v.x - v.y, v.y + v.x) : make_float2(v.x + v.y, v.y - v.x);
}
// 135 degrees: 45 and a quarter turn
template <bool INV>
__device__ __forceinline__ float2 lift135(float2 v) {
  return INV ? make_float2(-v.x - v.y, v.x - v.y) : make_float2(v.y - v.x, -v.x - v.y);
}

// v times exp(-+i theta) given (cos theta, sin theta)
template <bool INV>
__device__ __forceinline__ float2 rot(float2 v, float c, float s) {
  const float sn = INV ? s : -s;
  return make_float2(v.x * c - v.y * sn, v.x * sn + v.y * c);
}

// 16-point DFT in place as 4 x 4: element r = 4a + b, output k = k1 + 4 k2.
// DFT4 over a for each b, times exp(-+2 pi i b k1 / 16), DFT4 over b for each
// k1; X[k1 + 4 k2] ends in v[4 k1 + k2].
template <bool INV>
__device__ __forceinline__ void dft16_tail(float2 (&v)[16]) {
  dft4<INV>(v[0], v[1], v[2], v[3]);
  {   // k1 = 1: b k1 / 16 turns of 22.5, 45 and 67.5 degrees
    v[5] = lift22<INV>(v[5]);
    v[7] = lift67<INV>(v[7]);
    const float2 w = lift45<INV>(v[6]);
    dft4_scaled<INV>(DFT_S1, cfma(DFT_R2, w, v[4]), cfma(-DFT_R2, w, v[4]), v[4], v[5], v[6], v[7]);
  }
  {   // k1 = 2: 45, 90, 135
    v[9] = lift45<INV>(v[9]);
    v[11] = lift135<INV>(v[11]);
    dft4_scaled<INV>(DFT_R2, add_turned<INV>(v[8], v[10]), add_turned<!INV>(v[8], v[10]), v[8], v[9], v[10], v[11]);
  }
  {   // k1 = 3: 67.5, 135, 202.5
    v[13] = lift67<INV>(v[13]);
    const float2 w = lift135<INV>(v[14]);
    v[15] = lift202<INV>(v[15]);
    dft4_scaled<INV>(DFT_S1, cfma(DFT_R2, w, v[12]), cfma(-DFT_R2, w, v[12]), v[12], v[13], v[14], v[15]);
  }
}
template <bool INV>
__device__ __forceinline__ void dft16(float2 (&v)[16]) {
#pragma unroll
  for (int b = 0; b < 4; ++b) dft4<INV>(v[b], v[4 + b], v[8 + b], v[12 + b]);
  dft16_tail<INV>(v);
}

// dft16 with v[8..15] = 0 (the upper half of a zero-padded input): the first
// DFT4s see two inputs
template <bool INV>
__device__ __forceinline__ void dft16_half_in(float2 (&v)[16]) {
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const float2 a0 = v[b], a1 = v[4 + b];
    v[b] = cadd(a0, a1);
    v[4 + b] = add_turned<INV>(a0, a1);
    v[8 + b] = csub(a0, a1);
    v[12 + b] = add_turned<!INV>(a0, a1);
  }
  dft16_tail<INV>(v);
}

// --------------------------------------------------------- other lengths --
// N-point DFT in place, natural order in and out, N = 2^a 3^b 5^c: N = A B
// with n = B a + b, k = k1 + A k2: DFT_A over a, times exp(-+2 pi i b k1 / N),
// DFT_B over b.
// The odd factor first: 64 mixed beams 2630 -> 2615 us, four at 160^3 402 -> 396.
constexpr int dft_first(int n) { return n % 5 == 0 && n > 5 ? 5 : n % 3 == 0 && n > 3 ? 3 : n % 8 == 0 && n > 8 ? 4 : n % 4 == 0 ? 4 : n % 2 == 0 ? 2 : n % 3 == 0 ? 3 : 5; }

template <bool INV, int N>
struct Dft {
  static __device__ __forceinline__ void run(float2 (&x)[N]) {
    constexpr int A = dft_first(N), B = N / A;
    float2 y[B][A];
#pragma unroll
    for (int b = 0; b < B; ++b) {
#pragma unroll
      for (int a = 0; a < A; ++a) y[b][a] = x[B * a + b];
      Dft<INV, A>::run(y[b]);
    }
    constexpr Table T{};
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      float2 t[B];
#pragma unroll
      for (int b = 0; b < B; ++b) {
        const int m = b * k1;                       // < N
        t[b] = y[b][k1];
        if (8 * m == N) {
          const float s = T.c[m];                   // cos 45 = sin 45
          t[b] = cscale(lift45<INV>(t[b]), s);
        } else if (4 * m == N) {
          t[b] = INV ? make_float2(-t[b].y, t[b].x) : make_float2(t[b].y, -t[b].x);
        } else if (2 * m == N) {
          t[b] = make_float2(-t[b].x, -t[b].y);
        } else if (m > 0) {
          t[b] = rot<INV>(t[b], T.c[m], T.s[m]);
        }
      }
      Dft<INV, B>::run(t);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) x[k1 + A * k2] = t[k2];
    }
  }
  struct Table {
    float c[N] = {}, s[N] = {};
    constexpr Table() {
      for (int m = 0; m < N; ++m) {
        c[m] = (float)ct_cos(m, N);
        s[m] = (float)ct_sin(m, N);
      }
    }
  };
};
template <bool INV>
struct Dft<INV, 1> {
  static __device__ __forceinline__ void run(float2 (&)[1]) {}
};
template <bool INV>
struct Dft<INV, 2> {
  static __device__ __forceinline__ void run(float2 (&x)[2]) {
    const float2 a = x[0], b = x[1];
    x[0] = cadd(a, b);
    x[1] = csub(a, b);
  }
};
// X0 = a + s, X1,2 = a - s/2 -+ i (sqrt 3 / 2) d with s = b + c, d = b - c
template <bool INV>
struct Dft<INV, 3> {
  static __device__ __forceinline__ void run(float2 (&x)[3]) {
    constexpr float H = 0.86602540378443865f;   // sqrt(3) / 2
    const float2 a = x[0], b = x[1], c = x[2];
    const float2 s = cadd(b, c), id = turned_diff<INV>(b, c), t = cfma(-0.5f, s, a);
    x[0] = cadd(a, s);
    x[1] = cfma(H, id, t);
    x[2] = cfma(-H, id, t);
  }
};
template <bool INV>
struct Dft<INV, 4> {
  static __device__ __forceinline__ void run(float2 (&x)[4]) { dft4<INV>(x[0], x[1], x[2], x[3]); }
};
// with c_k, s_k the cosine and sine of 72 k degrees, p = x1 + x4, q = x2 + x3,
// m = x1 - x4, r = x2 - x3: X1,4 = x0 + c1 p + c2 q -+ i (s1 m + s2 r),
// X2,3 = x0 + c2 p + c1 q -+ i (s2 m - s1 r)
template <bool INV>
struct Dft<INV, 5> {
  static __device__ __forceinline__ void run(float2 (&x)[5]) {
    constexpr float C1 = 0.30901699437494742f, C2 = -0.80901699437494742f;
    constexpr float S1 = 0.95105651629515357f, S2 = 0.58778525229247313f;
    const float2 a = x[0];
    const float2 p = cadd(x[1], x[4]), q = cadd(x[2], x[3]);
    const float2 im = turned_diff<INV>(x[1], x[4]), ir = turned_diff<INV>(x[2], x[3]);   // -+i m, -+i r
    const float2 u = cfma(C2, q, cfma(C1, p, a)), v = cfma(C1, q, cfma(C2, p, a));
    const float2 g = cfma(S2, ir, cscale(im, S1)), h = cfma(-S1, ir, cscale(im, S2));
    x[0] = cadd(cadd(a, p), q);
    x[1] = cadd(u, g);
    x[4] = csub(u, g);
    x[2] = cadd(v, h);
    x[3] = csub(v, h);
  }
};

}  // namespace ch
