// Short DFTs in registers, shared by the FFT passes of the cone stage.
#pragma once

#include "ch_internal.cuh"

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

// -------------------------------------------------------------- radix 4 --
// 4-point DFT in place (forward: X1 = d02 - i d13; inverse: d02 + i d13)
template <bool INV>
__device__ __forceinline__ void dft4(float2& a0, float2& a1, float2& a2, float2& a3) {
  const float2 s02 = make_float2(a0.x + a2.x, a0.y + a2.y), d02 = make_float2(a0.x - a2.x, a0.y - a2.y);
  const float2 s13 = make_float2(a1.x + a3.x, a1.y + a3.y), d13 = make_float2(a1.x - a3.x, a1.y - a3.y);
  const float2 mi = INV ? make_float2(-d13.y, d13.x) : make_float2(d13.y, -d13.x);
  a0 = make_float2(s02.x + s13.x, s02.y + s13.y);
  a1 = make_float2(d02.x + mi.x, d02.y + mi.y);
  a2 = make_float2(s02.x - s13.x, s02.y - s13.y);
  a3 = make_float2(d02.x - mi.x, d02.y - mi.y);
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
  constexpr float C1 = 0.92387953251128674f;   // cos(pi/8)
  constexpr float S1 = 0.38268343236508977f;   // sin(pi/8)
  constexpr float R2 = 0.70710678118654752f;   // cos(pi/4)
  v[5] = rot<INV>(v[5], C1, S1);     // b k1 = 1
  v[9] = rot<INV>(v[9], R2, R2);     // 2
  v[13] = rot<INV>(v[13], S1, C1);   // 3
  v[6] = rot<INV>(v[6], R2, R2);     // 2
  v[10] = INV ? make_float2(-v[10].y, v[10].x) : make_float2(v[10].y, -v[10].x);   // times -+i   // 4
  v[14] = rot<INV>(v[14], -R2, R2);  // 6
  v[7] = rot<INV>(v[7], S1, C1);     // 3
  v[11] = rot<INV>(v[11], -R2, R2);  // 6
  v[15] = rot<INV>(v[15], -C1, -S1); // 9
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) dft4<INV>(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
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
    const float2 mi = INV ? make_float2(-a1.y, a1.x) : make_float2(a1.y, -a1.x);   // -+i a1
    v[b] = make_float2(a0.x + a1.x, a0.y + a1.y);
    v[4 + b] = make_float2(a0.x + mi.x, a0.y + mi.y);
    v[8 + b] = make_float2(a0.x - a1.x, a0.y - a1.y);
    v[12 + b] = make_float2(a0.x - mi.x, a0.y - mi.y);
  }
  dft16_tail<INV>(v);
}

// --------------------------------------------------------- other lengths --
// N-point DFT in place, natural order in and out, N = 2^a 3^b 5^c: N = A B
// with n = B a + b, k = k1 + A k2: DFT_A over a, times exp(-+2 pi i b k1 / N),
// DFT_B over b.
constexpr int dft_first(int n) { return n % 8 == 0 && n > 8 ? 8 : n % 4 == 0 ? 4 : n % 2 == 0 ? 2 : n % 3 == 0 ? 3 : 5; }

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
          t[b] = INV ? make_float2(s * (t[b].x - t[b].y), s * (t[b].x + t[b].y))
                     : make_float2(s * (t[b].x + t[b].y), s * (t[b].y - t[b].x));
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
    x[0] = make_float2(a.x + b.x, a.y + b.y);
    x[1] = make_float2(a.x - b.x, a.y - b.y);
  }
};
// X0 = a + s, X1,2 = a - s/2 -+ i (sqrt 3 / 2) d with s = b + c, d = b - c
template <bool INV>
struct Dft<INV, 3> {
  static __device__ __forceinline__ void run(float2 (&x)[3]) {
    constexpr float H = 0.86602540378443865f;   // sqrt(3) / 2
    const float2 a = x[0], b = x[1], c = x[2];
    const float2 s = make_float2(b.x + c.x, b.y + c.y), d = make_float2(b.x - c.x, b.y - c.y);
    const float2 t = make_float2(a.x - 0.5f * s.x, a.y - 0.5f * s.y);
    const float2 u = INV ? make_float2(-H * d.y, H * d.x) : make_float2(H * d.y, -H * d.x);
    x[0] = make_float2(a.x + s.x, a.y + s.y);
    x[1] = make_float2(t.x + u.x, t.y + u.y);
    x[2] = make_float2(t.x - u.x, t.y - u.y);
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
    const float2 p = make_float2(x[1].x + x[4].x, x[1].y + x[4].y), m = make_float2(x[1].x - x[4].x, x[1].y - x[4].y);
    const float2 q = make_float2(x[2].x + x[3].x, x[2].y + x[3].y), r = make_float2(x[2].x - x[3].x, x[2].y - x[3].y);
    const float2 u = make_float2(a.x + C1 * p.x + C2 * q.x, a.y + C1 * p.y + C2 * q.y);
    const float2 v = make_float2(a.x + C2 * p.x + C1 * q.x, a.y + C2 * p.y + C1 * q.y);
    const float2 g = make_float2(S1 * m.x + S2 * r.x, S1 * m.y + S2 * r.y);
    const float2 h = make_float2(S2 * m.x - S1 * r.x, S2 * m.y - S1 * r.y);
    const float2 ig = INV ? make_float2(-g.y, g.x) : make_float2(g.y, -g.x);     // -+i g
    const float2 ih = INV ? make_float2(-h.y, h.x) : make_float2(h.y, -h.x);
    x[0] = make_float2(a.x + p.x + q.x, a.y + p.y + q.y);
    x[1] = make_float2(u.x + ig.x, u.y + ig.y);
    x[4] = make_float2(u.x - ig.x, u.y - ig.y);
    x[2] = make_float2(v.x + ih.x, v.y + ih.y);
    x[3] = make_float2(v.x - ih.x, v.y - ih.y);
  }
};

}  // namespace ch
