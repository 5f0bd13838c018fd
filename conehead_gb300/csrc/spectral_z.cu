// z passes of the spectral cone stage at lengths L = 16 N2 (48 to 512).
//
// One beam's lines along z are real and zero from nz on, and the convolution
// needs L >= nz points only: modulo (z^L + i) the linear convolution's upper
// half wraps with a factor -i, so it lands in the imaginary part and the dose
// is the real part.  On the transform that is a twist: line value n times
// exp(-2 pi i n / (4 L)) before a complex DFT of length L, the conjugate after
// the inverse, and the real part.  (Two beams as real and imaginary part of
// one transform of 2 nz - 1 points cost the same; a beam on its own, or the
// last of an odd count, paid for two.  Five passes of one beam at 128^3: 108 ->
// 59 us, plane kernel 82 -> 43 us.)
//
// With n = N2 n1 + n2 and k = k1 + 16 k2 the twist splits into
// exp(-2 pi i n1 / 64), constants of the 16-point stage, and a factor of n2
// that joins the twiddle: exp(-2 pi i n2 (4 k1 + 1) / (4 L)).
//
// Lines along z are contiguous, so lanes run along z: thread (n2, line) with
// n2 fastest in the 16-point stages (consecutive z: TERMA reads and dose writes
// are coalesced).  The N2-point stages read or write A: [line][k] with k1
// fastest (128-byte runs), or plane-major [k][line] (PLANE) with the line
// fastest.  The exchange holds row 16 n2 + k1 of line c at c P + r + r / 16:
// consecutive k1 and consecutive n2 (17 slots apart) fall in 16 banks, and for
// PLANE, where lanes run across the lines, P is odd.

#include "spectral_16n.cuh"

namespace ch {

extern __shared__ float2 spec_sm[];

template <int N2, bool PLANE>
constexpr int z_pitch() { return 17 * N2 + ((PLANE && N2 % 2 == 0) ? 1 : 0); }
template <int N2, bool PLANE>
constexpr int z_smem() { return (16 * z_pitch<N2, PLANE>() + 16 * N2) * 8; }
template <int N2, bool PLANE>
__device__ __forceinline__ int zslot(int r, int c) { return c * z_pitch<N2, PLANE>() + r + (r >> 4); }

// cos and sin of 2 pi m / 64
struct Twist {
  float c[16] = {}, s[16] = {};
  constexpr Twist() {
    for (int m = 0; m < 16; ++m) {
      c[m] = (float)ct_cos(m, 64);
      s[m] = (float)ct_sin(m, 64);
    }
  }
};

template <int N2, bool PLANE>
__global__ void __launch_bounds__(r16n_threads<N2>(), r16n_ctas<N2>()) spec_z_forward_kernel(SpecLaunch P) {
  constexpr int L = 16 * N2, T = r16n_threads<N2>();
  float2* const xb = spec_sm;
  float2* const twb = spec_sm + 16 * z_pitch<N2, PLANE>();
  const SpecBeam& bm = P.p[blockIdx.y];
  const int nl = P.g.n[0] * P.g.n[1], nz = P.g.n[2];
  const int l0 = blockIdx.x * 16;
  after_trigger();
  // stage-1 twiddles exp(-2 pi i n2 (4 m + 1) / (4 L)) at m N2 + n2
  for (int i = threadIdx.x; i < L; i += T) twb[i] = __ldg(P.g.tq + (i % N2) * (4 * (i / N2) + 1));
  after_wait();
  // lines that may hold TERMA (the others are zero and are not read)
  __shared__ unsigned char zf[16];
  bool mine = false;
  if (threadIdx.x < 16) {
    const int l = l0 + threadIdx.x;
    mine = l < nl && (!bm.l || bm.l[l] != 0);
    zf[threadIdx.x] = mine;
  }
  if (!__syncthreads_or(mine)) {
    if (P.g.skip) return;
    // no TERMA on these lines: zeros, two values per 16-byte store
    if constexpr (PLANE) {
      for (int e = threadIdx.x; e < L * 8; e += T)
        *reinterpret_cast<float4*>(bm.a + (size_t)(e >> 3) * P.g.lp + l0 + (e & 7) * 2) =
            make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    } else {
      const int lines = min(16, nl - l0);
      float4* a4 = reinterpret_cast<float4*>(bm.a + (size_t)l0 * L);
      for (int e = threadIdx.x; e < lines * L / 2; e += T) a4[e] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    return;
  }
  if (threadIdx.x < 16 * N2) {
    constexpr Twist W{};
    const int n2 = threadIdx.x % N2, c = threadIdx.x / N2, l = l0 + c;
    const bool live = zf[c];
    const float* t = bm.t + (size_t)(l < nl ? l : 0) * P.g.zp;
    float2 v[16];
#pragma unroll
    for (int n1 = 0; n1 < 16; ++n1) {
      const int z = N2 * n1 + n2;
      v[n1].x = load_after(t + z, live && z < nz);
    }
#pragma unroll
    for (int n1 = 0; n1 < 16; ++n1) v[n1] = make_float2(v[n1].x * W.c[n1], -v[n1].x * W.s[n1]);
    dft16<false>(v);
    // X[m] of the DFT16 sits in v[4 (m mod 4) + m / 4]
#pragma unroll
    for (int m = 0; m < 16; ++m)
      xb[zslot<N2, PLANE>(16 * n2 + m, c)] = cmul(v[4 * (m & 3) + (m >> 2)], twb[m * N2 + n2]);
  }
  __syncthreads();
  if (threadIdx.x < 256) {
    const int lo = threadIdx.x & 15, hi = threadIdx.x >> 4;
    const int k1 = PLANE ? hi : lo, c = PLANE ? lo : hi, l = l0 + c;
    float2 a[N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2) a[n2] = xb[zslot<N2, PLANE>(16 * n2 + k1, c)];
    Dft<false, N2>::run(a);
    if (l < nl) {
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2) {
        const int k = k1 + 16 * k2;
        bm.a[PLANE ? (size_t)k * P.g.lp + l : (size_t)l * L + k] = a[k2];
      }
    }
  }
}

template <int N2, bool PLANE>
__global__ void __launch_bounds__(r16n_threads<N2>(), r16n_ctas<N2>()) spec_z_inverse_kernel(SpecLaunch P) {
  constexpr int L = 16 * N2, T = r16n_threads<N2>();
  float2* const xb = spec_sm;
  float2* const twb = spec_sm + 16 * z_pitch<N2, PLANE>();
  const SpecBeam& bm = P.p[blockIdx.y];
  const int nl = P.g.n[0] * P.g.n[1], nz = P.g.n[2];
  const int l0 = blockIdx.x * 16;
  after_trigger();
  // stage-A twiddles at 16 n2 + k1, one per thread
  static_assert(L <= T, "one table entry per thread");
  const int i_mine = min((int)threadIdx.x, L - 1);
  const float2 w_mine = __ldg(P.g.tq + (i_mine >> 4) * (4 * (i_mine & 15) + 1));
  after_wait();
  const int lo = threadIdx.x & 15, hi = threadIdx.x >> 4;
  float2 a[N2];
  if (threadIdx.x < 256) {
    const int k1 = PLANE ? hi : lo, c = PLANE ? lo : hi, l = l0 + c;
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) {
      const int k = k1 + 16 * k2;
      a[k2] = load_after(bm.a + (PLANE ? (size_t)k * P.g.lp + l : (size_t)l * L + k), l < nl);
    }
  }
  if (threadIdx.x < L) twb[threadIdx.x] = w_mine;
  __syncthreads();   // twiddle table
  if (threadIdx.x < 256) {
    const int k1 = PLANE ? hi : lo, c = PLANE ? lo : hi;
    Dft<true, N2>::run(a);
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2) {
      const float2 w = twb[16 * n2 + k1];
      xb[zslot<N2, PLANE>(16 * n2 + k1, c)] = cmul(a[n2], make_float2(w.x, -w.y));
    }
  }
  __syncthreads();
  if (threadIdx.x < 16 * N2) {
    constexpr Twist W{};
    const int n2 = threadIdx.x % N2, c = threadIdx.x / N2, l = l0 + c;
    float2 v[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = xb[zslot<N2, PLANE>(16 * n2 + q, c)];
    dft16<true>(v);
    if (l < nl) {
      float* d = bm.d + (size_t)l * nz;
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        const int z = n2 + N2 * m;
        const float2 y = v[4 * (m & 3) + (m >> 2)];
        if (z < nz) d[z] = y.x * W.c[m] - y.y * W.s[m];
      }
    }
  }
}

template <int N2, bool PLANE>
static cudaError_t z_setup() {
  cudaError_t e = cudaFuncSetAttribute(spec_z_forward_kernel<N2, PLANE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       z_smem<N2, PLANE>());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(spec_z_inverse_kernel<N2, PLANE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             z_smem<N2, PLANE>());
  return e;
}

cudaError_t setup_spec_z() {
  cudaError_t e = cudaSuccess;
#define Z_SETUP(N2) \
  if (e == cudaSuccess) e = z_setup<N2, false>(); \
  if (e == cudaSuccess) e = z_setup<N2, true>();
  SPEC_N2(Z_SETUP)
#undef Z_SETUP
  return e;
}

// The z pass of a launch; false when its length is not one of SPEC_N2's.
bool launch_spec_z(const SpecLaunch& L, bool inverse, cudaStream_t st) {
  const dim3 grid((L.g.n[0] * L.g.n[1] + 15) / 16, L.n_beams);
  switch (L.g.M[2]) {
#define Z_CASE(N2)                                                                                          \
  case 16 * N2:                                                                                             \
    if (L.g.plane && !inverse)                                                                              \
      launch_after(L.g.after, spec_z_forward_kernel<N2, true>, grid, r16n_threads<N2>(), z_smem<N2, true>(), st, L); \
    else if (L.g.plane)                                                                                     \
      launch_after(L.g.after, spec_z_inverse_kernel<N2, true>, grid, r16n_threads<N2>(), z_smem<N2, true>(), st, L); \
    else if (!inverse)                                                                                      \
      launch_after(L.g.after, spec_z_forward_kernel<N2, false>, grid, r16n_threads<N2>(), z_smem<N2, false>(), st, L); \
    else                                                                                                    \
      launch_after(L.g.after, spec_z_inverse_kernel<N2, false>, grid, r16n_threads<N2>(), z_smem<N2, false>(), st, L); \
    return true;
    SPEC_N2(Z_CASE)
#undef Z_CASE
  }
  return false;
}

}  // namespace ch
