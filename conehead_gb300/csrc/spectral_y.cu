// y passes of the spectral cone stage at periods M = 16 N2 (48 to 512), 16
// lines (consecutive kz, 128-byte rows) per CTA:
//   forward (A -> B), n = N2 n1 + n2, k = k1 + 16 k2:
//     stage 1, thread (c, n2): 16-point DFT over n1 (n1 < 8 nonzero: the
//       upper half of the padded input) of row N2 n1 + n2, times
//       exp(-2 pi i n2 k1 / M), out to shared memory row N2 k1 + n2;
//     stage 2, thread (c, k1): N2-point DFT over n2 -> rows k1 + 16 k2 of B;
//   inverse (B -> A), k = k1 + 16 k2, n = n2 + N2 n1:
//     stage A, thread (c, k1): N2-point DFT over k2 -> n2, times
//       exp(+2 pi i n2 k1 / M), out to shared memory row 16 n2 + k1;
//     stage B, thread (c, n2): 16-point DFT over k1 -> rows n2 + N2 n1,
//       n1 < 8, written where < ny.
// Rows of A whose line holds no TERMA are zero: the z pass does not write them and
// the forward pass does not read them (launch_spec_beams has the figures).
// A row of 16 lines is 128 bytes, one half-warp access: no swizzle is needed.

#include "spectral_16n.cuh"

namespace ch {

extern __shared__ float2 spec_sm[];

template <int N2>
constexpr int y_smem() { return (16 * N2 * 16 + 16 * N2) * 8; }

template <bool INV, int N2, bool AHEAD>
__global__ void __launch_bounds__(r16n_threads<N2>(), r16n_ctas<N2>()) spec_y_kernel(SpecLaunch P) {
  constexpr int M = 16 * N2, T = r16n_threads<N2>();
  float2* const xb = spec_sm;                 // exchange, row r at 16 r
  float2* const twb = spec_sm + M * 16;       // exp(-2 pi i k / M)
  const SpecBeam& bm = P.p[blockIdx.y];
  const int L = P.g.M[2], ny = P.g.n[1];
  const int nkb = L >> 4;
  const int x = blockIdx.x / nkb, kz0 = (blockIdx.x - x * nkb) << 4;
  const float2* const src = (INV ? bm.b + (size_t)x * M * L : bm.a + (size_t)x * ny * L) + kz0;
  float2* const dst = (INV ? bm.a + (size_t)x * ny * L : bm.b + (size_t)x * M * L) + kz0;
  const int c = threadIdx.x & 15, h = threadIdx.x >> 4;   // h: n2 (stages 1, B) or k1 (stages 2, A)
  static_assert(M <= T, "one table entry per thread");
  after_trigger();
  const float2 w_mine = __ldg(P.g.tw[1] + min((int)threadIdx.x, M - 1));
  after_wait();
  const unsigned char* const lines = !INV && P.g.skip && bm.l ? bm.l + x * ny : nullptr;
  if (AHEAD) {
    const unsigned next = blockIdx.x + SPEC_AHEAD;
    const int x2 = next / nkb, kz2 = (next - x2 * nkb) << 4, row = threadIdx.x;
    if (next < gridDim.x && row < (INV ? M : ny) && (!lines || bm.l[x2 * ny + row] != 0))
      prefetch_row((INV ? bm.b + ((size_t)x2 * M + row) * L : bm.a + ((size_t)x2 * ny + row) * L) + kz2);
  }
  // the inputs are in flight while the table is published
  float2 v[16], a[N2];
  if (!INV) {
    if (threadIdx.x < 16 * N2) {
#pragma unroll
      for (int n1 = 0; n1 < 8; ++n1) {
        const int y = N2 * n1 + h;
        v[n1] = load_after<(N2 > 12)>(src + (size_t)y * L + c, y < ny && (!lines || lines[y] != 0));
      }
    }
  } else if (threadIdx.x < 256) {
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) a[k2] = load_after<(N2 > 12)>(src + (size_t)(h + 16 * k2) * L + c, true);
  }
  if (threadIdx.x < M) twb[threadIdx.x] = w_mine;
  __syncthreads();   // twiddle table
  if (!INV) {
    if (threadIdx.x < 16 * N2) {
      // stage 1, thread (c, n2 = h)
      dft16_half_in<false>(v);
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        float2 t = v[4 * (m & 3) + (m >> 2)];
        if (m > 0) t = cmul(t, twb[h * m]);
        xb[(m * N2 + h) * 16 + c] = t;
      }
    }
    __syncthreads();
    if (threadIdx.x < 256) {
      // stage 2, thread (c, k1 = h)
#pragma unroll
      for (int n2 = 0; n2 < N2; ++n2) a[n2] = xb[(h * N2 + n2) * 16 + c];
      Dft<false, N2>::run(a);
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2) dst[(size_t)(h + 16 * k2) * L + c] = a[k2];
    }
  } else {
    if (threadIdx.x < 256) {
      // stage A, thread (c, k1 = h)
      Dft<true, N2>::run(a);
#pragma unroll
      for (int n2 = 0; n2 < N2; ++n2) {
        float2 t = a[n2];
        if (n2 > 0) {
          const float2 w = twb[n2 * h];
          t = cmul(t, make_float2(w.x, -w.y));
        }
        xb[(n2 * 16 + h) * 16 + c] = t;
      }
    }
    __syncthreads();
    if (threadIdx.x < 16 * N2) {
      // stage B, thread (c, n2 = h)
#pragma unroll
      for (int q = 0; q < 16; ++q) v[q] = xb[(h * 16 + q) * 16 + c];
      dft16<true>(v);
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        const int y = h + N2 * m;
        if (y < ny) dst[(size_t)y * L + c] = v[4 * (m & 3) + (m >> 2)];
      }
    }
  }
}

template <int N2>
static cudaError_t y_setup() {
  cudaError_t e = cudaSuccess;
  void (*const k[4])(SpecLaunch) = {spec_y_kernel<false, N2, false>, spec_y_kernel<false, N2, true>,
                                    spec_y_kernel<true, N2, false>, spec_y_kernel<true, N2, true>};
  for (auto f : k)
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, y_smem<N2>());
  return e;
}

cudaError_t setup_spec_y() {
  cudaError_t e = cudaSuccess;
#define Y_SETUP(N2) \
  if (e == cudaSuccess) e = y_setup<N2>();
  SPEC_N2(Y_SETUP)
#undef Y_SETUP
  return e;
}

// The y pass of a launch; false when its period is not one of SPEC_N2's.
bool launch_spec_y(const SpecLaunch& L, bool inverse, cudaStream_t st) {
  const dim3 grid(L.g.n[0] * (L.g.M[2] / 16), L.n_beams);
  switch (L.g.M[1]) {
#define Y_CASE(N2)                                                                                     \
  case 16 * N2:                                                                                        \
    launch_after(L.g.after,                                                                            \
                 inverse ? (L.g.ahead ? spec_y_kernel<true, N2, true> : spec_y_kernel<true, N2, false>) \
                         : (L.g.ahead ? spec_y_kernel<false, N2, true> : spec_y_kernel<false, N2, false>), \
                 grid, r16n_threads<N2>(), y_smem<N2>(), st, L);                                       \
    return true;
    SPEC_N2(Y_CASE)
#undef Y_CASE
  }
  return false;
}

}  // namespace ch
