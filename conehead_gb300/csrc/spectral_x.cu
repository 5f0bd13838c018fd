// x pass of the spectral cone stage at periods M = 16 N2 (48 to 512), and the
// forward transforms of full lines that build S^.
//
// x pass: 16 lines (consecutive kz) per CTA.  Forward (stages 1 and 2 of
// spectral_y.cu), the product with S^ and the inverse (stages A and B) chain in
// one kernel: stage 2, the product and stage A stay in the same thread's
// registers, two exchanges for the transform pair.  The CTA's M x 16 block of
// S^ is staged in shared memory by cp.async during stage 1; consecutive CTAs
// take the same lines of consecutive beams, so it comes from L2 after the first.

#include "spectral_16n.cuh"

namespace ch {

extern __shared__ float2 spec_sm[];

// exchange and S^ block, and up to N2 = 24 a twiddle table (432 x 16 without
// it leaves two CTAs per SM).  CTAs per SM: as many as shared memory and
// spill-free registers allow; measured against one more and one fewer, cone
// stage of 8 beams, fewer / this / more: 64^3 69.9 / 67.9 / 68 us, 144^3 715 /
// 671 us / (no room), 160^3 924 / 971 us at 3 CTAs of N2 = 20.  Without the
// staged S^ block (read through L2 in stage 2): 160^3 842 -> 1072-1184 us.
template <int N2>
constexpr bool x_table() { return N2 <= 24; }
template <int N2>
constexpr int x_smem() { return (2 * 16 * N2 * 16 + (x_table<N2>() ? 16 * N2 : 0)) * 8; }
template <int N2>
constexpr int x_ctas() { return N2 <= 10 ? 5 : N2 <= 12 ? 4 : N2 <= 18 ? 3 : 2; }

template <int N2, bool AHEAD>
__global__ void __launch_bounds__(r16n_threads<N2>(), x_ctas<N2>()) spec_x_kernel(SpecLaunch P) {
  constexpr int M = 16 * N2, T = r16n_threads<N2>();
  float2* const xb = spec_sm;                 // exchange, row r at 16 r
  float2* const sb = spec_sm + M * 16;        // S^ block, row kx at 16 kx
  float2* const twb = spec_sm + 2 * M * 16;   // exp(-2 pi i k / M)
  const int beam = blockIdx.x % P.n_beams, blk = blockIdx.x / P.n_beams;
  const int My = P.g.M[1], L = P.g.M[2];
  const int nkb = L >> 4;
  const int ky = blk / nkb, kz0 = (blk - ky * nkb) << 4;
  const size_t xs = (size_t)My * L, off = (size_t)ky * L + kz0;
  float2* const b = P.p[beam].b + off;
  const int nx = P.g.n[0];
  const int c = threadIdx.x & 15, h = threadIdx.x >> 4;   // h: n2 (stages 1, B) or k1 (stages 2, A)
  after_trigger();
  {
    // S^ rows of the CTA's 16 lines: M x 128 bytes, 16 bytes per copy
    const float2* sh = P.g.shat + off;
    for (int e = threadIdx.x; e < 8 * M; e += T) {
      const int i = e >> 3, cp = (e & 7) * 2;
      const unsigned d = (unsigned)__cvta_generic_to_shared(sb + i * 16 + cp);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(sh + (size_t)i * xs + cp));
    }
    asm volatile("cp.async.commit_group;\n" ::);
  }
  static_assert(M <= T, "one table entry per thread");
  const float2 w_mine = x_table<N2>() ? __ldg(P.g.tw[0] + min((int)threadIdx.x, M - 1)) : make_float2(0.0f, 0.0f);
  after_wait();   // S^ and the twiddles are older than any kernel of this call
  if (AHEAD) {
    const unsigned next = blockIdx.x + SPEC_AHEAD;
    if (next < gridDim.x && (int)threadIdx.x < nx) {
      const int blk2 = next / P.n_beams, ky2 = blk2 / nkb, kz2 = (blk2 - ky2 * nkb) << 4;
      prefetch_row(P.p[next - blk2 * P.n_beams].b + (size_t)ky2 * L + kz2 + threadIdx.x * xs);
    }
  }
  float2 v[16];
  if (threadIdx.x < 16 * N2) {
#pragma unroll
    for (int n1 = 0; n1 < 8; ++n1) {
      const int x = N2 * n1 + h;
      v[n1] = load_after<(N2 > 12)>(b + (size_t)x * xs + c, x < nx);
    }
  }
  auto tw = [&](int i) { return x_table<N2>() ? twb[i] : __ldg(P.g.tw[0] + i); };
  if (x_table<N2>()) {
    if (threadIdx.x < M) twb[threadIdx.x] = w_mine;
    __syncthreads();   // twiddle table
  }
  if (threadIdx.x < 16 * N2) {
    // forward stage 1, thread (c, n2 = h): rows N2 n1 + n2, n1 < 8
    dft16_half_in<false>(v);
    // X[m] of the DFT16 sits in v[4 (m mod 4) + m / 4]
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      float2 y = v[4 * (m & 3) + (m >> 2)];
      if (m > 0) y = cmul(y, tw(h * m));
      xb[(m * N2 + h) * 16 + c] = y;
    }
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();   // exchange written, S^ landed
  float2 a[N2];
  if (threadIdx.x < 256) {
    // forward stage 2, thread (c, k1 = h); the product; inverse stage A
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2) a[n2] = xb[(h * N2 + n2) * 16 + c];
    Dft<false, N2>::run(a);
    const float cs = P.g.conj ? -1.0f : 1.0f;
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) {
      const float2 sv = sb[(h + 16 * k2) * 16 + c];
      a[k2] = cmul(a[k2], make_float2(sv.x, cs * sv.y));
    }
    Dft<true, N2>::run(a);
  }
  __syncthreads();   // every read of the exchange done
  if (threadIdx.x < 256) {
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2) {
      float2 y = a[n2];
      if (n2 > 0) {
        const float2 w = tw(n2 * h);
        y = cmul(y, make_float2(w.x, -w.y));
      }
      xb[(n2 * 16 + h) * 16 + c] = y;
    }
  }
  __syncthreads();
  if (threadIdx.x < 16 * N2) {
    // inverse stage B, thread (c, n2 = h): rows n2 + N2 n1
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = xb[(h * 16 + q) * 16 + c];
    dft16<true>(v);
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const int x = h + N2 * m;
      if (x < nx) b[(size_t)x * xs + c] = v[4 * (m & 3) + (m >> 2)];
    }
  }
}

// Forward transform of full lines in place (S^): element i of line (o, c),
// c < 16, at o1 os1 + o2 os2 + c cs + i is with o = o1 nb + o2; the z axis
// multiplies by the twist first (spectral_z.cu).  Lanes run along whichever of
// line and element is contiguous, with the exchange of the y or of the z passes
// (lanes across the lines of the z axis read 8 bytes of every 32: 201^3 364 -> 138 us).
template <int N2>
__global__ void __launch_bounds__(r16n_threads<N2>(), 1) spec_full_kernel(SpecFull F) {
  float2* const xb = spec_sm;
  const int t = threadIdx.x;
  const bool along = F.is == 1;
  const int o1 = blockIdx.x / F.nb, o2 = blockIdx.x - o1 * F.nb;
  float2* const data = F.data + (size_t)o1 * F.os1 + (size_t)o2 * F.os2;
  // slot of row (n2, k1) of line c
  const int sc = along ? 17 * N2 : 1, sn = along ? 17 : 16, sk = along ? 1 : 16 * N2;
  if (t < 16 * N2) {
    const int n2 = along ? t % N2 : t >> 4, c = along ? t / N2 : t & 15;
    const float2* const line = data + (size_t)c * F.cs;
    float2 v[16];
#pragma unroll
    for (int n1 = 0; n1 < 16; ++n1) {
      const int i = N2 * n1 + n2;
      v[n1] = line[(size_t)i * F.is];
      if (F.tq) v[n1] = cmul(v[n1], __ldg(F.tq + i));
    }
    dft16<false>(v);
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      float2 y = v[4 * (m & 3) + (m >> 2)];
      if (m > 0) y = cmul(y, __ldg(F.tw + n2 * m));
      xb[m * sk + n2 * sn + c * sc] = y;
    }
  }
  __syncthreads();
  if (t < 256) {
    const int k1 = along ? t & 15 : t >> 4, c = along ? t >> 4 : t & 15;
    float2* const line = data + (size_t)c * F.cs;
    float2 a[N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2) a[n2] = xb[k1 * sk + n2 * sn + c * sc];
    Dft<false, N2>::run(a);
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) line[(size_t)(k1 + 16 * k2) * F.is] = a[k2];
  }
}

template <int N2>
constexpr int full_smem() { return 16 * 17 * N2 * 8; }

template <int N2>
static cudaError_t x_setup() {
  cudaError_t e = cudaFuncSetAttribute(spec_x_kernel<N2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, x_smem<N2>());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(spec_x_kernel<N2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, x_smem<N2>());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(spec_full_kernel<N2>, cudaFuncAttributeMaxDynamicSharedMemorySize, full_smem<N2>());
  return e;
}

cudaError_t setup_spec_x() {
  cudaError_t e = cudaSuccess;
#define X_SETUP(N2) \
  if (e == cudaSuccess) e = x_setup<N2>();
  SPEC_N2(X_SETUP)
#undef X_SETUP
  return e;
}

// The x pass of a launch; false when its period is not one of SPEC_N2's.
bool launch_spec_x(const SpecLaunch& L, cudaStream_t st) {
  const unsigned grid = (unsigned)(L.g.M[1] * (L.g.M[2] / 16) * L.n_beams);
  switch (L.g.M[0]) {
#define X_CASE(N2)                                                                  \
  case 16 * N2:                                                                     \
    launch_after(L.g.after, L.g.ahead ? spec_x_kernel<N2, true> : spec_x_kernel<N2, false>, grid, r16n_threads<N2>(), \
                 x_smem<N2>(), st, L);                                              \
    return true;
    SPEC_N2(X_CASE)
#undef X_CASE
  }
  return false;
}

bool launch_spec_full(const SpecFull& F, int M, unsigned blocks, cudaStream_t st) {
  switch (M) {
#define F_CASE(N2)                                                                  \
  case 16 * N2:                                                                     \
    spec_full_kernel<N2><<<blocks, r16n_threads<N2>(), full_smem<N2>(), st>>>(F);  \
    return true;
    SPEC_N2(F_CASE)
#undef F_CASE
  }
  return false;
}

}  // namespace ch
