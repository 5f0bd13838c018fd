// Collapsed-cone stage as a spectral convolution (replaces the per-voxel
// scatter of conehead/conehead.py:385-488 by the same linear operator).
//
// Every walk from a voxel centre visits the same offsets O_u[m] with the same
// weights w_u[m], so the cone stage is one linear convolution with a fixed
// stencil:
//     dose(v) = sum_s T(s) S(v - s),   S(o) = sum_u sum_m w_u[m] [O_u[m] = o].
// Walks stop where they leave the grid, i.e. only |o_k| <= n_k - 1 connects
// two voxels of the grid, so along x and y a circular convolution of period
// M_k >= 2 n_k - 1 equals the linear one on the grid.  Along z, where TERMA and
// dose are real, the convolution is taken modulo (z^L + i) with L >= nz: what
// wraps lands in the imaginary part (spectral_z.cu).  So
//     dose = Re IFFT( FFT(T) . S^ ),   S^ = FFT(S) / (Mx My L),
// each transform twisted along z, S^ computed once per grid shape and kernel.
//
// The five passes over a beam are batches of 1-D FFTs along one axis:
//   z forward  TERMA [nx][ny][nz] (pitch zp)       -> A [nx][ny][L]
//   y forward  A (y < ny)                          -> B [nx][My][L]
//   x          B (x < nx): forward, times S^, inverse, x < nx kept (in place)
//   y inverse  B                                   -> A (y < ny)
//   z inverse  A                                   -> dose [nx][ny][nz]
// They skip the zero padding, and every global sweep is coalesced: lines along
// z are read and written along z, lines along y and x are taken in blocks of
// consecutive kz.  Lengths of 48 to 512 that are 16 N2 for an N2 of SPEC_N2
// take the kernels of spectral_z.cu, spectral_y.cu and spectral_x.cu; longer
// ones (2^a, 3 * 2^a) the general kernels here.  With periods of 256 along x
// and y the y and x passes run as one kernel per kz plane (spec_plane_kernel).
//
// General kernels: a CTA holds up to 4096 complex values (L lines, L the
// largest power of two with L M <= 4096) in shared memory, element (i, line c)
// at i * L + (c ^ (i mod L)) so that both line-major and index-major sweeps are
// free of bank conflicts, and runs Stockham stages of radix 16, 3, 4 and 2 with
// twiddles from a host-built table.

#include <algorithm>
#include <cmath>
#include <vector>

#include "spectral_16n.cuh"

namespace ch {

__device__ __forceinline__ int swz(int i, int c, int L) { return i * L + (c ^ (i & (L - 1))); }

// One Stockham stage from src to dst (element (i, line c) layout above) on L
// lines of period M; Ns is the product of the radices done so far, tw[k] =
// exp(-2 pi i k / M).  Butterfly j of a line reads j + r M/R, multiplies by
// tw[r k M/(Ns R)] with k = j mod Ns, and writes (j - k) R + k + r Ns.  A
// thread takes one butterfly at a time.
// hin: the first stage of a transform whose input's upper half is zero (it
// reads only r < 8); hout: the last stage of one whose output's upper half
// is not wanted (it writes only the lower half).
template <bool INV>
__device__ __forceinline__ void stage16(const float2* src, float2* dst, int M, int L, int logL, int Ns,
                                        const float2* __restrict__ tw, bool hin, bool hout) {
  const int MR = M / 16, nb = L * MR, step = M / (Ns * 16);
  for (int bf = threadIdx.x; bf < nb; bf += SPEC_THREADS) {
    const int c = bf & (L - 1), j = bf >> logL, k = j % Ns;
    float2 v[16];
    if (hin) {
#pragma unroll
      for (int r = 0; r < 8; ++r) v[r] = src[swz(j + r * MR, c, L)];
      dft16_half_in<INV>(v);     // first stage: k = 0, no twiddles
      const int o = j << 4;
#pragma unroll
      for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
        for (int k2 = 0; k2 < 4; ++k2) dst[swz(o + (k1 + 4 * k2) * Ns, c, L)] = v[4 * k1 + k2];
      continue;
    }
#pragma unroll
    for (int r = 0; r < 16; ++r) v[r] = src[swz(j + r * MR, c, L)];
    if (k) {
#pragma unroll
      for (int r = 1; r < 16; ++r) {
        float2 w = __ldg(tw + r * k * step);
        if (INV) w.y = -w.y;
        v[r] = cmul(v[r], w);
      }
    }
    dft16<INV>(v);
    const int o = (j - k) * 16 + k;
    if (hout) {
      // outputs o + q Ns with q = k1 + 4 k2 < 8 are the lower half
#pragma unroll
      for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
        for (int k2 = 0; k2 < 2; ++k2) dst[swz(o + (k1 + 4 * k2) * Ns, c, L)] = v[4 * k1 + k2];
    } else {
#pragma unroll
      for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
        for (int k2 = 0; k2 < 4; ++k2) dst[swz(o + (k1 + 4 * k2) * Ns, c, L)] = v[4 * k1 + k2];
    }
  }
}

template <bool INV>
__device__ __forceinline__ void stage3(const float2* src, float2* dst, int M, int L, int logL, int Ns,
                                       const float2* __restrict__ tw) {
  const int MR = M / 3, nb = L * MR, step = M / (Ns * 3);
  for (int bf = threadIdx.x; bf < nb; bf += SPEC_THREADS) {
    const int c = bf & (L - 1), j = bf >> logL, k = j % Ns;
    float2 v0 = src[swz(j, c, L)], v1 = src[swz(j + MR, c, L)], v2 = src[swz(j + 2 * MR, c, L)];
    float2 w1 = __ldg(tw + k * step), w2 = __ldg(tw + 2 * k * step);
    if (INV) {
      w1.y = -w1.y;
      w2.y = -w2.y;
    }
    v1 = cmul(v1, w1);
    v2 = cmul(v2, w2);
    float2 v[3] = {v0, v1, v2};
    Dft<INV, 3>::run(v);
    const int o = (j - k) * 3 + k;
    dst[swz(o, c, L)] = v[0];
    dst[swz(o + Ns, c, L)] = v[1];
    dst[swz(o + 2 * Ns, c, L)] = v[2];
  }
}

template <bool INV>
__device__ __forceinline__ void stage4(const float2* src, float2* dst, int M, int L, int logL, int Ns,
                                       const float2* __restrict__ tw, bool hout) {
  const int MR = M / 4, nb = L * MR, step = M / (Ns * 4);
  for (int bf = threadIdx.x; bf < nb; bf += SPEC_THREADS) {
    const int c = bf & (L - 1), j = bf >> logL, k = j % Ns;
    float2 v[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) v[r] = src[swz(j + r * MR, c, L)];
#pragma unroll
    for (int r = 1; r < 4; ++r) {
      float2 w = __ldg(tw + r * k * step);
      if (INV) w.y = -w.y;
      v[r] = cmul(v[r], w);
    }
    dft4<INV>(v[0], v[1], v[2], v[3]);
    const int o = (j - k) * 4 + k;
    if (hout) {
      dst[swz(o, c, L)] = v[0];
      dst[swz(o + Ns, c, L)] = v[1];
    } else {
#pragma unroll
      for (int r = 0; r < 4; ++r) dst[swz(o + r * Ns, c, L)] = v[r];
    }
  }
}

template <bool INV>
__device__ __forceinline__ void stage2(const float2* src, float2* dst, int M, int L, int logL, int Ns,
                                       const float2* __restrict__ tw, bool hout) {
  const int MR = M / 2, nb = L * MR, step = M / (Ns * 2);
  for (int bf = threadIdx.x; bf < nb; bf += SPEC_THREADS) {
    const int c = bf & (L - 1), j = bf >> logL, k = j % Ns;
    float2 w = __ldg(tw + k * step);
    if (INV) w.y = -w.y;
    const float2 a0 = src[swz(j, c, L)], a1 = cmul(src[swz(j + MR, c, L)], w);
    const int o = (j - k) * 2 + k;
    dst[swz(o, c, L)] = make_float2(a0.x + a1.x, a0.y + a1.y);
    if (!hout) dst[swz(o + Ns, c, L)] = make_float2(a0.x - a1.x, a0.y - a1.y);
  }
}

// FFT of the L lines of period M (2^a or 3 * 2^a, a >= 4) held in src,
// ping-ponging with dst; returns the buffer holding the result.  INV uses
// the conjugate twiddles (no 1/M scale).  Stages: radix 16, then radix 3 for
// a period with a factor 3, then radix 16 while four or more factors of two
// remain, then radix 4 and 2; every stage ends with one barrier.  The caller
// has synchronised after filling src.  half_in: the input's upper half is
// zero; half_out: only the output's lower half is wanted (the upper half of
// the result buffer is then left stale).
template <bool INV>
__device__ __forceinline__ float2* fft_block(float2* src, float2* dst, int M, int logL,
                                             const float2* __restrict__ tw, bool half_in, bool half_out) {
  const int L = 1 << logL;
  const int a = __ffs(M) - 1;
  const bool three = (M >> a) == 3;
  int twos = a - 4, Ns = 16;
  auto next = [&] {
    __syncthreads();
    float2* t = src;
    src = dst;
    dst = t;
  };
  stage16<INV>(src, dst, M, L, logL, 1, tw, half_in, half_out && M == 16);
  next();
  if (three) {
    stage3<INV>(src, dst, M, L, logL, Ns, tw);
    next();
    Ns *= 3;
  }
  while (twos >= 4) {
    stage16<INV>(src, dst, M, L, logL, Ns, tw, false, half_out && twos == 4);
    next();
    Ns *= 16;
    twos -= 4;
  }
  if (twos >= 2) {
    stage4<INV>(src, dst, M, L, logL, Ns, tw, half_out && twos == 2);
    next();
    Ns *= 4;
    twos -= 2;
  }
  if (twos >= 1) {
    stage2<INV>(src, dst, M, L, logL, Ns, tw, half_out);
    next();
  }
  return src;
}

// ------------------------------------------------- line block transfers --
// L lines of a pass along y or x: element (i, c) at base + i * stride + c
// (the lines are L consecutive kz).  Two adjacent lines move in one 16-byte
// access (stride, base and c are even); every load of a thread is issued
// before its shared-memory stores.  Rows i >= n are zero (the padding).
__device__ __forceinline__ void load_lines(const float2* __restrict__ base, size_t stride, int n, int M, int L,
                                           int logL, float2* sm) {
  if (L >= 2) {
    float4 v[SPEC_ELEMS / SPEC_THREADS / 2];
#pragma unroll
    for (int q = 0; q < SPEC_ELEMS / SPEC_THREADS / 2; ++q) {
      const int e = threadIdx.x + q * SPEC_THREADS;
      const int c = (e & (L / 2 - 1)) * 2, i = e >> (logL - 1);
      v[q] = i < n ? __ldg(reinterpret_cast<const float4*>(base + (size_t)i * stride + c))
                   : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
#pragma unroll
    for (int q = 0; q < SPEC_ELEMS / SPEC_THREADS / 2; ++q) {
      const int e = threadIdx.x + q * SPEC_THREADS;
      const int c = (e & (L / 2 - 1)) * 2, i = e >> (logL - 1);
      if (i < M) {
        sm[swz(i, c, L)] = make_float2(v[q].x, v[q].y);
        sm[swz(i, c + 1, L)] = make_float2(v[q].z, v[q].w);
      }
    }
  } else {
    for (int i = threadIdx.x; i < M; i += SPEC_THREADS)
      sm[swz(i, 0, L)] = i < n ? base[(size_t)i * stride] : make_float2(0.0f, 0.0f);
  }
}

__device__ __forceinline__ void store_lines(const float2* res, float2* __restrict__ base, size_t stride, int n,
                                            int L, int logL) {
  if (L >= 2) {
    for (int e = threadIdx.x; e < n * L / 2; e += SPEC_THREADS) {
      const int c = (e & (L / 2 - 1)) * 2, i = e >> (logL - 1);
      const float2 a = res[swz(i, c, L)], b = res[swz(i, c + 1, L)];
      *reinterpret_cast<float4*>(base + (size_t)i * stride + c) = make_float4(a.x, a.y, b.x, b.y);
    }
  } else {
    for (int i = threadIdx.x; i < n; i += SPEC_THREADS) base[(size_t)i * stride] = res[swz(i, 0, L)];
  }
}

// --------------------------------------------------------- general passes --
// The period and log2 of the lines per CTA are read from the launch (P.g.M and
// P.g.logL): the largest power of two L with L M <= 4096 for lines along z;
// lines along y and x are taken in blocks of L consecutive kz, so L also
// divides Mz.
extern __shared__ float2 spec_sm[];

// z forward: lines (x, y), TERMA in, times the twist, A out.
__global__ void __launch_bounds__(SPEC_THREADS, SPEC_CTAS_PER_SM) spec_z_forward_general_kernel(SpecLaunch P) {
  float2* sm = spec_sm;
  float2* sm2 = spec_sm + SPEC_ELEMS;
  const SpecBeam& bm = P.p[blockIdx.y];
  const int Mz = P.g.M[2], logL = P.g.logL[2], L = 1 << logL;
  const int nl = P.g.n[0] * P.g.n[1], nz = P.g.n[2], l0 = blockIdx.x * L;
  auto store = [&](int l, int i, float2 v) { bm.a[P.g.plane ? (size_t)i * P.g.lp + l : (size_t)l * Mz + i] = v; };
  // lines that may hold TERMA (the others are zero and are not read); a block
  // without any transforms to zero
  __shared__ unsigned char zf[SPEC_ELEMS / SPEC_MIN_GENERAL];
  bool mine = false;
  if (threadIdx.x < L) {
    const int l = l0 + threadIdx.x;
    mine = l < nl && (!bm.l || __ldg(bm.l + l) != 0);
    zf[threadIdx.x] = mine;
  }
  if (!__syncthreads_or(mine)) {
    for (int e = threadIdx.x; e < L * Mz; e += SPEC_THREADS) {
      const int l = l0 + e / Mz;
      if (l < nl) store(l, e % Mz, make_float2(0.0f, 0.0f));
    }
    return;
  }
  for (int e = threadIdx.x; e < L * Mz; e += SPEC_THREADS) {
    const int c = e / Mz, i = e - c * Mz, l = l0 + c;
    const float x = (zf[c] && i < nz) ? __ldg(bm.t + (size_t)l * P.g.zp + i) : 0.0f;
    const float2 w = __ldg(P.g.tq + i);
    sm[swz(i, c, L)] = make_float2(x * w.x, x * w.y);
  }
  __syncthreads();
  const float2* res = fft_block<false>(sm, sm2, Mz, logL, P.g.tw[2], false, false);
  for (int e = threadIdx.x; e < L * Mz; e += SPEC_THREADS) {
    const int c = e / Mz, i = e - c * Mz, l = l0 + c;
    if (l < nl) store(l, i, res[swz(i, c, L)]);
  }
}

// z inverse: lines (x, y), A in, times the conjugate twist, real part out.
__global__ void __launch_bounds__(SPEC_THREADS, SPEC_CTAS_PER_SM) spec_z_inverse_general_kernel(SpecLaunch P) {
  float2* sm = spec_sm;
  float2* sm2 = spec_sm + SPEC_ELEMS;
  const SpecBeam& bm = P.p[blockIdx.y];
  const int Mz = P.g.M[2], logL = P.g.logL[2], L = 1 << logL;
  const int nl = P.g.n[0] * P.g.n[1], nz = P.g.n[2], l0 = blockIdx.x * L;
  for (int e = threadIdx.x; e < L * Mz; e += SPEC_THREADS) {
    const int c = e / Mz, i = e - c * Mz, l = l0 + c;
    sm[swz(i, c, L)] =
        l < nl ? bm.a[P.g.plane ? (size_t)i * P.g.lp + l : (size_t)l * Mz + i] : make_float2(0.0f, 0.0f);
  }
  __syncthreads();
  const float2* res = fft_block<true>(sm, sm2, Mz, logL, P.g.tw[2], false, false);
  for (int e = threadIdx.x; e < L * Mz; e += SPEC_THREADS) {
    const int c = e / Mz, i = e - c * Mz, l = l0 + c;
    if (l < nl && i < nz) {
      const float2 v = res[swz(i, c, L)], w = __ldg(P.g.tq + i);
      bm.d[(size_t)l * nz + i] = v.x * w.x + v.y * w.y;
    }
  }
}

// y forward (A -> B) or inverse (B -> A): lines (x, kz) in blocks of L kz.
template <bool INV>
__global__ void __launch_bounds__(SPEC_THREADS, SPEC_CTAS_PER_SM) spec_y_general_kernel(SpecLaunch P) {
  float2* sm = spec_sm;
  float2* sm2 = spec_sm + SPEC_ELEMS;
  const SpecBeam& bm = P.p[blockIdx.y];
  const int My = P.g.M[1], Mz = P.g.M[2];
  const int logL = P.g.logL[1], L = 1 << logL;
  const int nkb = Mz >> logL;
  const int x = blockIdx.x / nkb, kz0 = (blockIdx.x - x * nkb) << logL;
  const int ny = P.g.n[1];
  const int n_in = INV ? My : ny, n_out = INV ? ny : My;
  const float2* src = INV ? bm.b + (size_t)x * My * Mz : bm.a + (size_t)x * ny * Mz;
  float2* dst = INV ? bm.a + (size_t)x * ny * Mz : bm.b + (size_t)x * My * Mz;
  load_lines(src + kz0, Mz, n_in, My, L, logL, sm);
  __syncthreads();
  const float2* res = fft_block<INV>(sm, sm2, My, logL, P.g.tw[1], !INV, INV);
  store_lines(res, dst + kz0, Mz, n_out, L, logL);
}

// x pass on B, lines (ky, kz) in blocks of L kz: forward, times S^ (or its
// conjugate), inverse, x < nx kept.
__global__ void __launch_bounds__(SPEC_THREADS, SPEC_CTAS_PER_SM) spec_x_general_kernel(SpecLaunch P) {
  float2* sm = spec_sm;
  float2* sm2 = spec_sm + SPEC_ELEMS;
  const int beam = blockIdx.x % P.n_beams, blk = blockIdx.x / P.n_beams;
  const int Mx = P.g.M[0], My = P.g.M[1], Mz = P.g.M[2];
  const int logL = P.g.logL[0], L = 1 << logL;
  const int nkb = Mz >> logL;
  const int ky = blk / nkb, kz0 = (blk - ky * nkb) << logL;
  const size_t xs = (size_t)My * Mz, off = (size_t)ky * Mz + kz0;
  float2* b = P.p[beam].b + off;
  const int nx = P.g.n[0];
  load_lines(b, xs, nx, Mx, L, logL, sm);
  __syncthreads();
  float2* res = fft_block<false>(sm, sm2, Mx, logL, P.g.tw[0], true, false);
  const float2* sh = P.g.shat + off;
  for (int e = threadIdx.x; e < L * Mx; e += SPEC_THREADS) {
    float2 s = __ldg(sh + (size_t)(e >> logL) * xs + (e & (L - 1)));
    if (P.g.conj) s.y = -s.y;
    const int k = swz(e >> logL, e & (L - 1), L);
    res[k] = cmul(res[k], s);
  }
  __syncthreads();
  res = fft_block<true>(res, res == sm ? sm2 : sm, Mx, logL, P.g.tw[0], false, true);
  store_lines(res, b, xs, nx, L, logL);
}

// Forward transform of full lines in place (S^), one CTA per line.
__global__ void __launch_bounds__(SPEC_THREADS, SPEC_CTAS_PER_SM) spec_full_general_kernel(SpecFull F, int M) {
  const int o1 = blockIdx.x / F.nb, o2 = blockIdx.x - o1 * F.nb;
  float2* const line = F.data + (size_t)o1 * F.os1 + (size_t)o2 * F.os2 + (size_t)blockIdx.y * F.cs;
  for (int i = threadIdx.x; i < M; i += SPEC_THREADS) {
    float2 v = line[(size_t)i * F.is];
    if (F.tq) v = cmul(v, __ldg(F.tq + i));
    spec_sm[i] = v;
  }
  __syncthreads();
  const float2* res = fft_block<false>(spec_sm, spec_sm + SPEC_ELEMS, M, 0, F.tw, false, false);
  for (int i = threadIdx.x; i < M; i += SPEC_THREADS) line[(size_t)i * F.is] = res[i];
}

// ------------------------------------------------------------ plane path --
// Periods of 256 along x and y.  The y and x transforms of one kz plane (with
// the S^ product and both inverses) run in one kernel on the plane's spectrum
// held on chip, so the intermediate B [nx][My][L] of the five-pass path never
// reaches memory; A is laid out plane-major, A[kz][l] with l = x ny + y and
// plane pitch lp, so a plane is one contiguous block.
//
// Helpers: one warp transforms two lines of 256 (lanes
// 0-15 the first, 16-31 the second; lane j of a line holds butterfly j) with
// an exchange buffer of its own, so only __syncwarp orders the two stages.
// A 64-bit shared access is served per half warp, i.e. per line here: each
// line has its own 256 elements, element i at i ^ ((i / 16) mod 16), so that
// the stage-1 writes (rows 16 j + q) and the stage-2 reads (rows j + 16 r)
// of a line's 16 lanes fall in 16 different banks.
__device__ __forceinline__ int wx(int i, int c) { return c * 256 + (i ^ ((i >> 4) & 15)); }

template <bool INV>
__device__ __forceinline__ void w16_first(float2 (&v)[16], bool hin, float2* wb, int j, int c) {
  if (hin)
    dft16_half_in<INV>(v);
  else
    dft16<INV>(v);
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) wb[wx(16 * j + k1 + 4 * k2, c)] = v[4 * k1 + k2];
}

// stage 2 with the twiddles exp(-2 pi i r j / 256), r = 0..15, of butterfly
// j from a shared table row twj = tws + 18 j (rows padded to 144 bytes), two
// twiddles per 16-byte load: the 16 lanes of a line then read 8 distinct
// 16-byte bank groups, two wavefronts, the minimum for 256 bytes (every
// transform of the plane kernel has period 256)
constexpr int PLANE_TW_ROW = 18;
template <bool INV>
__device__ __forceinline__ void w16_second(const float2* wb, float2 (&v)[16], int j, int c, const float2* twj) {
#pragma unroll
  for (int r = 0; r < 16; ++r) v[r] = wb[wx(j + 16 * r, c)];
  const float4* tw4 = reinterpret_cast<const float4*>(twj);
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    const float4 t = tw4[m];
    if (m > 0) v[2 * m] = cmul(v[2 * m], make_float2(t.x, INV ? -t.y : t.y));
    v[2 * m + 1] = cmul(v[2 * m + 1], make_float2(t.z, INV ? -t.w : t.w));
  }
  dft16<INV>(v);
}

// distributed shared memory: the partner CTA's copy of a shared address
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"((uint32_t)__cvta_generic_to_shared(p)),
               "r"(rank));
  return out;
}
__device__ __forceinline__ void st_cluster(uint32_t a, float2 v) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ float2 ld_cluster(uint32_t a) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
  return v;
}
// split cluster barrier: release/acquire where one CTA reads what the other
// wrote, relaxed where it only orders running and exiting
__device__ __forceinline__ void cluster_arrive_release() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_arrive_relaxed() {
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

// One kz plane of one beam per cluster of two CTAs.  CTA r of the
// cluster holds the ky in [128 r, 128 r + 128) of the plane's spectrum,
// Y[x][ky - 128 r] (x < nx <= 128; 128 KB), in its shared memory, element
// (x, k) at x * 128 + (k ^ (x mod 16)) so that a row (lanes along ky) and a
// column (lanes along x) are both conflict-free:
//   1. y forward: CTA r transforms rows x in [64 r, 64 r + 64) of A (y < ny,
//      the upper half zero; rows without TERMA skip the transform) and stores each output ky into the CTA that holds it (its
//      own shared memory or its partner's);
//   2. per ky column of its half: x forward (x < nx), times S^[kz][ky][kx]
//      (or its conjugate), x inverse (x < nx kept), in place;
//   3. y inverse of its rows: the 256 ky of a row come half from each CTA;
//      rows y < ny go back to A.
// Every warp owns two lines at a time (rows in 1 and 3, columns in 2) with
// its own exchange buffer, so warps never wait for each other inside a
// phase.  The next pair's rows of A (phase 1) are loaded while the current
// pair transforms, the S^ values of a column pair while its forward
// transform runs.  Cluster barriers start the kernel (the partner is
// running before its shared memory is written; waited on just before the
// first stores), separate the phases (release/acquire) and end it (the
// partner has read this CTA's half before it exits); every thread reaches
// each of them once.  Consecutive clusters take the same kz of consecutive
// beams, so that plane of S^ comes from L2 after the first.
constexpr int PLANE_THREADS = 512;
constexpr int PLANE_WARPS = PLANE_THREADS / 32;
static_assert(SPEC_PLANE_SMEM >= (128 * 128 + PLANE_WARPS * 2 * 256 + 16 * PLANE_TW_ROW) * 8,
              "plane kernel shared memory");

template <int R>
__device__ __forceinline__ void plane_store_rows(float2* Y, uint32_t peer, int x, int jx, const float2 (&v)[16]) {
  // outputs ky = j + 16 q, q = k1 + 4 k2: q < 8 in CTA 0, q >= 8 in CTA 1
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) {
      const int off = x * 128 + jx + 16 * (k1 + 4 * (k2 & 1));
      if ((k2 >> 1) == R)
        Y[off] = v[4 * k1 + k2];
      else
        st_cluster(peer + 8u * (uint32_t)off, v[4 * k1 + k2]);
    }
}

template <int R>
__device__ __forceinline__ void plane_load_row(const float2* Y, uint32_t peer, int x, int jx, float2 (&v)[16]) {
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const int off = x * 128 + jx + 16 * (q & 7);
    v[q] = (q >> 3) == R ? Y[off] : ld_cluster(peer + 8u * (uint32_t)off);
  }
}

template <bool AFTER>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PLANE_THREADS, 1) spec_plane_kernel(SpecLaunch P) {
  constexpr int H = SPEC_PLANE_M / 2;              // ky per CTA, and the largest nx
  float2* const Y = spec_sm;                         // [H][H], swizzled
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j = lane & 15, c = lane >> 4;            // butterfly, line of the warp
  float2* const wb = spec_sm + H * H + warp * 2 * SPEC_PLANE_M;
  const int r = (int)cluster_rank();
  const uint32_t peer = cluster_addr(Y, (uint32_t)(r ^ 1));
  const int nx = P.g.n[0], ny = P.g.n[1];
  const float cs = P.g.conj ? -1.0f : 1.0f;
  // stage-2 twiddles of every butterfly (period 256): [j][r], rows of 18
  float2* const tws = spec_sm + H * H + PLANE_WARPS * 2 * SPEC_PLANE_M;
  if (threadIdx.x < 256) {
    const int tj = threadIdx.x >> 4, tr = threadIdx.x & 15;
    tws[PLANE_TW_ROW * tj + tr] = __ldg(P.g.tw[0] + tr * tj);
  }
  __syncthreads();
  const float2* const tw = tws + PLANE_TW_ROW * j;
  constexpr int ROWS = H / 2 / (2 * PLANE_WARPS);    // row pairs per warp in phases 1 and 3
  constexpr int COLS = H / (2 * PLANE_WARPS);        // column pairs per warp in phase 2
  const int beam = blockIdx.x >> 1, kz = blockIdx.y;
  float2* const plane = P.p[beam].a + (size_t)kz * P.g.lp;
  const float2* const sh = P.g.shat + (size_t)kz * SPEC_PLANE_M * SPEC_PLANE_M + (size_t)H * r * SPEC_PLANE_M;
  auto row_of = [&](int it) { return (H / 2) * r + 2 * (PLANE_WARPS * it + warp) + c; };
  auto load_a = [&](int it, float2 (&v)[8]) {        // rows of A: y < ny, the upper half zero
    const int x = row_of(it);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int y = j + 16 * q;
      if (AFTER)
        v[q] = load_after(plane + (size_t)x * ny + y, x < nx && y < ny);
      else
        v[q] = (x < nx && y < ny) ? __ldg(plane + (size_t)x * ny + y) : make_float2(0.0f, 0.0f);
    }
  };
  auto col_of = [&](int it) { return 2 * (PLANE_WARPS * it + warp) + c; };

  cluster_arrive_relaxed();
  if (AFTER) {
    after_trigger();
    after_wait();   // S^ and the twiddles are older than any kernel of this call
  }
  float2 pa[8];
  load_a(0, pa);

  // ---- 1. y forward
  for (int it = 0; it < ROWS; ++it) {
    const int x = row_of(it);
    float2 v[16];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      v[q] = pa[q];
      v[q + 8] = make_float2(0.0f, 0.0f);
    }
    if (it + 1 < ROWS) load_a(it + 1, pa);
    // two rows without TERMA (a beam lights a band of the
    // plane): their spectra are zero, the transform is skipped
    bool nz = false;
#pragma unroll
    for (int q = 0; q < 8; ++q) nz = nz || v[q].x != 0.0f || v[q].y != 0.0f;
    if (__any_sync(0xffffffffu, nz)) {
      w16_first<false>(v, true, wb, j, c);
      __syncwarp();
      w16_second<false>(wb, v, j, c, tw);
      __syncwarp();
    }
    if (it == 0) cluster_wait();                      // the partner runs: its half may be written
    if (x < nx) {
      if (r == 0)
        plane_store_rows<0>(Y, peer, x, j ^ (x & 15), v);
      else
        plane_store_rows<1>(Y, peer, x, j ^ (x & 15), v);
    }
  }
  cluster_arrive_release();
  cluster_wait();

  // ---- 2. x forward, times S^, x inverse, on the CTA's ky columns
  for (int it = 0; it < COLS; ++it) {
    const int k = col_of(it);
    float2 v[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int x = j + 16 * q;
      v[q] = (q < 8 && x < nx) ? Y[x * H + (k ^ j)] : make_float2(0.0f, 0.0f);
    }
    float2 sv[16];                        // S^[kz][ky][kx = j + 16 q], in flight during the forward transform
    {
      const float2* row = sh + (size_t)k * SPEC_PLANE_M + j;
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        sv[q] = __ldg(row + 16 * q);
        sv[q].y *= cs;
      }
    }
    w16_first<false>(v, true, wb, j, c);
    __syncwarp();
    w16_second<false>(wb, v, j, c, tw);
    __syncwarp();
    float2 u[16];
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
      for (int k2 = 0; k2 < 4; ++k2) u[k1 + 4 * k2] = cmul(v[4 * k1 + k2], sv[k1 + 4 * k2]);
    w16_first<true>(u, false, wb, j, c);
    __syncwarp();
    w16_second<true>(wb, u, j, c, tw);
    __syncwarp();
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
      for (int k2 = 0; k2 < 2; ++k2) {
        const int x = j + 16 * (k1 + 4 * k2);
        if (x < nx) Y[x * H + (k ^ j)] = u[4 * k1 + k2];
      }
  }
  cluster_arrive_release();
  cluster_wait();

  // ---- 3. y inverse: the 256 ky of a row, half from each CTA
  for (int it = 0; it < ROWS; ++it) {
    const int x = row_of(it);
    float2 v[16];
    if (x < nx) {
      if (r == 0)
        plane_load_row<0>(Y, peer, x, j ^ (x & 15), v);
      else
        plane_load_row<1>(Y, peer, x, j ^ (x & 15), v);
    } else {
#pragma unroll
      for (int q = 0; q < 16; ++q) v[q] = make_float2(0.0f, 0.0f);
    }
    w16_first<true>(v, false, wb, j, c);
    __syncwarp();
    w16_second<true>(wb, v, j, c, tw);
    __syncwarp();
    if (x < nx) {
#pragma unroll
      for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
        for (int k2 = 0; k2 < 2; ++k2) {
          const int y = j + 16 * (k1 + 4 * k2);
          if (y < ny) plane[(size_t)x * ny + y] = v[4 * k1 + k2];
        }
    }
  }
  // the partner's loads of this CTA's half have all returned (their values
  // were used above) before it arrives: relaxed suffices
  cluster_arrive_relaxed();
  cluster_wait();
}

// S^ [Mx][My][L] -> [L][My][Mx]: 32 x 32 (kx, kz) tiles through shared
// memory, one ky per blockIdx.z
__global__ void spec_transpose_kernel(const float2* __restrict__ in, float2* __restrict__ out, int Mx, int My,
                                      int Mz) {
  __shared__ float2 t[32][33];
  const int ky = blockIdx.z, kx0 = blockIdx.y * 32, kz0 = blockIdx.x * 32;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int kx = kx0 + i, kz = kz0 + threadIdx.x;
    if (kx < Mx && kz < Mz) t[i][threadIdx.x] = in[((size_t)kx * My + ky) * Mz + kz];
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int kz = kz0 + i, kx = kx0 + threadIdx.x;
    if (kx < Mx && kz < Mz) out[((size_t)kz * My + ky) * Mx + kx] = t[threadIdx.x][i];
  }
}

__global__ void spec_scatter_kernel(const long long* __restrict__ idx, const float* __restrict__ val, int n,
                                    float* __restrict__ S) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) S[idx[k]] = val[k];
}

// ---------------------------------------------------------------- host --
// Lengths, ascending: 16 N2 for the N2 of SPEC_N2, then 2^a and 3 * 2^a.
const std::vector<int>& spec_lengths() {
  static const std::vector<int> v = [] {
    std::vector<int> p;
#define LENGTH(N2) p.push_back(16 * N2);
    SPEC_N2(LENGTH)
#undef LENGTH
    for (int m = SPEC_MIN_GENERAL; m <= SPEC_MAX_PERIOD; m *= 2) {
      p.push_back(m);
      if (m * 4 / 3 <= SPEC_MAX_PERIOD) p.push_back(m * 4 / 3);
    }
    return p;
  }();
  return v;
}

static int at_least(int n) {
  for (int m : spec_lengths())
    if (m >= n) return m;
  return 0;
}
int spec_period(int n) { return at_least(2 * n - 1); }
int spec_length_z(int nz) { return at_least(nz); }

// Twiddles of every length M back to back: exp(-2 pi i k / M), k < M, then the
// quarter steps exp(-2 pi i k / (4 M)), k < 4 M.
std::vector<float2> spec_twiddles() {
  std::vector<float2> t;
  auto add = [&](int N) {
    for (int k = 0; k < N; ++k) {
      const double a = -2.0 * 3.14159265358979323846 * (double)k / (double)N;
      t.push_back(make_float2((float)std::cos(a), (float)std::sin(a)));
    }
  };
  for (int M : spec_lengths()) {
    add(M);
    add(4 * M);
  }
  return t;
}

size_t spec_twiddle_offset(int M) {
  size_t o = 0;
  for (int m : spec_lengths()) {
    if (m == M) return o;
    o += 5 * (size_t)m;
  }
  return o;
}

// log2 of the lines per CTA of a general pass of period M: the largest power of
// two L with L M <= SPEC_ELEMS, for passes along y and x also dividing Mz
int spec_lines_log2(int M) {
  int l = 0;
  while ((2 << l) * M <= SPEC_ELEMS) ++l;
  return l;
}
int spec_pass_lines_log2(int M, int Mz) {
  int t = 0;
  while (((Mz >> t) & 1) == 0) ++t;
  return std::min(spec_lines_log2(M), t);
}

cudaError_t setup_spec_z();
cudaError_t setup_spec_y();
cudaError_t setup_spec_x();
bool launch_spec_z(const SpecLaunch& L, bool inverse, cudaStream_t st);
bool launch_spec_y(const SpecLaunch& L, bool inverse, cudaStream_t st);
bool launch_spec_x(const SpecLaunch& L, cudaStream_t st);
bool launch_spec_full(const SpecFull& F, int M, unsigned blocks, cudaStream_t st);

cudaError_t setup_spec_kernels() {
  cudaError_t e = setup_spec_z();
  if (e == cudaSuccess) e = setup_spec_y();
  if (e == cudaSuccess) e = setup_spec_x();
  for (const void* f : {(const void*)spec_z_forward_general_kernel, (const void*)spec_z_inverse_general_kernel,
                        (const void*)spec_y_general_kernel<false>, (const void*)spec_y_general_kernel<true>,
                        (const void*)spec_x_general_kernel, (const void*)spec_full_general_kernel})
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, SPEC_SMEM);
  for (const void* f : {(const void*)spec_plane_kernel<false>, (const void*)spec_plane_kernel<true>})
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, SPEC_PLANE_SMEM);
  return e;
}

void launch_spec_transpose(const float2* in, float2* out, int Mx, int My, int Mz, cudaStream_t st) {
  spec_transpose_kernel<<<dim3((Mz + 31) / 32, (Mx + 31) / 32, My), dim3(32, 8), 0, st>>>(in, out, Mx, My, Mz);
}

static void z_pass(const SpecLaunch& L, bool inverse, cudaStream_t st) {
  if (launch_spec_z(L, inverse, st)) return;
  const int lines = 1 << L.g.logL[2];
  const dim3 g((L.g.n[0] * L.g.n[1] + lines - 1) / lines, L.n_beams);
  if (inverse)
    spec_z_inverse_general_kernel<<<g, SPEC_THREADS, SPEC_SMEM, st>>>(L);
  else
    spec_z_forward_general_kernel<<<g, SPEC_THREADS, SPEC_SMEM, st>>>(L);
}

static void y_pass(const SpecLaunch& L, bool inverse, cudaStream_t st) {
  if (launch_spec_y(L, inverse, st)) return;
  const dim3 g(L.g.n[0] * (L.g.M[2] >> L.g.logL[1]), L.n_beams);
  if (inverse)
    spec_y_general_kernel<true><<<g, SPEC_THREADS, SPEC_SMEM, st>>>(L);
  else
    spec_y_general_kernel<false><<<g, SPEC_THREADS, SPEC_SMEM, st>>>(L);
}

// The passes of a launch start while their predecessors end where they are
// short: the work array A holds at most SPEC_AFTER_MAX values.  Cone stages
// without / with, same kernels: one beam 40^3 24.8 / 16.4 us, 64^3 28.8 / 21.8,
// 96^3 45 / 36, 160^3 131 / 118; 7 beams 64^3 61.7 / 48.8, 96^3 166 / 152, 128^3
// (14.7 M) 297 / 297, 144^3 (20.9 M) 521 / 566, 192^3 1293 / 1404, one 192^3 (7.1
// M) 233 / 239: a large pass
// gains nothing and its successor's CTAs take its last wave's place.
constexpr long long SPEC_AFTER_MAX = 6 << 20;

// Lines are asked for ahead where the y and x passes' work array B does not stay in
// L2 (129 MB): cone stage without / with, one beam at 192^3 (113 MB) 209 / 228 us,
// at 201^3 (167 MB) 346 / 329, at 256^3 697 / 626; four at 144^3 (191 MB) 282 / 281,
// 192^3 717 / 675; 16 at 64^3 (67 MB) 98 / 99, 96^3 (226 MB) 324 / 312.
constexpr long long SPEC_AHEAD_MIN = 18 << 20;   // complex values of B

void launch_spec_beams(SpecLaunch& L, cudaStream_t st) {
  // rows of A without TERMA are neither written nor read where the y pass goes
  // by the line flags (the kernels of lengths to 512): cone stage of 4 beams at 144^3 308 -> 298 us, 7 at 192^3
  // 1282 -> 1252.  Not on the plane path, where the flags' latency (one CTA per
  // SM) costs more than the rows: 32 beams at 128^3 1260 -> 1362.
  L.g.skip = !L.g.plane && std::max(L.g.M[1], L.g.M[2]) <= 512;
  L.g.after = (long long)L.n_beams * L.g.n[0] * L.g.n[1] * L.g.M[2] <= SPEC_AFTER_MAX ? 1 : 0;
  L.g.ahead = (long long)L.n_beams * L.g.n[0] * L.g.M[1] * L.g.M[2] >= SPEC_AHEAD_MIN ? 1 : 0;
  z_pass(L, false, st);
  if (L.g.plane) {
    // clusters of two along x: consecutive clusters take the same kz plane of
    // consecutive beams
    launch_after(L.g.after, L.g.after ? spec_plane_kernel<true> : spec_plane_kernel<false>,
                 dim3(2 * L.n_beams, L.g.M[2]), PLANE_THREADS, SPEC_PLANE_SMEM, st, L);
  } else {
    y_pass(L, false, st);
    if (!launch_spec_x(L, st))
      spec_x_general_kernel<<<(unsigned)(L.g.M[1] * (L.g.M[2] >> L.g.logL[0]) * L.n_beams), SPEC_THREADS, SPEC_SMEM,
                              st>>>(L);
    y_pass(L, true, st);
  }
  z_pass(L, true, st);
}

// The three forward passes over the folded stencil [Mx][My][L], in place.
void launch_spec_build(const SpecGrid& g, const long long* idx, const float* val, int n_val, float2* s,
                       cudaStream_t st) {
  if (n_val > 0)
    spec_scatter_kernel<<<(n_val + 255) / 256, 256, 0, st>>>(idx, val, n_val, reinterpret_cast<float*>(s));
  const size_t Mx = g.M[0], My = g.M[1], L = g.M[2];
  const int nb = (int)(L / 16);
  // lines along z in groups of 16 (My is a multiple of 16), along y and x in blocks of 16 kz
  const SpecFull f[3] = {{s, g.tw[2], g.tq, 1, 16 * L, 0, L, 1},
                         {s, g.tw[1], nullptr, nb, My * L, 16, 1, L},
                         {s, g.tw[0], nullptr, nb, L, 16, 1, My * L}};
  const int M[3] = {(int)L, (int)My, (int)Mx};
  const unsigned blocks[3] = {(unsigned)(Mx * My / 16), (unsigned)(Mx * nb), (unsigned)(My * nb)};
  for (int k = 0; k < 3; ++k)
    if (!launch_spec_full(f[k], M[k], blocks[k], st))
      spec_full_general_kernel<<<dim3(blocks[k], 16), SPEC_THREADS, SPEC_SMEM, st>>>(f[k], M[k]);
}

}  // namespace ch
