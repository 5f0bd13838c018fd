// FFT passes of lengths 16 N2 with a 16-point and an N2-point DFT in
// registers and one shared-memory exchange between them (spectral.cu has the
// method; spectral_z.cu, spectral_y.cu and spectral_x.cu the kernels).
//
// Lengths: N2 in SPEC_N2, i.e. 48 to 512.  2^a and 3 * 2^a alone wasted up to
// half of an axis: 160 voxels need a period of 319 and took 384 (x pass of 16
// beams 1515 us, 913 us at 320), 201 need 401 and took 512 through four
// shared-memory stages of the general kernels (x pass of one beam 871 us at two
// beams' cost, 236 us at 432).
#pragma once

#include "ch_internal.cuh"
#include "spectral_dft.cuh"

namespace ch {

#define SPEC_N2(X) X(3) X(4) X(5) X(6) X(8) X(9) X(10) X(12) X(15) X(16) X(18) X(20) X(24) X(27) X(32)

// A CTA takes 16 lines: 16 N2 threads in the 16-point stages, 256 in the
// N2-point ones.  r16n_ctas: CTAs per SM of the y and z passes, which stream and
// gain from warps in flight until the N2-point stage spills.  Cone stage of 8
// beams at 4, 3, 2, 1 CTAs (N2 up to 12, 16, 24, 32) / these / one more:
// 96^3 197 / 186 / 210 us, 144^3 671 / 592 / 611, 160^3 925 / 842 / 871, 192^3
// 1519 / 1423 / 1506, 201^3 3009 / 2583 / 3195.
template <int N2>
constexpr int r16n_threads() { return 16 * N2 > 256 ? 16 * N2 : 256; }
template <int N2>
constexpr int r16n_ctas() { return N2 <= 12 ? 6 : N2 <= 16 ? 5 : N2 <= 20 ? 4 : N2 <= 24 ? 3 : 2; }

// The y and x passes have two or three CTAs per SM, all waiting for memory at
// their start: each asks L2 for the lines of the CTA SPEC_AHEAD further on, one
// row of 128 bytes per thread (76 and 228 CTAs ahead: within 1%; 608 in the y
// pass: nothing gained).  Cone stage without / x alone / both, seven beams at 192^3
// 1248 / 1205 / 1168 us, 64 mixed beams 2654 / 2608 / 2563.  Nothing gained in the z
// passes, 1.5% lost in the plane kernel.
constexpr int SPEC_AHEAD = 152;
__device__ __forceinline__ void prefetch_row(const float2* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

}  // namespace ch
