// Jaw + MLCX block map rasterised on the device (conehead/block.py:87-215).
//
// The reference builds a float32 map of |leaf span| x 4000 cells (0.1 mm) on
// the host from the plan's leaf positions and copies it to the GPU on every
// dose call (conehead/conehead.py:555).  Here the host passes the leaf table
// (a few KB, by value as the kernel parameter) and the kernel writes only the
// window the dose path reads -- the jaw opening -- straight into the crop
// buffer that ch_beam.block points at.
//
// A warp per map row: the leaf pair covering it is found once per row
// (binary search over row0[], a uniform constant-bank read) and the value of a
// leaf's body once per row; a lane writes four consecutive columns at a time.  The values
// are those of the reference's arithmetic: the leaf ramp is multiplied in
// float64 and rounded to float32 (numpy's in-place multiply of a float32
// array by float64 linspace values), then subtracted from 1 in float32.  Only
// the 15 cells of a leaf's tip need that product (two lanes per clock and SM):
// with it on every cell, one cell per thread, 1600 x 1600 cells (10 MB) took 17
// us, this 10 us (a search through cold constants and two tips a row).

#include "ch_internal.cuh"

namespace ch {
namespace {

// tongue-and-groove profile of row i of a leaf w rows high: the writes
// rows 0, 1, 2 = 0.2, 0.5, 0.75 then rows w-1, w-2, w-3 = 0.2, 0.5, 0.75,
// later writes winning where they meet (conehead/block.py:148-155)
__device__ __forceinline__ float leaf_profile(int i, int w) {
  float v = 1.0f;
  if (i == 0) v = 0.2f;
  if (i == 1) v = 0.5f;
  if (i == 2) v = 0.75f;
  if (i == w - 1) v = 0.2f;
  if (i == w - 2) v = 0.5f;
  if (i == w - 3) v = 0.75f;
  return v;
}

__device__ __forceinline__ float leaf_value(float profile, double ramp) {
  return __fsub_rn(1.0f, __double2float_rn(__dmul_rn((double)profile, ramp)));
}

__global__ void __launch_bounds__(256) mlc_raster_kernel(const ch_mlc m, float* __restrict__ out, int rows,
                                                         int cols, int r0, int c0, int vec) {
  const int rr = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (rr >= rows) return;   // whole warp
  const int r = r0 + rr;
  const bool row_open = r >= m.open_r0 && r < m.open_r1;
  // leaf pair of this row: the last n with row0[n] <= r, if r lies inside it
  int pair = -1;
  if (row_open) {
    int lo = 0, hi = m.n_pairs - 1;
    while (lo <= hi) {
      const int mid = (lo + hi) >> 1;
      if (m.row0[mid] <= r) {
        pair = mid;
        lo = mid + 1;
      } else {
        hi = mid - 1;
      }
    }
    if (pair >= 0 && r >= m.row0[pair] + m.rows[pair]) pair = -1;
  }
  int a_end = 0, b_start = 0;
  float prof_a = 0.0f, prof_b = 0.0f;
  if (pair >= 0) {
    const int i = r - m.row0[pair], w = m.rows[pair];
    prof_a = leaf_profile(i, w);
    prof_b = leaf_profile(w - 1 - i, w);
    a_end = m.a_end[pair];
    b_start = m.b_start[pair];
  }
  const float body_a = __fsub_rn(1.0f, prof_a), body_b = __fsub_rn(1.0f, prof_b);
  for (int cc = 4 * lane; cc < cols; cc += 128) {
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = c0 + cc + q;
      v[q] = 0.0f;
      if (row_open && c >= m.open_c0 && c < m.open_c1) {
        v[q] = 1.0f;
        if (pair >= 0) {
          if (c >= b_start && c < m.map_cols - 1) {
            // bank B: bank A's leaf turned by 180 degrees, tip at its first columns
            const int j = c - b_start;
            v[q] = j < CH_MLC_TIP_CELLS ? leaf_value(prof_b, m.tip[CH_MLC_TIP_CELLS - 1 - j]) : body_b;
          } else if (c < a_end) {
            const int k = c - (a_end - CH_MLC_TIP_CELLS);
            v[q] = k >= 0 ? leaf_value(prof_a, m.tip[k]) : body_a;
          }
        }
      }
    }
    float* d = out + (size_t)rr * cols + cc;
    if (vec) {
      *reinterpret_cast<float4*>(d) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (cc + q < cols) d[q] = v[q];
    }
  }
}

}  // namespace

void launch_mlc_raster(const ch_mlc& m, float* out, int rows, int cols, int r0, int c0, cudaStream_t st) {
  // 16-byte stores where every row starts on their boundary
  const int vec = (cols & 3) == 0 && (reinterpret_cast<size_t>(out) & 15) == 0;
  mlc_raster_kernel<<<(rows + 7) / 8, 256, 0, st>>>(m, out, rows, cols, r0, c0, vec);
}

}  // namespace ch
