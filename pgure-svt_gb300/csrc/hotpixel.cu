// hotpixel.cu — the reference's hot-pixel filter (HotPixelFilter,
// hotpixel.hpp:19-64) on the GPU, applied by the command-line tool before
// denoising.
//
// Per uint16 frame: med = median of the column medians; mad = median of the
// column medians of |frame - med| times 1/0.6745; every pixel with
// |x - med| > threshold * mad (converted to uint16) is an outlier.  Outliers are then replaced in
// column-major order, in place: an interior one by the mean of the 4th and
// 5th of its 8 sorted neighbours (as they are at that moment, so earlier
// replacements feed later ones), an edge one by med, both truncated to uint16.
//
// Reproduced from the reference's element types (Armadillo 9.880.1, absent
// from the reference tree, restated from its documented behaviour): the
// medians of uint16 data are uint16 (an even count gives lo + (hi - lo) / 2
// in integer arithmetic); `frame - med` converts med to uint16 and subtracts
// in uint16, so values below med wrap around modulo 65536 (abs() of an
// unsigned value is the value).
//
// GB300 mapping: one CTA per (frame, column) for the column medians (radix
// selection on 16-bit keys in shared memory), one CTA per frame for the
// median of medians, and one per frame for the outlier flags and the
// order-dependent replacement, a wavefront over the columns.
#include <algorithm>

#include "pgsvt.h"
#include "pgsvt_internal.h"

namespace pgsvt {
namespace {

// k-th smallest of n uint16 values val(i) (two 8-bit radix passes)
template <class F>
__device__ uint32_t select16(F val, int n, int k, unsigned* hist, int* sh) {
  uint32_t prefix = 0u, mask = 0u;
  for (int shift = 8; shift >= 0; shift -= 8) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) hist[i] = 0u;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const uint32_t v = val(i);
      if ((v & mask) == prefix) atomicAdd(&hist[(v >> shift) & 255u], 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int acc = 0, dg = 0;
      for (; dg < 255; ++dg) {
        if (acc + (int)hist[dg] > k) break;
        acc += (int)hist[dg];
      }
      sh[0] = dg;
      sh[1] = k - acc;
    }
    __syncthreads();
    prefix |= (uint32_t)sh[0] << shift;
    mask |= 255u << shift;
    k = sh[1];
    __syncthreads();
  }
  return prefix;
}

// Armadillo median() of n uint16 values: the middle one, or lo + (hi - lo)/2
template <class F>
__device__ uint32_t median16(F val, int n, unsigned* hist, int* sh) {
  if (n % 2) return select16(val, n, n / 2, hist, sh);
  const uint32_t lo = select16(val, n, n / 2 - 1, hist, sh);
  const uint32_t hi = select16(val, n, n / 2, hist, sh);
  return lo + (hi - lo) / 2u;
}

// pass 0: column medians of the frame; pass 1: of |frame - med| (uint16 wrap)
__global__ void __launch_bounds__(256) k_col_median(const uint16_t* seq, int nr, int nc,
                                                    const uint32_t* med, int pass,
                                                    uint16_t* colmed) {
  const int c = blockIdx.x, f = blockIdx.y;
  __shared__ unsigned hist[256];
  __shared__ int sh[2];
  const uint16_t* col = seq + ((size_t)f * nc + c) * nr;
  const uint16_t m = pass ? (uint16_t)med[f] : 0;
  auto val = [&](int i) -> uint32_t {
    return pass ? (uint16_t)(col[i] - m) : col[i];
  };
  const uint32_t v = median16(val, nr, hist, sh);
  if (threadIdx.x == 0) colmed[(size_t)f * nc + c] = (uint16_t)v;
}

// median of a frame's column medians
__global__ void __launch_bounds__(256) k_frame_median(const uint16_t* colmed, int nc,
                                                      uint32_t* out) {
  const int f = blockIdx.x;
  __shared__ unsigned hist[256];
  __shared__ int sh[2];
  const uint16_t* cm = colmed + (size_t)f * nc;
  const uint32_t v = median16([&](int i) -> uint32_t { return cm[i]; }, nc, hist, sh);
  if (threadIdx.x == 0) out[f] = v;
}

// ascending order of two values
__device__ __forceinline__ void order2(uint32_t& a, uint32_t& b) {
  const uint32_t lo = min(a, b), hi = max(a, b);
  a = lo;
  b = hi;
}

// ascending order of four values
__device__ __forceinline__ void order4(uint32_t (&v)[4]) {
  order2(v[0], v[1]);
  order2(v[2], v[3]);
  order2(v[0], v[2]);
  order2(v[1], v[3]);
  order2(v[1], v[2]);
}

// Flags and order-dependent replacement, one block per frame.
//
// An outlier's new value depends on the pixels before it in column-major order
// as replaced, (r-1,c), (r-1..r+1,c-1), and on those after it as they were.  All
// of the former have a smaller r + 2c and all of the latter a larger one, so
// the pixels of equal r + 2c can be replaced together: a thread owns a column
// and runs two rows behind its left neighbour.  About half of a frame's pixels
// are outliers (values below the median wrap around), so the chain of
// dependences is the whole frame's, nr + 2 nc steps; what bounds the kernel is
// the latency of one step.  So a step reads no global memory on its chain: the
// left column's newest value comes through shared memory (two buffers, one
// barrier per step), the own and the right column's unmodified values are read
// kAhead rows before they are needed, and the flag is computed from the pixel.
// 15 frames of 512 x 512, GB300: the whole call 313 -> 1.22 ms (one thread per
// frame that walked every flag took 311.8 ms of it).
constexpr int kAhead = 8;
constexpr int kStripe = 512;  // columns at a time: 1024 threads would spill

__global__ void __launch_bounds__(kStripe) k_hot_replace(uint16_t* seq, int nr, int nc,
                                                      const uint32_t* med, const uint32_t* madm,
                                                      double thr) {
  __shared__ uint16_t newest[2][kStripe];
  const int f = blockIdx.x, t = threadIdx.x, nt = blockDim.x;
  uint16_t* a = seq + (size_t)f * nr * nc;
  const uint32_t m = med[f];
  // the comparison converts threshold * mad to uint16 (Armadillo's relational
  // operators take the element type)
  const double td = thr * ((double)madm[f] * (1.0 / 0.6745));
  const uint32_t tu = !(td > 0.0) ? 0u : (td >= 65535.0 ? 65535u : (uint32_t)(uint16_t)td);
  for (int c0 = 0; c0 < nc; c0 += nt) {  // stripes of columns
    const int c = c0 + t;
    const bool col = c < nc;
    const uint16_t* own = a + (size_t)c * nr;
    const bool right = c + 1 < nc;
    const bool left = t == 0 && c0 > 0;  // the stripe before this one, final
    uint16_t on[kAhead], rn[kAhead], ln[kAhead];  // rows r + 1 of the coming steps
    auto fetch = [&](int s) {
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        const int r1 = s + q - 2 * t + 1;
        const bool in = col && r1 >= 0 && r1 < nr;
        on[q] = in ? own[r1] : 0;
        rn[q] = in && right ? own[nr + r1] : 0;
        ln[q] = in && left ? own[r1 - nr] : 0;
      }
    };
    // rows r-1, r, r+1: left column (replaced), own (replaced above, then as
    // it was), right column (as it was)
    uint32_t l0 = 0, l1 = 0, l2 = 0, up = 0, o1 = 0, o2 = 0, r0 = 0, r1 = 0, r2 = 0;
    const int steps = nr + 2 * min(nt, nc - c0) - 1;  // from step -1 (row 0 enters o2)
    fetch(-1);
    for (int s0 = -1; s0 < steps; s0 += kAhead) {
      uint16_t oc[kAhead], rc[kAhead], lc[kAhead];
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        oc[q] = on[q];
        rc[q] = rn[q];
        lc[q] = ln[q];
      }
      fetch(s0 + kAhead);
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        const int s = s0 + q, r = s - 2 * t;
        l0 = l1;
        l1 = l2;
        l2 = t > 0 ? newest[(s + 1) & 1][t - 1] : lc[q];
        o1 = o2;
        o2 = oc[q];
        r0 = r1;
        r1 = r2;
        r2 = rc[q];
        uint32_t v = o1;
        const bool in = col && r >= 0 && r < nr;
        if (in && ((o1 - m) & 0xffffu) > tu) {
          if (r > 0 && r < nr - 1 && c > 0 && right) {
            uint32_t x[4] = {l0, l1, l2, up}, y[4] = {r0, r1, r2, o2};
            order4(x);
            order4(y);
            // the lower and the upper half of the eight: the 4th is the
            // largest of the lower, the 5th the least of the upper
            const uint32_t w3 = max(max(min(x[0], y[3]), min(x[1], y[2])),
                                    max(min(x[2], y[1]), min(x[3], y[0])));
            const uint32_t w4 = min(min(max(x[0], y[3]), max(x[1], y[2])),
                                    min(max(x[2], y[1]), max(x[3], y[0])));
            v = (w3 + w4) >> 1;
          } else {
            v = m & 0xffffu;
          }
          a[(size_t)c * nr + r] = (uint16_t)v;
        }
        up = v;
        newest[s & 1][t] = (uint16_t)v;
        __syncthreads();
      }
    }
    __syncthreads();  // the next stripe reads this one's last column
  }
}

}  // namespace

cudaError_t launch_hot_pixel(uint16_t* seq, int nr, int nc, int nimg, double thr, uint16_t* colmed,
                             uint32_t* med, uint32_t* madm, cudaStream_t s) {
  k_col_median<<<dim3(nc, nimg), 256, 0, s>>>(seq, nr, nc, nullptr, 0, colmed);
  k_frame_median<<<nimg, 256, 0, s>>>(colmed, nc, med);
  k_col_median<<<dim3(nc, nimg), 256, 0, s>>>(seq, nr, nc, med, 1, colmed);
  k_frame_median<<<nimg, 256, 0, s>>>(colmed, nc, madm);
  const int threads = std::min(kStripe, (nc + 31) / 32 * 32);
  k_hot_replace<<<nimg, threads, 0, s>>>(seq, nr, nc, med, madm, thr);
  return cudaGetLastError();
}

}  // namespace pgsvt
