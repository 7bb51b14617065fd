// svd_split.cu — SVD forms that run as several kernels, each with a small
// code footprint (one kernel holding all phases thrashed the instruction
// cache) and its own register budget:
//
// QR-preconditioned form, Casorati matrices of 17..64 rows (patch sides
// 5..8) and windows of up to 15 frames.  A one-sided Jacobi sweep costs work
// proportional to the rows of the matrix it orthogonalises.  For an m x n
// Casorati matrix B with m > n the kernels first reduce B to the n x n
// triangle R of its Householder QR factorisation (B = Q R), then run the
// Jacobi sweeps on X = R^T, whose rotated columns X W = U_X S give the right
// singular vectors of B directly (R = W S U_X^T, so B = (Q W) S U_X^T):
// v_t = U_X e_t, and the left ones follow from B itself, u_t = B v_t / s_t.
// Q and W are never formed.
//   k_qr      16 lanes per patch: Householder reflections on four columns at a
//             time in registers; X = R^T to a scratch array
//   k_xsweep  4 lanes x (NC/4) rows per patch, eight patches per warp: the
//             register-form Jacobi sweeps of svd_kernel.cuh (same rotations,
//             same convergence rules) on X; the singular values, sorted, and
//             the rotated columns that can survive back to the scratch
//   k_qr_out  16 lanes x 4 rows per patch: u_t = B v_t / s_t, the stored
//             factors and the risk projections h_t = u_t^T G v_t.
//
// Two-kernel register form, at most 16 rows and windows of up to 15 frames
// (the default for patch sides 2..4): k_bsweep runs the register form's
// sweeps on B at four resident blocks per SM, k_bout the factors, exactly as
// the single-kernel form computes them.
#include <cuda.h>

#include <cstring>

#include "svd_kernel.cuh"

namespace pgsvt {
namespace svdk {

// Tensor maps of the factors kernel's staged tiles: the normalised windows,
// the risk fields of copies 0 and 1/2, and the probe codes of copies 1/2.
struct BoutMaps {
  CUtensorMap u, f0, f2, d2;
};

namespace {

constexpr int kQL = 16;  // lanes per patch in the QR and the epilogue
constexpr int kQR = 4;   // rows per lane there

template <int NC>
struct QrDims {
  static constexpr int RX = (NC + 3) / 4;  // rows of X per lane in the sweeps
  static constexpr int XR = 4 * RX;        // rows of X (NC rounded up to 4)
  static constexpr int CS = XR + 1;        // column stride of X staged in shared memory
};

// One patch's source: window, trajectory and the perturbation of its copy.
struct PatchSrc {
  const float* uw;
  const uint32_t* posw;
  const int8_t* d1;
  const int8_t* d2code;
  size_t poff, F;
  int posidx, P, S, c;
  float pa, pb0;
  __device__ void init(const Problem& pb, const DeviceBuffers& d, int p, int c_, int w) {
    const Geometry& g = pb.g;
    const WinConst& wc = d.wc[w];
    F = g.F();
    P = g.P;
    S = g.S;
    c = c_;
    uw = d.u + (size_t)w * g.cube();
    posidx = d.plist[p];
    posw = d.pos + (size_t)w * g.nwin * g.P;
    poff = (size_t)w * d.probe_stride;
    d1 = d.d1;
    d2code = d.d2code;
    pa = pb0 = 0.f;
    if (c == 1 || c == 2) {  // pgure.hpp:80-82
      const double sg = (c == 1) ? 1.0 : -1.0;
      pa = (float)(sg * d.d2neg * wc.eps2);
      pb0 = (float)(sg * d.d2pos * wc.eps2);
    } else if (c == 3) {
      pa = (float)wc.eps1;
    }
  }
  __device__ size_t base(int k) const {  // slice k of the trajectory
    const uint32_t pc = __ldg(posw + (size_t)k * P + posidx);
    return (size_t)k * F + (pc & 0xffffu) + (size_t)(pc >> 16) * S;
  }
  __device__ float value(size_t kidx) const {
    float v = __ldg(uw + kidx);
    if (c == 1 || c == 2) v += __ldg(d2code + poff + kidx) ? pa : pb0;
    else if (c == 3) v += (float)__ldg(d1 + poff + kidx) * pa;
    return v;
  }
};

__device__ __forceinline__ float half_sum(float v) {  // over the 16 lanes of a half-warp
#pragma unroll
  for (int o = 1; o < kQL; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---- TMA staging of frame tiles (k_bout_tma)
//
// The 32 patches of a factors block are 8 x 4 neighbouring grid positions
// (the tile order of the kept patches), so in every slice of the window their
// trajectory positions fall in a small box.  One thread of the block loads,
// per slice, a tile of the normalised window, of the risk field and of the
// probe codes around that box with cp.async.bulk.tensor into the block's own
// shared memory (one mbarrier, bounded wait); the lanes then assemble their
// Casorati rows from shared memory.  Slices whose box does not fit a tile,
// and blocks that straddle two windows or copies, read global memory as the
// unstaged kernel does.  The tensor maps cover this device's buffers only.
constexpr int kTR = 24, kTC = 12;  // fp32 tile: rows (inner, 96 bytes) x columns
constexpr int kTRP = 32;           // probe-code tile rows (uint8, 32 bytes)
constexpr int kTile = kTR * kTC, kPTile = kTRP * kTC;
constexpr unsigned kSpinPolls = 1u << 22;  // bounded mbarrier polls

__device__ __forceinline__ uint32_t smem_addr(const void* ptr) {
  return (uint32_t)__cvta_generic_to_shared(ptr);
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (unsigned it = 0; it < kSpinPolls; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok) return true;
  }
  return false;
}

__device__ __forceinline__ void tma_tile3(uint32_t dst, const CUtensorMap* map, int x, int y, int z,
                                          uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];"
      :: "r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}

// ---- Householder QR of every patch's Casorati matrix, X = R^T to xq
// ([item][NC][XR]; column k of X = row k of R).  Four rows per lane, four columns
// at a time in registers: the reflections of the earlier columns come from shared
// memory, one after the other, and their four dot products share one exchange
// over the lanes (each in half_sum's order).  What bounds it is the L1 data pipe
// (80% busy: gathers, shuffles and shared memory), and all columns in shared memory
// with one exchange per dot product took four times the last two.  256 x 256 x 24, 8 x 8 patches, GB300:
// 22.4 -> 14.3 ms in 3 launches.

// |v|^2 of a reflection below which it is left out: its column has no norm left
// (equal columns, as of saturated pixels, leave 1e-7 of the norm each time), and
// 2 / |v|^2 would overflow and make the patch's columns NaN.
constexpr float kTinyColumn = 1e-36f;

// f[i] = beta * half_sum(t[i])
__device__ __forceinline__ void half_sums4(const float (&t)[4], float beta, float (&f)[4]) {
  const int lane = threadIdx.x & 31;
  const bool b0 = lane & 1, b1 = lane & 2;
  float k0 = b0 ? t[2] : t[0], k1 = b0 ? t[3] : t[1];
  k0 += __shfl_xor_sync(0xffffffffu, b0 ? t[0] : t[2], 1);
  k1 += __shfl_xor_sync(0xffffffffu, b0 ? t[1] : t[3], 1);
  float v = b1 ? k1 : k0;
  v += __shfl_xor_sync(0xffffffffu, b1 ? k0 : k1, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  v += __shfl_xor_sync(0xffffffffu, v, 8);
  v *= beta;  // lanes 0, 2, 1, 3 of every four hold t[0..3]'s
#pragma unroll
  for (int i = 0; i < 4; ++i) f[i] = __shfl_sync(0xffffffffu, v, (i >> 1) | ((i & 1) << 1), 4);
}

template <int NC>
__global__ void __launch_bounds__(128, 8) k_qr(Problem pb, DeviceBuffers d, int nitems) {
  using D = QrDims<NC>;
  constexpr int kRows = kQL * kQR;
  const Geometry& g = pb.g;
  const int lane = threadIdx.x & 31, l16 = lane & (kQL - 1);
  const int slot = threadIdx.x >> 4;  // patch of the block (8 per block)
  const int gid = blockIdx.x * 8 + slot;
  const bool live = gid < nitems;
  const int nwin = g.nwin, M = g.M;
  constexpr int kKept = D::XR - 4;  // reflections that a later column needs
  __shared__ __align__(16) float Hs[8][kKept * kRows];  // their vectors
  __shared__ float Bt[8][kKept];                        // and factors
  int p, c, w;
  {
    const int gg = live ? gid : 0;
    p = gg % g.NP;
    const int r = gg / g.NP;
    c = r % d.ncopies;
    w = r / d.ncopies;
  }
  PatchSrc src;
  src.init(pb, d, p, c, w);
  const int r0 = l16 * kQR;
  int roff[kQR];
#pragma unroll
  for (int r = 0; r < kQR; ++r)
    roff[r] = r0 + r < M ? ((r0 + r) % g.bs) + ((r0 + r) / g.bs) * g.S : -1;
  float* H = Hs[slot] + r0;
  float* xo = d.xq + ((size_t)gid * NC + r0) * D::XR;
  for (int j0 = 0; j0 < D::XR; j0 += 4) {
    float b[4][kQR];  // columns j0 .. j0 + 3 (svt.hpp:101-109)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool colok = live && j0 + i < nwin;
      const size_t at = colok ? src.base(j0 + i) : 0;
#pragma unroll
      for (int r = 0; r < kQR; ++r)
        b[i][r] = (colok && roff[r] >= 0) ? src.value(at + roff[r]) : 0.f;
    }
    const int jn = min(j0, nwin);
    for (int j = 0; j < jn; ++j) {
      const float4 v4 = *reinterpret_cast<const float4*>(H + j * kRows);
      const float* v = &v4.x;
      float t[4], f[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        t[i] = 0.f;
#pragma unroll
        for (int r = 0; r < kQR; ++r) t[i] = fmaf(v[r], b[i][r], t[i]);
      }
      half_sums4(t, Bt[slot][j], f);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int r = 0; r < kQR; ++r) b[i][r] = fmaf(-f[i], v[r], b[i][r]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int jj = j0 + i;
      if (jj >= nwin) break;  // warp-uniform
      float ss = 0.f;         // |rows >= jj of column jj|^2
#pragma unroll
      for (int r = 0; r < kQR; ++r)
        if (r0 + r >= jj) ss = fmaf(b[i][r], b[i][r], ss);
      ss = half_sum(ss);
      const float xj = __shfl_sync(0xffffffffu, b[i][i], j0 >> 2, kQL);  // row jj
      const float alpha = xj >= 0.f ? -sqrtf(ss) : sqrtf(ss);
      const float vtv = 2.f * (ss - xj * alpha);  // |x - alpha e_jj|^2
      const float beta = vtv > kTinyColumn ? 2.f / vtv : 0.f;
      float4 v4;
      float* v = &v4.x;
#pragma unroll
      for (int r = 0; r < kQR; ++r) {
        const int e = r0 + r;
        v[r] = e > jj ? b[i][r] : (e == jj ? xj - alpha : 0.f);
        if (e == jj) b[i][r] = alpha;
        else if (e > jj) b[i][r] = 0.f;
      }
      if (jj < kKept) {
        *reinterpret_cast<float4*>(H + jj * kRows) = v4;
        if (l16 == 0) Bt[slot][jj] = beta;
      }
      float t[4] = {0.f, 0.f, 0.f, 0.f}, f[4];
#pragma unroll
      for (int n = i + 1; n < 4; ++n)
#pragma unroll
        for (int r = 0; r < kQR; ++r) t[n] = fmaf(v[r], b[n][r], t[n]);
      if (i < 2) {
        half_sums4(t, beta, f);
      } else if (i == 2) {
        f[3] = beta * half_sum(t[3]);
      }
#pragma unroll
      for (int n = i + 1; n < 4; ++n)
#pragma unroll
        for (int r = 0; r < kQR; ++r) b[n][r] = fmaf(-f[n], v[r], b[n][r]);
    }
    __syncwarp();  // Bt
    // X column k = row k of R (rows >= nwin of R are zero)
    if (live)
#pragma unroll
      for (int r = 0; r < kQR; ++r)
        if (r0 + r < NC) {
          float4 t;
          t.x = j0 + 0 < nwin ? b[0][r] : 0.f;
          t.y = j0 + 1 < nwin ? b[1][r] : 0.f;
          t.z = j0 + 2 < nwin ? b[2][r] : 0.f;
          t.w = j0 + 3 < nwin ? b[3][r] : 0.f;
          *reinterpret_cast<float4*>(xo + r * D::XR + j0) = t;
        }
  }
}

// ---- end of a sweep kernel: the column norms (the singular values) of one
// patch per lane group, sorted, and the rotated columns of the triplets that
// can survive the threshold, in that order: xq [item][rank][XR], the count in
// nlive.  Lane q takes columns 4n + q: their sums come from a
// reduce-scatter (the lanes added in lanes_sum's order), their ranks from
// comparisons with every column (ties by index); sorting in the factors
// kernels took more instructions there than the factors themselves.  `get`:
// this lane's row r of column k; `slot`: the lane group's scratch (32 floats).
template <int NC, int RX, int XR, class Get>
__device__ __forceinline__ void store_sorted(const Problem& pb, const DeviceBuffers& d, Get get,
                                             float* slot, int q, int gid, bool live) {
  constexpr int N4 = (NC + 3) / 4;
  const Geometry& g = pb.g;
  const int gbase = (threadIdx.x & 31) & ~3;
  const bool b0 = (q & 1) != 0, b1 = (q & 2) != 0;
  float s[N4];
  float smax = 0.f;
#pragma unroll
  for (int n = 0; n < N4; ++n) {
    float t[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = 4 * n + j;
      t[j] = 0.f;
      if (k < NC - 1)
#pragma unroll
        for (int r = 0; r < RX; ++r) t[j] = fmaf(get(r, k), get(r, k), t[j]);
    }
    const float u0 = (b0 ? t[1] : t[0]) + __shfl_xor_sync(0xffffffffu, b0 ? t[0] : t[1], 1);
    const float u1 = (b0 ? t[3] : t[2]) + __shfl_xor_sync(0xffffffffu, b0 ? t[2] : t[3], 1);
    s[n] = sqrtf((b1 ? u1 : u0) + __shfl_xor_sync(0xffffffffu, b1 ? u0 : u1, 2));
    smax = fmaxf(smax, s[n]);
  }
  smax = fmaxf(smax, __shfl_xor_sync(0xffffffffu, smax, 1));
  smax = fmaxf(smax, __shfl_xor_sync(0xffffffffu, smax, 2));
  int p = 0, c = 0, w = 0;
  if (live) {
    p = gid % g.NP;
    const int r = gid / g.NP;
    c = r % d.ncopies;
    w = r / d.ncopies;
  }
  const float upper = (float)d.wc[w].upper;
  int nl = 0, rank[N4];
#pragma unroll
  for (int n = 0; n < N4; ++n) {
    nl += 4 * n + q < NC && can_survive(pb, s[n], smax, upper);
    rank[n] = 0;
  }
  nl += __shfl_xor_sync(0xffffffffu, nl, 1);
  nl += __shfl_xor_sync(0xffffffffu, nl, 2);
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    const float sj = __shfl_sync(0xffffffffu, s[j >> 2], gbase | (j & 3));
#pragma unroll
    for (int n = 0; n < N4; ++n) rank[n] += sj > s[n] || (sj == s[n] && j < 4 * n + q);
  }
  // (a NaN column has no rank, and a value without a column is -1)
  __syncwarp();
  int* ir = reinterpret_cast<int*>(slot + 16);
#pragma unroll
  for (int n = 0; n < N4; ++n) slot[4 * n + q] = -1.f;
  __syncwarp();
#pragma unroll
  for (int n = 0; n < N4; ++n)
    if (4 * n + q < NC) {
      const bool num = s[n] == s[n];
      if (num) slot[rank[n]] = s[n];
      ir[4 * n + q] = num ? rank[n] : NC;
    }
  __syncwarp();
  if (live) {
    const size_t NP = g.NP;
    float* svo = d.sv + (((size_t)w * 4 + c) * g.NC) * NP + p;
    float* hvo = d.hv + (((size_t)w * 4 + c) * g.NC) * NP + p;
#pragma unroll
    for (int n = 0; n < N4; ++n) {
      const int t = 4 * n + q;
      if (t < NC) {
        svo[(size_t)t * NP] = slot[t];
        if (t >= nl) hvo[(size_t)t * NP] = 0.f;
      }
    }
    if (q == 0) d.nlive[((size_t)w * 4 + c) * NP + p] = nl;
    float* xo = d.xq + (size_t)gid * NC * XR + q * RX;
#pragma unroll
    for (int k = 0; k < NC - 1; ++k) {
      const int t = ir[k];
      if (t >= nl) continue;
      if constexpr (RX == 4) {
        *reinterpret_cast<float4*>(xo + t * XR) =
            make_float4(get(0, k), get(1, k), get(2, k), get(3, k));
      } else {
#pragma unroll
        for (int r = 0; r < RX; ++r) xo[t * XR + r] = get(r, k);
      }
    }
  }
  __syncwarp();
}

// ---- Jacobi sweeps on X, four lanes per patch, eight patches per warp
template <int NC>
__global__ void __launch_bounds__(128, 4) k_xsweep(Problem pb, DeviceBuffers d, int nitems) {
  using D = QrDims<NC>;
  constexpr int RX = D::RX, CS = D::CS;
  const int lane = threadIdx.x & 31, q = lane & 3;
  const int slot = threadIdx.x >> 2;  // patch of the block (32 per block)
  const int gid = blockIdx.x * 32 + slot;
  const bool live = gid < nitems;
  __shared__ __align__(16) float Xs[32][(NC * CS + 3) / 4 * 4];
  float* X = Xs[slot];
  const float* xi = d.xq + (size_t)(live ? gid : 0) * NC * D::XR;
  RegCols<RX, NC> A;
#pragma unroll
  for (int k = 0; k < NC; ++k)
#pragma unroll
    for (int r = 0; r < RX; ++r) A.put(r, k, live ? __ldg(xi + k * D::XR + q * RX + r) : 0.f);
  unsigned fp64_tests = 0;
  const int sweeps = register_sweeps<RX, 4, NC, CS, 1>(A, X, q, pb.g.nwin, fp64_tests);
  if (lane == 0) atomicAdd(d.counters + 1, (unsigned long long)(sweeps + 1));
  if (q == 0 && fp64_tests) atomicAdd(d.counters + 2, (unsigned long long)fp64_tests);
  store_sorted<NC, RX, D::XR>(pb, d, [&](int r, int k) { return A(r, k); }, X, q, gid, live);
}

// ---- the factors: u_t = B v_t / s_t, h_t = u_t^T G v_t, for the nl triplets
// that can survive (already sorted, see store_sorted).  Few of them can (about
// 5 of 15 at 8 x 8 patches), so up to kQT are formed side by side while one
// slice of B, then of G, is in registers: nothing is held across slices and
// the loads of many warps overlap.  256 x 256 x 24, 8 x 8 patches, GB300: 56.2 ->
// 22.6 ms in 3 launches (before, B held in registers and the columns sorted here).
constexpr int kQT = 8;

template <int NC>
__global__ void __launch_bounds__(128, 5) k_qr_out(Problem pb, DeviceBuffers d, int nitems) {
  using D = QrDims<NC>;
  const Geometry& g = pb.g;
  const int lane = threadIdx.x & 31, l16 = lane & (kQL - 1);
  const int slot = threadIdx.x >> 4;
  const int gid = blockIdx.x * 8 + slot;
  const bool live = gid < nitems;
  const int nwin = g.nwin, M = g.M;
  __shared__ __align__(16) float Vs[8][NC][kQT];  // v_t of the triplets at hand
  int p, c, w;
  {
    const int gg = live ? gid : 0;
    p = gg % g.NP;
    const int r = gg / g.NP;
    c = r % d.ncopies;
    w = r / d.ncopies;
  }
  const int nl = live ? d.nlive[((size_t)w * 4 + c) * g.NP + p] : 0;
  const int nl_max = max(nl, __shfl_xor_sync(0xffffffffu, nl, 16));
  if (nl_max == 0) return;  // warp-uniform
  const float* X = d.xq + (size_t)(live ? gid : 0) * NC * D::XR;
  int roff[kQR];
#pragma unroll
  for (int r = 0; r < kQR; ++r) {
    const int e = l16 * kQR + r;
    roff[r] = e < M ? (e % g.bs) + (e / g.bs) * g.S : -1;
  }
  const size_t NP = g.NP;
  const int NCg = g.NC;
  const float* svo = d.sv + (((size_t)w * 4 + c) * NCg) * NP + p;
  float* hvo = d.hv + (((size_t)w * 4 + c) * NCg) * NP + p;
  const float* fld = (c == 0) ? d.fld0 : (c == 3 ? d.fld1 : d.fld2);
  const float* fw_ = (pb.optimize && fld) ? fld + (size_t)w * g.cube() : nullptr;
  PatchSrc src;
  src.init(pb, d, p, c, w);
  const bool keep = c == 0 && live && d.U0 && d.V0;
  for (int t0 = 0; t0 < nl_max; t0 += kQT) {
    const int nt = min(kQT, nl_max - t0);  // warp-uniform
    float inv[kQT];
    __syncwarp();
#pragma unroll
    for (int t = 0; t < kQT; ++t) {
      inv[t] = 0.f;
      if (t < nt) {
        const float st = t0 + t < nl ? svo[(size_t)(t0 + t) * NP] : 0.f;
        inv[t] = st > 0.f ? 1.f / st : 0.f;
        // v_t = X's rotated column t times inv
        if (l16 < NC) {
          const float v = (t0 + t < nl && l16 < nwin) ? X[(t0 + t) * D::XR + l16] * inv[t] : 0.f;
          Vs[slot][l16][t] = v;
          if (keep && t0 + t < nl && l16 < nwin)
            d.V0[g.v_at(w, p) + ((t0 + t) * nwin + l16) * 32] = v;
        }
      } else if (l16 < NC) {
        Vs[slot][l16][t] = 0.f;
      }
    }
    __syncwarp();
    float a[kQT][kQR];  // u_t rows
#pragma unroll
    for (int t = 0; t < kQT; ++t)
#pragma unroll
      for (int r = 0; r < kQR; ++r) a[t][r] = 0.f;
#pragma unroll 3
    for (int k = 0; k < nwin; ++k) {
      float B[kQR];
      const size_t b = live ? src.base(k) : 0;
#pragma unroll
      for (int r = 0; r < kQR; ++r) B[r] = (live && roff[r] >= 0) ? src.value(b + roff[r]) : 0.f;
      float v[kQT];
#pragma unroll
      for (int t = 0; t < kQT; t += 4)
        *reinterpret_cast<float4*>(v + t) = *reinterpret_cast<const float4*>(&Vs[slot][k][t]);
#pragma unroll
      for (int t = 0; t < kQT; ++t)
        if (t < nt)
#pragma unroll
          for (int r = 0; r < kQR; ++r) a[t][r] = fmaf(B[r], v[t], a[t][r]);
    }
#pragma unroll
    for (int t = 0; t < kQT; ++t) {
#pragma unroll
      for (int r = 0; r < kQR; ++r) {
        a[t][r] *= inv[t];
        if (keep && t0 + t < nl && roff[r] >= 0)
          d.U0[g.u_at(w, p) + ((t0 + t) * M + l16 * kQR + r) * 32] = a[t][r];
      }
    }
    if (fw_) {
      // h_t = sum_k v_k (G_k . u_t): the lanes' partial sums, one reduction
      float h[kQT];
#pragma unroll
      for (int t = 0; t < kQT; ++t) h[t] = 0.f;
#pragma unroll 3
      for (int k = 0; k < nwin; ++k) {
        float G[kQR];
        const size_t b = live ? src.base(k) : 0;
#pragma unroll
        for (int r = 0; r < kQR; ++r) G[r] = (live && roff[r] >= 0) ? __ldg(fw_ + b + roff[r]) : 0.f;
        float v[kQT];
#pragma unroll
        for (int t = 0; t < kQT; t += 4)
          *reinterpret_cast<float4*>(v + t) = *reinterpret_cast<const float4*>(&Vs[slot][k][t]);
#pragma unroll
        for (int t = 0; t < kQT; ++t)
          if (t < nt) {
            float gu = 0.f;
#pragma unroll
            for (int r = 0; r < kQR; ++r) gu = fmaf(G[r], a[t][r], gu);
            h[t] = fmaf(v[t], gu, h[t]);
          }
      }
#pragma unroll
      for (int t = 0; t < kQT; ++t)
        if (t < nt) {
          const float hs = half_sum(h[t]);
          if (live && t0 + t < nl && l16 == 0) hvo[(size_t)(t0 + t) * NP] = hs;
        }
    }
  }
}

// ---- the same two-kernel split without the QR, for patches of at most 16
// rows (sides 2..4): the sweeps on B itself at four resident blocks per SM,
// then the factors from the rotated columns (u_t = a_t / s_t, v_t = B^T u_t
// / s_t), exactly as the single-kernel register form computes them: the same
// operations in the same order, so the results are identical to it.
template <int NC>
__global__ void __launch_bounds__(128, 4) k_bsweep(Problem pb, DeviceBuffers d, int nitems) {
  constexpr int RX = 4, XR = 16, CS = XR + 1;
  const Geometry& g = pb.g;
  const int lane = threadIdx.x & 31, q = lane & 3;
  const int slot = threadIdx.x >> 2;  // patch of the block (32 per block)
  const int gid = blockIdx.x * 32 + slot;
  const bool live = gid < nitems;
  const int nwin = g.nwin, M = g.M;
  __shared__ __align__(16) float Xs[32][(NC * CS + 3) / 4 * 4];
  float* X = Xs[slot];
  PatchSrc src;
  {
    const int gg = live ? gid : 0, r = gg / g.NP;
    src.init(pb, d, gg % g.NP, r % d.ncopies, r / d.ncopies);
  }
  int roff[RX];
#pragma unroll
  for (int r = 0; r < RX; ++r) {
    const int e = q * RX + r;
    roff[r] = (live && e < M) ? (e % g.bs) + (e / g.bs) * g.S : -1;
  }
  RegCols<RX, NC> A;
#pragma unroll
  for (int k = 0; k < NC; ++k) {
    const bool colok = live && k < nwin;
    const size_t b = colok ? src.base(k) : 0;
#pragma unroll
    for (int r = 0; r < RX; ++r) A.put(r, k, (colok && roff[r] >= 0) ? src.value(b + roff[r]) : 0.f);
  }
  unsigned fp64_tests = 0;
  const int sweeps = register_sweeps<RX, 4, NC, CS, 1>(A, X, q, nwin, fp64_tests);
  if (lane == 0) atomicAdd(d.counters + 1, (unsigned long long)(sweeps + 1));
  if (q == 0 && fp64_tests) atomicAdd(d.counters + 2, (unsigned long long)fp64_tests);
  store_sorted<NC, RX, XR>(pb, d, [&](int r, int k) { return A(r, k); }, X, q, gid, live);
}

// The factors of the nl triplets that can survive (already sorted, see
// store_sorted): one or two of 15 as a rule, so up to kBT are formed side by
// side while one slice of B and G is in registers.  Nothing is held across
// slices (the earlier form kept all of B and G, at 16 warps per SM, and was
// bound by the latency of its loads and by sorting the columns).  256 x 256 x
// 100, GB300: 35.0 -> 15.3 ms in 13 launches, still bound by the latency of the
// gathers: 7 blocks per SM (72 registers), where 8 took 16.6 and 6 or 10 16.8 ms.
constexpr int kBT = 4;

template <int NC>
__global__ void __launch_bounds__(128, 7) k_bout(Problem pb, DeviceBuffers d, int nitems) {
  constexpr int RX = 4, XR = 16;
  const Geometry& g = pb.g;
  const int lane = threadIdx.x & 31, q = lane & 3;
  const int gid = blockIdx.x * 32 + (threadIdx.x >> 2);
  const bool live = gid < nitems;
  const int nwin = g.nwin, M = g.M;
  int p, c, w;
  {
    const int gg = live ? gid : 0;
    p = gg % g.NP;
    const int r = gg / g.NP;
    c = r % d.ncopies;
    w = r / d.ncopies;
  }
  const int nl = live ? d.nlive[((size_t)w * 4 + c) * g.NP + p] : 0;
  const int nl_max = __reduce_max_sync(0xffffffffu, nl);
  if (nl_max == 0) return;  // warp-uniform
  const float* X = d.xq + (size_t)(live ? gid : 0) * NC * XR + q * RX;
  int roff[RX];
#pragma unroll
  for (int r = 0; r < RX; ++r) {
    const int e = q * RX + r;
    roff[r] = (live && e < M) ? (e % g.bs) + (e / g.bs) * g.S : -1;
  }
  const size_t NP = g.NP;
  const int NCg = g.NC;
  const float* svo = d.sv + (((size_t)w * 4 + c) * NCg) * NP + p;
  float* hvo = d.hv + (((size_t)w * 4 + c) * NCg) * NP + p;
  const float* fld = (c == 0) ? d.fld0 : (c == 3 ? d.fld1 : d.fld2);
  const float* fw_ = (pb.optimize && fld) ? fld + (size_t)w * g.cube() : nullptr;
  PatchSrc src;
  src.init(pb, d, p, c, w);
  const bool keep = c == 0 && live && d.U0 && d.V0;
  for (int t0 = 0; t0 < nl_max; t0 += kBT) {
    const int nt = min(kBT, nl_max - t0);  // warp-uniform
    float a[kBT][RX], inv[kBT], h[kBT];    // u_t rows, 1 / s_t
#pragma unroll
    for (int t = 0; t < kBT; ++t) {
      const bool use = t0 + t < nl;
      const float st = use ? svo[(size_t)(t0 + t) * NP] : 0.f;
      inv[t] = st > 0.f ? 1.f / st : 0.f;
      const float4 x = use ? *reinterpret_cast<const float4*>(X + (t0 + t) * XR)
                           : make_float4(0.f, 0.f, 0.f, 0.f);
      const float* xp = &x.x;
      h[t] = 0.f;
#pragma unroll
      for (int r = 0; r < RX; ++r) {
        a[t][r] = xp[r] * inv[t];
        if (keep && use && roff[r] >= 0)
          d.U0[g.u_at(w, p) + ((t0 + t) * M + q * RX + r) * 32] = a[t][r];
      }
    }
    // v_t = B^T u_t / s_t and h_t = u_t^T G v_t = sum_k v_k (G_k . u_t)
#pragma unroll 3
    for (int k = 0; k < nwin; ++k) {
      const size_t b = live ? src.base(k) : 0;
      float B[RX], G[RX];
#pragma unroll
      for (int r = 0; r < RX; ++r) {
        B[r] = roff[r] >= 0 ? src.value(b + roff[r]) : 0.f;
        G[r] = fw_ && roff[r] >= 0 ? __ldg(fw_ + b + roff[r]) : 0.f;
      }
#pragma unroll
      for (int t = 0; t < kBT; ++t) {
        if (t >= nt) break;
        float bu = 0.f;
#pragma unroll
        for (int r = 0; r < RX; ++r) bu = fmaf(B[r], a[t][r], bu);
        const float vk = lanes_sum<4>(bu) * inv[t];
        if (keep && t0 + t < nl && (k & 3) == q)
          d.V0[g.v_at(w, p) + ((t0 + t) * nwin + k) * 32] = vk;
        float gu = 0.f;
#pragma unroll
        for (int r = 0; r < RX; ++r) gu = fmaf(G[r], a[t][r], gu);
        h[t] = fmaf(vk, gu, h[t]);
      }
    }
    if (fw_) {
#pragma unroll
      for (int t = 0; t < kBT; ++t)
        if (t < nt) {
          const float hs = lanes_sum<4>(h[t]);
          if (live && t0 + t < nl && q == 0) hvo[(size_t)(t0 + t) * NP] = hs;
        }
    }
  }
}

// The same from TMA-staged frame tiles (see above).
template <int NC>
__global__ void __launch_bounds__(128, 4)
    k_bout_tma(Problem pb, DeviceBuffers d, int nitems, const __grid_constant__ BoutMaps tm) {
  constexpr int RX = 4, XR = 16;
  const Geometry& g = pb.g;
  const int lane = threadIdx.x & 31, q = lane & 3;
  const int gid = blockIdx.x * 32 + (threadIdx.x >> 2);
  const bool live = gid < nitems;
  const int nwin = g.nwin, M = g.M;
  int p, c, w;
  {
    const int gg = live ? gid : 0;
    p = gg % g.NP;
    const int r = gg / g.NP;
    c = r % d.ncopies;
    w = r / d.ncopies;
  }
  const float* X = d.xq + (size_t)(live ? gid : 0) * NC * XR;
  int roff[RX];
#pragma unroll
  for (int r = 0; r < RX; ++r) {
    const int e = q * RX + r;
    roff[r] = (live && e < M) ? (e % g.bs) + (e / g.bs) * g.S : -1;
  }
  const size_t NP = g.NP;
  const int NCg = g.NC;
  const float* svo = d.sv + (((size_t)w * 4 + c) * NCg) * NP + p;
  float* hvo = d.hv + (((size_t)w * 4 + c) * NCg) * NP + p;
  const int nl = live ? d.nlive[((size_t)w * 4 + c) * g.NP + p] : 0;
  const int nl_max = __reduce_max_sync(0xffffffffu, nl);
  const float* fld = (c == 0) ? d.fld0 : (c == 3 ? d.fld1 : d.fld2);
  const float* fw_ = (pb.optimize && fld) ? fld + (size_t)w * g.cube() : nullptr;
  PatchSrc src;
  src.init(pb, d, p, c, w);
  // B in registers and, in shared memory, this lane's rows of the field G along
  // the trajectory (each lane reads back only what it wrote)
  float B[RX][NC];
  float* gs;
  {
    // dynamic shared memory: [Gs (padded rows) | field tiles]; the window
    // and probe tiles share the Gs region, which is written only after
    // every lane has assembled B
    constexpr int GSS = NC * 4 * RX + 16;  // Gs floats per patch (+16: no bank conflicts)
    constexpr int GS_BYTES = 32 * GSS * 4;
    static_assert(NC * (kTile * 4 + kPTile) <= GS_BYTES, "window tiles must fit the Gs region");
    extern __shared__ unsigned char dyn_smem[];
    unsigned char* sbase = (unsigned char*)(((uintptr_t)dyn_smem + 127) & ~(uintptr_t)127);
    float* gsm = (float*)sbase;
    float* ut = (float*)sbase;
    uint8_t* ptl = sbase + NC * kTile * 4;
    float* ftl = (float*)(sbase + GS_BYTES);
    __shared__ __align__(8) unsigned long long bar;
    __shared__ int fymin[NC], fymax[NC], fxmin[NC], fxmax[NC], fy0[NC], fyp0[NC], fx0[NC];
    __shared__ int cta_ok;
    const int tid = threadIdx.x;
    const uint32_t bara = smem_addr(&bar);
    const bool probes = (c == 1 || c == 2);
    if (tid < NC) {
      fymin[tid] = fxmin[tid] = 0x7fffffff;
      fymax[tid] = fxmax[tid] = -1;
    }
    if (tid == 0) {
      const int g0 = blockIdx.x * 32, g1 = min(nitems, g0 + 32) - 1;
      const int r0 = g0 / g.NP, r1 = g1 / g.NP;  // (window, copy) of the first and last item
      cta_ok = (r0 == r1) && (r0 % d.ncopies) <= 2;
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bara), "r"(1) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // trajectory position of slice k of this patch (row | col << 16)
    auto posk = [&](int k) -> uint32_t {
      return (live && k < nwin) ? __ldg(src.posw + (size_t)k * src.P + src.posidx) : 0u;
    };
    if (cta_ok) {
#pragma unroll 1
      for (int k = 0; k < nwin; ++k) {
        const uint32_t pc = posk(k);
        const int y = (int)(pc & 0xffffu), x = (int)(pc >> 16);
        const int ylo = __reduce_min_sync(0xffffffffu, live ? y : 0x7fffffff);
        const int yhi = __reduce_max_sync(0xffffffffu, live ? y : -1);
        const int xlo = __reduce_min_sync(0xffffffffu, live ? x : 0x7fffffff);
        const int xhi = __reduce_max_sync(0xffffffffu, live ? x : -1);
        if (lane == 0) {
          atomicMin(&fymin[k], ylo);
          atomicMax(&fymax[k], yhi);
          atomicMin(&fxmin[k], xlo);
          atomicMax(&fxmax[k], xhi);
        }
      }
    }
    __syncthreads();
    if (tid == 0) {
      unsigned bytes = 0;
      for (int k = 0; k < NC; ++k) {
        fy0[k] = -1;
        if (!cta_ok || k >= nwin || fymin[k] > fymax[k]) continue;
        const int y0 = fymin[k] & ~3, yp0 = fymin[k] & ~15, x0 = fxmin[k];
        bool fit = fymax[k] + g.bs - y0 <= kTR && fxmax[k] + g.bs - x0 <= kTC;
        if (probes) fit = fit && fymax[k] + g.bs - yp0 <= kTRP;
        if (!fit) continue;
        fy0[k] = y0;
        fyp0[k] = yp0;
        fx0[k] = x0;
        bytes += kTile * 4 + (fw_ ? kTile * 4 : 0) + (probes ? kPTile : 0);
      }
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                   :: "r"(bara), "r"(bytes) : "memory");
      const int zp = d.probe_stride ? w * nwin : 0;
      for (int k = 0; k < NC; ++k) {
        if (k >= nwin || fy0[k] < 0) continue;
        tma_tile3(smem_addr(ut + k * kTile), &tm.u, fy0[k], fx0[k], w * nwin + k, bara);
        if (fw_)
          tma_tile3(smem_addr(ftl + k * kTile), c == 0 ? &tm.f0 : &tm.f2, fy0[k], fx0[k],
                    w * nwin + k, bara);
        if (probes) tma_tile3(smem_addr(ptl + k * kPTile), &tm.d2, fyp0[k], fx0[k], zp + k, bara);
      }
    }
    __syncthreads();
    const bool ok = mbar_wait(bara, 0);
    if (__syncthreads_or(!ok)) {  // a copy did not land in time: report, drain, stop
      if (tid == 0) atomicAdd(d.counters + 4, 1ull);
      mbar_wait(bara, 0);
      return;
    }
    // tile offsets of this lane's rows (row e of the Casorati matrix is pixel
    // (e % bs, e / bs) of the patch)
    int toff[RX], poff[RX];
#pragma unroll
    for (int r = 0; r < RX; ++r) {
      const int e = q * RX + r;
      toff[r] = e % g.bs + (e / g.bs) * kTR;
      poff[r] = e % g.bs + (e / g.bs) * kTRP;
    }
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      const bool colok = live && k < nwin && nl_max > 0;
      const uint32_t pc = colok ? posk(k) : 0u;
      const int y = (int)(pc & 0xffffu), x = (int)(pc >> 16);
      if (colok && fy0[k] >= 0) {
        const float* ub = ut + k * kTile + (y - fy0[k]) + (x - fx0[k]) * kTR;
        const uint8_t* pbs = ptl + k * kPTile + (y - fyp0[k]) + (x - fx0[k]) * kTRP;
#pragma unroll
        for (int r = 0; r < RX; ++r) {
          float v = 0.f;
          if (roff[r] >= 0) {
            v = ub[toff[r]];
            if (probes) v += pbs[poff[r]] ? src.pa : src.pb0;
          }
          B[r][k] = v;
        }
      } else {
        const size_t b = colok ? (size_t)k * src.F + y + (size_t)x * src.S : 0;
#pragma unroll
        for (int r = 0; r < RX; ++r) B[r][k] = (colok && roff[r] >= 0) ? src.value(b + roff[r]) : 0.f;
      }
    }
    __syncthreads();  // the window and probe tiles are dead: Gs takes their place
    gs = gsm + (size_t)(threadIdx.x >> 2) * GSS + q * RX;
    if (fw_) {
#pragma unroll
      for (int k = 0; k < NC; ++k) {
        const bool colok = live && k < nwin && nl_max > 0;
        const uint32_t pc = colok ? posk(k) : 0u;
        const int y = (int)(pc & 0xffffu), x = (int)(pc >> 16);
        float4 g4 = make_float4(0.f, 0.f, 0.f, 0.f);
        float* gp = &g4.x;
        if (colok && fy0[k] >= 0) {
          const float* fb = ftl + k * kTile + (y - fy0[k]) + (x - fx0[k]) * kTR;
#pragma unroll
          for (int r = 0; r < RX; ++r)
            if (roff[r] >= 0) gp[r] = fb[toff[r]];
        } else if (colok) {
          const size_t b = (size_t)k * src.F + y + (size_t)x * src.S;
#pragma unroll
          for (int r = 0; r < RX; ++r)
            if (roff[r] >= 0) gp[r] = __ldg(fw_ + b + roff[r]);
        }
        *reinterpret_cast<float4*>(gs + k * 4 * RX) = g4;
      }
    }
  }
  for (int t = 0; t < nl_max; ++t) {
    const bool use = t < nl;
    const float st = use ? svo[(size_t)t * NP] : 0.f;
    const float inv = st > 0.f ? 1.f / st : 0.f;
    float a[RX];  // u_t rows
#pragma unroll
    for (int r = 0; r < RX; ++r) a[r] = (use ? X[t * XR + q * RX + r] : 0.f) * inv;
    if (c == 0 && live && use && d.U0 && d.V0) {
#pragma unroll
      for (int r = 0; r < RX; ++r)
        if (roff[r] >= 0) d.U0[g.u_at(w, p) + (t * M + q * RX + r) * 32] = a[r];
    }
    // v_t = B^T u_t / s_t and h_t = u_t^T G v_t = sum_k v_k (G_k . u_t)
    float h = 0.f;
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      if (k >= nwin) break;  // uniform: keeps B[][k] in registers
      float bu = 0.f;
#pragma unroll
      for (int r = 0; r < RX; ++r) bu = fmaf(B[r][k], a[r], bu);
      bu = lanes_sum<4>(bu);
      const float vk = bu * inv;
      if (c == 0 && live && use && (k % 4) == q && d.V0)
        d.V0[g.v_at(w, p) + (t * nwin + k) * 32] = vk;
      if (fw_ && live && use) {
        const float4 g4 = *reinterpret_cast<const float4*>(gs + k * 4 * RX);
        const float* gp = &g4.x;
        float gu = 0.f;
#pragma unroll
        for (int r = 0; r < RX; ++r)
          if (roff[r] >= 0) gu = fmaf(gp[r], a[r], gu);
        h = fmaf(vk, gu, h);
      }
    }
    if (fw_) h = lanes_sum<4>(h);
    if (live && use && q == 0) hvo[(size_t)t * NP] = h;
  }
}

}  // namespace

template <int NC>
cudaError_t run_svd_qr(const Problem& pb, const DeviceBuffers& d, cudaStream_t s) {
  if (!d.xq) return cudaErrorInvalidValue;
  const int nitems = pb.W * d.ncopies * pb.g.NP;
  k_qr<NC><<<(nitems + 7) / 8, 128, 0, s>>>(pb, d, nitems);
  k_xsweep<NC><<<(nitems + 31) / 32, 128, 0, s>>>(pb, d, nitems);
  k_qr_out<NC><<<(nitems + 7) / 8, 128, 0, s>>>(pb, d, nitems);
  return cudaGetLastError();
}

template cudaError_t run_svd_qr<10>(const Problem&, const DeviceBuffers&, cudaStream_t);
template cudaError_t run_svd_qr<16>(const Problem&, const DeviceBuffers&, cudaStream_t);

namespace {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled through the runtime's driver entry point (no libcuda link)
EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault,
                                         &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
      return (EncodeTiledFn) nullptr;
    return (EncodeTiledFn)f;
  }();
  return fn;
}

// A 3-D map over `frames` column-major S x S frames (rows innermost) with a
// box of box_rows x box_cols x 1; a null buffer gives an unused zero map.
bool frame_map(CUtensorMap* m, CUtensorMapDataType dt, size_t esize, const void* base, int S,
               int frames, int box_rows, int box_cols) {
  std::memset(m, 0, sizeof(*m));
  if (!base) return true;
  const EncodeTiledFn enc = encode_tiled();
  if (!enc) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)S, (cuuint64_t)S, (cuuint64_t)frames};
  const cuuint64_t strides[2] = {(cuuint64_t)S * esize, (cuuint64_t)S * S * esize};
  const cuuint32_t box[3] = {(cuuint32_t)box_rows, (cuuint32_t)box_cols, 1};
  const cuuint32_t es[3] = {1, 1, 1};
  return enc(m, dt, 3, const_cast<void*>(base), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

template <int NC>
cudaError_t run_svd_split(const Problem& pb, const DeviceBuffers& d, cudaStream_t s, bool staged) {
  if (!d.xq) return cudaErrorInvalidValue;
  const int nitems = pb.W * d.ncopies * pb.g.NP;
  const int S = pb.g.S, nwin = pb.g.nwin;
  k_bsweep<NC><<<(nitems + 31) / 32, 128, 0, s>>>(pb, d, nitems);
  // the factors from shared-memory tiles staged by TMA (when asked for and
  // every map's row stride is a multiple of 16 bytes), else from global
  // memory; the same values either way, so identical results
  BoutMaps tm;
  bool tma = staged && S % 16 == 0 && d.counters != nullptr;
  if (tma) {
    const int pframes = d.probe_stride ? pb.W * nwin : nwin;
    tma = frame_map(&tm.u, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, d.u, S, pb.W * nwin, kTR, kTC) &&
          frame_map(&tm.f0, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, pb.optimize ? d.fld0 : nullptr, S,
                    pb.W * nwin, kTR, kTC) &&
          frame_map(&tm.f2, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, pb.optimize ? d.fld2 : nullptr, S,
                    pb.W * nwin, kTR, kTC) &&
          frame_map(&tm.d2, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, d.ncopies > 1 ? d.d2code : nullptr,
                    S, pframes, kTRP, kTC);
  }
  if (tma) {
    constexpr int GSS = NC * 16 + 16;
    const size_t shm = (size_t)32 * GSS * 4 + (size_t)NC * kTile * 4 + 128;
    const cudaError_t e = cudaFuncSetAttribute(
        k_bout_tma<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm);
    if (e != cudaSuccess) return e;
    k_bout_tma<NC><<<(nitems + 31) / 32, 128, shm, s>>>(pb, d, nitems, tm);
  } else {
    k_bout<NC><<<(nitems + 31) / 32, 128, 0, s>>>(pb, d, nitems);
  }
  return cudaGetLastError();
}

template cudaError_t run_svd_split<10>(const Problem&, const DeviceBuffers&, cudaStream_t, bool);
template cudaError_t run_svd_split<16>(const Problem&, const DeviceBuffers&, cudaStream_t, bool);

}  // namespace svdk
}  // namespace pgsvt
