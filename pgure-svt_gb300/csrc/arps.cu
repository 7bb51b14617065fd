// arps.cu — ARPS block matching on the GPU with motion vectors identical to
// the reference's FP64 MotionEstimator (arps.hpp:52-375).
//
// One thread runs one motion-slot chain (<= 2 frame pairs that share a slot of
// the reference's `motions` cube, arps.hpp:121-130) for one grid position.
// Block costs (mean squared difference, arps.hpp:148-151) are computed in FP32
// from the normalised window together with a rigorous bound on their distance
// to the FP64 value; whenever the FP32 argmin of a diamond step is not certain
// under those bounds, every candidate of that step is recomputed exactly as the
// reference does (FP64 x/umax, FP64 squares, Armadillo's two-accumulator
// accu(), no fused multiply-add) and the FP64 argmin is taken.  The decisions,
// hence the motion vectors, are therefore the FP64 ones.
#include <cstring>

#include "pgsvt_internal.h"

namespace pgsvt {

namespace {


// How a block cost is computed.  kFloat: FP32 with an error bound.  Integer-
// valued input (at most 2^19) has exact sums of squared differences instead: in
// FP32 where m * max^2 <= 2^24 (kIntF), else in 64-bit integers (kInt64).
enum { kFloat, kIntF, kInt64 };

template <int MODE>
struct CostT { using type = float; };
template <>
struct CostT<kInt64> { using type = unsigned long long; };

struct ArpsCtx {
  const float* fa1;   // slices a1 and a2 that the costs read: the normalised
  const float* fa2;   // window, or the raw integers
  const float* xa1;   // input frames (exact f32 values) for the FP64 path
  const float* xa2;
  const double* xa1d; // input frames when the input is f64
  const double* xa2d;
  const double* pa1;  // FP64 normalised slices when precomputed (median
  const double* pa2;  // pre-filter: ties are frequent), else null
  double umax;
  int S;
  int mw;
  int bs;             // patch side (used when the kernel is not specialised)
};

// The reference block of one position.  BS > 0: its values in registers;
// BS == 0 (patch sides above 8): read from the frame where needed.
template <int BS, int MODE>
struct Block {
  using T = typename CostT<MODE>::type;
  float ref[BS > 0 ? BS * BS : 1];  // normalised values, or the raw integers
  const float* src = nullptr;       // BS == 0: the block's first element
  int S = 0;
  float a2 = 0.f;                   // kFloat: the sum of its squares

  __device__ __forceinline__ float at(int e, int nb) const {
    if constexpr (BS > 0) return ref[e];
    else return __ldg(src + (e % nb) + (size_t)(e / nb) * S);
  }

  __device__ void load(const ArpsCtx& c, int i, int j) {
    const float* sp = c.fa1 + (i + j * c.S);
    if constexpr (BS > 0) {
#pragma unroll
      for (int cc = 0; cc < BS; ++cc)
#pragma unroll
        for (int r = 0; r < BS; ++r) ref[r + cc * BS] = __ldg(sp + r + cc * c.S);
    } else {
      src = sp;
      S = c.S;
    }
    if constexpr (MODE == kFloat) {
      const int nb = BS > 0 ? BS : c.bs;
      for (int e = 0; e < nb * nb; ++e) a2 = fmaf(at(e, nb), at(e, nb), a2);
    }
  }

  // Cost of the candidate at offset off (row + column * S), with a bound on its
  // error.
  //
  // Integers: the exact sum of squared differences D.  The reference's
  // FP64 cost is D / (umax^2 m) up to an absolute error below
  // (m + 7) 2^-53 (values <= 1 after normalisation), while two different D
  // differ by at least 1 / (umax^2 m) > 2 (m + 7) 2^-53 for umax <= 2^19 and
  // m <= 64, or umax <= 2^17 and m <= 256 (the host enables the mode only
  // then): comparing D decides exactly as the reference does, except for
  // equal D.
  //
  // kFloat: a bound on |cost32 - cost64| (u = 2^-24, m = bs^2): the
  // FP32 operands differ from the reference's FP64 ones by <= 2u|a| (the
  // normalisation divides by the FP32-rounded maximum), so every difference
  // by <= 3u(|a|+|b|) and every square by <= 6u(|a|+|b|)^2; the m-term FMA
  // sum adds <= m u sum d^2 = m^2 u cost.  (|a|+|b|)^2 <= (2|a|+|d|)^2 <= 8a^2 + 2d^2
  // bounds the first sum by the reference block's squares and the cost itself
  // (adding the terms up per candidate took half of the arithmetic).  With
  // margin:
  //   err = u * (8 * (8 sum a^2 + 2 sum d^2) / m + (m + 4) * cost)
  __device__ __forceinline__ void cost(const ArpsCtx& c, int off, T& cst, float& err) const {
    const int nb = BS > 0 ? BS : c.bs;
    const float* sp = c.fa2 + off;
    if constexpr (MODE == kInt64) {
      unsigned long long acc = 0ull;
#pragma unroll
      for (int cc = 0; cc < nb; ++cc)
#pragma unroll
        for (int r = 0; r < nb; ++r) {
          const float d = at(r + cc * nb, nb) - __ldg(sp + r + cc * c.S);  // exact, |d| <= 2^19
          const int di = __float_as_int(d + 12582912.f) - 0x4B400000;      // 1.5 * 2^23
          acc += (unsigned long long)((long long)di * di);
        }
      cst = acc;
      err = 0.f;
    } else {
      float acc = 0.f;
#pragma unroll
      for (int cc = 0; cc < nb; ++cc)
#pragma unroll
        for (int r = 0; r < nb; ++r) {
          const float d = at(r + cc * nb, nb) - __ldg(sp + r + cc * c.S);
          acc = fmaf(d, d, acc);
        }
      if constexpr (MODE == kIntF) {
        cst = acc;
        err = 0.f;
      } else {
        const float m = (float)(nb * nb), oo = 1.0f / m;
        cst = acc * oo;
        err = 5.9604645e-8f * (8.f * (8.f * a2 + 2.f * acc) * oo + (m + 4.f) * cst);
      }
    }
  }

  // the candidate block at offset o equals the one at o2, element by element
  __device__ bool same(const ArpsCtx& c, int o, int o2) const {
    const int nb = BS > 0 ? BS : c.bs;
    bool eq = true;
#pragma unroll
    for (int cc = 0; cc < nb; ++cc)
#pragma unroll
      for (int r = 0; r < nb; ++r)
        eq &= __ldg(c.fa2 + o + r + cc * c.S) == __ldg(c.fa2 + o2 + r + cc * c.S);
    return eq;
  }
};

// Offset of slot k of a diamond of half-width st around the current position;
// slot 5 is the predicted motion (mx, my).
struct Diamond {
  int st, mx, my;
  __device__ __forceinline__ int dx(int k) const {
    return k == 1 ? -st : (k == 3 ? st : (k == 5 ? mx : 0));
  }
  __device__ __forceinline__ int dy(int k) const {
    return k == 0 ? -st : (k == 4 ? st : (k == 5 ? my : 0));
  }
};

__device__ __forceinline__ double src64(const ArpsCtx& c, const float* xf, const double* xd,
                                        size_t idx) {
  return xd ? xd[idx] : (double)xf[idx];
}

// Per-warp scratch of the exact (FP64) decisions.
template <int BS>
struct ArpsWarp {
  static constexpr int kSq = 256;  // squared differences per pass
  double sq[kSq];
  double cst[32 * 6];     // exact cost per (lane, slot)
  uint32_t pos[32 * 6];   // candidate (y, x) per (lane, slot), 16 bits each
  uint32_t blk[32];       // reference block (i, j) per lane, 16 bits each
  uint16_t cand[32 * 6];  // the warp's candidates to evaluate: lane * 6 + slot
};

// Exact reference costs (arps.hpp:148-151 as the reference evaluates them:
// FP64 x/umax, FP64 squares, Armadillo's two-accumulator accu(), no fused
// multiply-add) of every slot in `em` of every lane, computed by the whole
// warp at once: the squared differences of all candidate blocks are spread
// over the lanes, and the even- and odd-element accumulators of every
// candidate are summed in element order by two lanes.  The FP64 pipe runs a
// warp instruction at a fraction of the FP32 rate whatever its active lanes,
// so this takes a small part of the FP64 instructions (and of the latency) of
// per-thread evaluations.  Results in ws.cst[lane * 6 + slot].
template <int BS>
__device__ __noinline__ void warp_cost64(const ArpsCtx& c, ArpsWarp<BS>& ws, unsigned em, int i,
                                         int j, int y, int x, const Diamond dm, int nslot) {
  const int lane = threadIdx.x & 31;
  const int nb = BS > 0 ? BS : c.bs;
  const int m = nb * nb;
  const double oo = 1.0 / (double)m;
  // this lane's candidates, and their place in the warp's list
  const int mine = __popc(em);
  int first = mine;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, first, o);
    if (lane >= o) first += t;
  }
  const int total = __shfl_sync(0xffffffffu, first, 31);
  first -= mine;
  if (em) {
    ws.blk[lane] = ((uint32_t)i & 0xffffu) | ((uint32_t)j << 16);
    int r = first;
    for (int k = 0; k < nslot; ++k) {
      if (!((em >> k) & 1u)) continue;
      ws.pos[lane * 6 + k] = ((uint32_t)(y + dm.dy(k)) & 0xffffu) | ((uint32_t)(x + dm.dx(k)) << 16);
      ws.cand[r++] = (uint16_t)(lane * 6 + k);
    }
  }
  __syncwarp();
  const int per = min(16, ArpsWarp<BS>::kSq / m);  // two summing lanes per candidate
  for (int c0 = 0; c0 < total; c0 += per) {
    const int cn = min(per, total - c0);
    for (int t = lane; t < cn * m; t += 32) {
      const int cd = ws.cand[c0 + t / m];
      const int e = t % m, r = e % nb, cc = e / nb;
      const uint32_t pb = ws.blk[cd / 6], pk = ws.pos[cd];
      const int bi = (int)(pb & 0xffffu), bj = (int)(pb >> 16);
      const int py = (int)(pk & 0xffffu), px = (int)(pk >> 16);
      const size_t ka = (bi + r) + (size_t)(bj + cc) * c.S;
      const size_t kb = (py + r) + (size_t)(px + cc) * c.S;
      const double a = c.pa1 ? c.pa1[ka] : __ddiv_rn(src64(c, c.xa1, c.xa1d, ka), c.umax);
      const double b = c.pa2 ? c.pa2[kb] : __ddiv_rn(src64(c, c.xa2, c.xa2d, kb), c.umax);
      const double d = __dsub_rn(a, b);
      ws.sq[t] = __dmul_rn(d, d);
    }
    __syncwarp();
    double v = 0.0;
    if (lane < 2 * cn) {
      const double* q = ws.sq + (lane >> 1) * m;
      for (int e = lane & 1; e < m; e += 2) v = __dadd_rn(v, q[e]);
    }
    const double v2 = __shfl_down_sync(0xffffffffu, v, 1);
    if (lane < 2 * cn && !(lane & 1))
      ws.cst[ws.cand[c0 + (lane >> 1)]] = __dmul_rn(__dadd_rn(v, v2), oo);
    __syncwarp();
  }
}

// The slot chosen from the exact costs of the slots em: integer mode, the
// first of the least cost among the tied slots; otherwise the first index of
// the minimum over every evaluated slot (unevaluated ones count as 1e9).
__device__ int resolve_exact(bool integer, const double* cst, unsigned em, int nslot) {
  if (integer) {
    int kb = -1;
    double mm = 0.0;
    for (int k = 0; k < nslot; ++k) {
      if (!((em >> k) & 1u)) continue;
      if (kb < 0 || cst[k] < mm) {
        mm = cst[k];
        kb = k;
      }
    }
    return kb;
  }
  double c64[6];
  for (int k = 0; k < nslot; ++k) c64[k] = ((em >> k) & 1u) ? cst[k] : 1e9;
  double mm = c64[0];
  for (int k = 1; k < nslot; ++k) mm = fmin(mm, c64[k]);
  for (int k = 0; k < nslot; ++k)
    if (c64[k] == mm) return k;
  return 2;
}

// The slot of a step from the costs of the evaluated slots (bits of ev, slot 2
// always), or -1 with the slots to evaluate exactly in em.
//
// Integers: first index of the least D; equal D decided as the
// reference does: identical candidate blocks have identical FP64 costs (the
// first one wins; D = 0 are all copies of the reference block), otherwise the
// FP64 costs of the tied candidates decide.
//
// kFloat: first index of the minimum when the FP32 decision is certain under the
// error bounds, else every evaluated slot is to be evaluated exactly.
template <int BS, int MODE, class T>
__device__ __forceinline__ int decide(const ArpsCtx& c, const Block<BS, MODE>& blk, const T (&cs)[6],
                                      const float (&es)[6], unsigned ev, const Diamond& dm, int off,
                                      unsigned& em) {
  int ks = 2;
  T best = cs[2];
  float ebest = es[2];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    if (k == 2) continue;
    if (((ev >> k) & 1u) && (cs[k] < best || (cs[k] == best && k < ks))) {
      best = cs[k];
      ebest = es[k];
      ks = k;
    }
  }
  if constexpr (MODE == kFloat) {
    bool certain = true;
    const float hi = best + ebest;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      if (!((ev >> k) & 1u) || k == ks) continue;
      const float lo = cs[k] - es[k];
      if (k < ks ? !(lo > hi) : !(lo >= hi)) certain = false;
    }
    if (certain) return ks;
    em = ev;
    return -1;
  } else {
    unsigned tied = 0u;
#pragma unroll
    for (int k = 0; k < 6; ++k)
      if (((ev >> k) & 1u) && cs[k] == best) tied |= 1u << k;
    if (best == (T)0 || !(tied & (tied - 1u))) return ks;
    bool distinct = false;
    const int o2 = off + dm.dy(ks) + dm.dx(ks) * c.S;
    for (unsigned t = tied & ~(1u << ks); t; t &= t - 1u) {
      const int k = __ffs(t) - 1;
      if (!blk.same(c, off + dm.dy(k) + dm.dx(k) * c.S, o2)) distinct = true;
    }
    if (!distinct) return ks;
    em = tied;
    return -1;
  }
}

// ARPSMotionEstimation (arps.hpp:153-375) for one position of one frame pair.
// (my, mx) holds the predictor slot on entry and the new motion on exit.
// The lanes of a warp step through the diamond searches together (a lane
// whose search ended, or that holds no position, idles), so that the exact
// decisions any of them needs are taken by the whole warp.  `seen`: this
// thread's bitmap of visited cells, word q at seen[q * 128].
template <int BS, int MODE>
__device__ void arps_pair(const ArpsCtx& c, bool live, int it, int& my, int& mx, int& oy,
                          int& ox, ArpsWarp<BS>& ws, uint32_t* seen, unsigned& nexact) {
  using T = typename CostT<MODE>::type;
  const int lane = threadIdx.x & 31;
  const int S = c.S, M = c.mw, Wd = 2 * M + 1;
  const int nb = BS > 0 ? BS : c.bs;
  const int n1 = S - nb + 1;
  const int i = it % n1, j = it / n1;
  Block<BS, MODE> blk;
  blk.load(c, i, j);
  const int nw = (Wd * Wd + 31) / 32;
  for (int q = 0; q < nw; ++q) seen[q * 128] = 0u;
  int x = j, y = i;
  T cs[6];
  float es[6];
  blk.cost(c, i + j * S, cs[2], es[2]);
  {
    const int b = M * Wd + M;
    seen[(b >> 5) * 128] |= 1u << (b & 31);
  }
  // step 0 is the LDSP (arps.hpp:247-294), steps 1.. the SDSP (arps.hpp:299-368):
  // the same diamond, of the predictor's length and of 1, the first with the
  // predicted motion as a sixth candidate when it is off the axes and without
  // the search window's limits.  Every SDSP move enters an unvisited cell, so a
  // search ends within Wd*Wd moves.
  Diamond dm{2, 0, 0};
  bool six = false;
  if (j > 0) {
    const int ay = abs(my), ax = abs(mx);
    dm.st = (ax <= ay) ? ay : ax;
    six = !((ay == 0 && ax == dm.st) || (ax == 0 && ay == dm.st));
    dm.mx = mx;
    dm.my = my;
  }
  bool done = !live;
  for (int n = 0; n <= Wd * Wd + 1; ++n) {
    unsigned ev = 4u;
    if (!done) {
      const int o = y + x * S;
      auto slot = [&](int k, T& ck, float& ek) {  // cost of slot k, if it is a candidate
        const int ddx = dm.dx(k), ddy = dm.dy(k);
        const int hx = x + ddx, vy = y + ddy;
        bool ok = hx >= 0 && vy >= 0 && hx + nb <= S && vy + nb <= S;
        const int wy = vy - i, wx = hx - j;  // cell of the search window
        const bool in = wy >= -M && wy <= M && wx >= -M && wx <= M;
        const int b = (wy + M) * Wd + (wx + M);
        if (n > 0) ok = ok && in && !((seen[(b >> 5) * 128] >> (b & 31)) & 1u);
        if (!ok) return;
        blk.cost(c, o + ddy + ddx * S, ck, ek);
        ev |= 1u << k;
        if (in) seen[(b >> 5) * 128] |= 1u << (b & 31);
      };
      if (dm.st != 0) {
        if constexpr (BS > 0 && BS <= 4) {
#pragma unroll
          for (int k = 0; k < 5; ++k)
            if (k != 2) slot(k, cs[k], es[k]);
        } else {  // one copy of the cost code for the larger blocks
#pragma unroll 1
          for (int k = 0; k < 5; ++k) {
            if (k == 2) continue;
            T ck = (T)0;
            float ek = 0.f;
            slot(k, ck, ek);
#pragma unroll
            for (int q = 0; q < 5; ++q)
              if (q != 2 && q == k) {
                cs[q] = ck;
                es[q] = ek;
              }
          }
        }
      }
      if (n == 0 && six) slot(5, cs[5], es[5]);
    }
    int ks = 2;
    unsigned em = 0u;
    if (!done) ks = decide<BS, MODE>(c, blk, cs, es, ev, dm, y + x * S, em);
    if (__any_sync(0xffffffffu, em != 0u)) {
      const int nslot = n == 0 ? 6 : 5;
      warp_cost64<BS>(c, ws, em, i, j, y, x, dm, nslot);
      if (em) {
        ks = resolve_exact(MODE != kFloat, ws.cst + lane * 6, em, nslot);
        ++nexact;
      }
      __syncwarp();
    }
    if (!done) {
      x += dm.dx(ks);
      y += dm.dy(ks);
#pragma unroll
      for (int k = 0; k < 6; ++k)
        if (k != 2 && k == ks) {
          cs[2] = cs[k];
          es[2] = es[k];
        }
      if (n > 0 && ks == 2) done = true;
    }
    dm.st = 1;
    if (!__any_sync(0xffffffffu, !done)) break;
  }
  my = y - i;
  mx = x - j;
  oy = y;
  ox = x;
}

// Chain table of a batch in the kernel's parameters: its entries and the frame
// addresses that follow from them are uniform over a block.
struct ArpsTable {
  ArpsChain c[kArpsChains];
};

// Resident blocks per SM.  The walks of a warp diverge, so more warps hide more of
// their latency until the costs spill: patches of up to 4 x 4 pixels take 6 blocks
// (80 registers; 256 x 256 x 100 floats 11.1 -> 10.8 ms, 7 blocks 11.9) and, with
// integer costs, 7 (72; median-filtered 512 x 512 x 40 80.1 -> 69.4 ms, 6 blocks 74.4,
// 8 blocks 77.9), larger ones 5 (8 x 8 patches, bytes, 6.6 ms; 6 blocks 7.7).
template <int BS, int MODE>
constexpr int arps_blocks() {
  return BS >= 1 && BS <= 4 && MODE != kInt64 ? (MODE == kIntF ? 7 : 6) : 5;
}

// Bound by the instructions of the costs and their loads (nine tenths of them hit
// L1).  GB300, against one form with runtime candidate lists, 64-bit integer sums
// and per-candidate error sums: 256 x 256 x 100 floats 17.9 -> 10.8 ms; 256 x 256 x
// 24 bytes, 8 x 8 patches, 19.0 -> 6.6 ms; median-filtered 512 x 512 x 40 (two thirds
// of it exact tie decisions) 115 -> 69 ms.
template <int BS, int MODE>
__global__ void __launch_bounds__(128, arps_blocks<BS, MODE>())
    k_arps(Problem pb, DeviceBuffers d, const __grid_constant__ ArpsTable tab) {
  const Geometry& g = pb.g;
  const int it0 = blockIdx.x * blockDim.x + threadIdx.x;
  const int ch = blockIdx.y, w = blockIdx.z;
  const ArpsChain& cn = tab.c[w * d.nchains + ch];
  const int npairs = cn.npairs;
  if (npairs == 0) return;  // uniform over the block
  const bool live = it0 < g.P;
  const int it = live ? it0 : 0;
  __shared__ ArpsWarp<BS> wsh[4];
  extern __shared__ uint32_t seen[];  // [words][128]
  ArpsWarp<BS>& ws = wsh[threadIdx.x >> 5];
  const WinConst& wc = d.wc[w];
  const size_t F = g.F();
  // ARPS input: the median-filtered window when the pre-filter is on
  // (its values are integers, exact in FP32), else the window itself
  const bool med = d.zs != nullptr;
  const float* fw = med ? d.wz : d.u;
  const float* xw = med ? d.zs : d.xs;
  const double* xd = med ? nullptr : d.x64;
  ArpsCtx c;
  c.bs = g.bs;
  c.umax = med ? wc.wnorm : wc.unorm;
  c.S = g.S;
  c.mw = g.mw;
  int my = 0, mx = 0;
  unsigned nexact = 0u;
  for (int q = 0; q < npairs; ++q) {
    const int a1 = cn.a1[q], a2 = cn.a2[q];
    c.xa1 = xw + (size_t)(wc.s0 + a1) * F;
    c.xa2 = xw + (size_t)(wc.s0 + a2) * F;
    if constexpr (MODE == kFloat) {
      c.fa1 = fw + ((size_t)w * g.nwin + a1) * F;
      c.fa2 = fw + ((size_t)w * g.nwin + a2) * F;
    } else {
      c.fa1 = c.xa1;
      c.fa2 = c.xa2;
    }
    c.xa1d = xd ? xd + (size_t)(wc.s0 + a1) * F : nullptr;
    c.xa2d = xd ? xd + (size_t)(wc.s0 + a2) * F : nullptr;
    c.pa1 = d.w64 ? d.w64 + ((size_t)w * g.nwin + a1) * F : nullptr;
    c.pa2 = d.w64 ? d.w64 + ((size_t)w * g.nwin + a2) * F : nullptr;
    int oy, ox;
    arps_pair<BS, MODE>(c, live, it, my, mx, oy, ox, ws, seen + threadIdx.x, nexact);
    if (live) d.pos[((size_t)w * g.nwin + a2) * g.P + it] = (uint32_t)oy | ((uint32_t)ox << 16);
  }
  for (int o = 16; o > 0; o >>= 1) nexact += __shfl_xor_sync(0xffffffffu, nexact, o);
  if ((threadIdx.x & 31) == 0 && nexact) atomicAdd(d.counters, (unsigned long long)nexact);
}

template <int MODE>
void launch_k_arps(dim3 grid, size_t shm, const Problem& pb, const DeviceBuffers& d,
                   const ArpsTable& tab, cudaStream_t s) {
  switch (pb.g.bs) {
    case 2: k_arps<2, MODE><<<grid, 128, shm, s>>>(pb, d, tab); break;
    case 3: k_arps<3, MODE><<<grid, 128, shm, s>>>(pb, d, tab); break;
    case 4: k_arps<4, MODE><<<grid, 128, shm, s>>>(pb, d, tab); break;
    case 5: k_arps<5, MODE><<<grid, 128, shm, s>>>(pb, d, tab); break;
    case 6: k_arps<6, MODE><<<grid, 128, shm, s>>>(pb, d, tab); break;
    case 7: k_arps<7, MODE><<<grid, 128, shm, s>>>(pb, d, tab); break;
    case 8: k_arps<8, MODE><<<grid, 128, shm, s>>>(pb, d, tab); break;
    default: k_arps<0, MODE><<<grid, 128, shm, s>>>(pb, d, tab); break;  // sides 9..16
  }
}

// Reference slice (always) and, without motion estimation, the other slices:
// (0,0) in compat mode (arps.hpp:42), else the grid position.
__global__ void k_grid(Problem pb, DeviceBuffers d) {
  const Geometry& g = pb.g;
  const int it = blockIdx.x * blockDim.x + threadIdx.x;
  const int k = blockIdx.y, w = blockIdx.z;
  if (it >= g.P) return;
  const int ref = d.wc[w].ref;
  const int n1 = g.S - g.bs + 1;
  const uint32_t grid = (uint32_t)(it % n1) | ((uint32_t)(it / n1) << 16);
  uint32_t v;
  if (k == ref) v = grid;
  else if (pb.motion) return;  // written by k_arps
  else v = (pb.compat & 0x2) ? 0u : grid;
  d.pos[((size_t)w * g.nwin + k) * g.P + it] = v;
}

}  // namespace

cudaError_t launch_arps(const Problem& pb, const DeviceBuffers& d, cudaStream_t s) {
  const Geometry& g = pb.g;
  const int threads = 128;
  dim3 gg((g.P + threads - 1) / threads, g.nwin, pb.W);
  k_grid<<<gg, threads, 0, s>>>(pb, d);
  if (!pb.motion || d.nchains == 0) return cudaGetLastError();
  dim3 ga((g.P + threads - 1) / threads, d.nchains, pb.W);
  if (pb.W * d.nchains > kArpsChains) return cudaErrorInvalidValue;
  ArpsTable tab;
  std::memcpy(tab.c, d.chains, sizeof(ArpsChain) * pb.W * d.nchains);
  const int wd = 2 * g.mw + 1;
  const size_t shm = (size_t)((wd * wd + 31) / 32) * 128 * sizeof(uint32_t);
  if (!d.zs && !d.int_input) launch_k_arps<kFloat>(ga, shm, pb, d, tab, s);
  else if ((double)g.M * d.arps_max * d.arps_max <= 16777216.0)
    launch_k_arps<kIntF>(ga, shm, pb, d, tab, s);
  else launch_k_arps<kInt64>(ga, shm, pb, d, tab, s);
  return cudaGetLastError();
}

}  // namespace pgsvt
