// eval.cu — singular-value thresholding, overlap averaging and the PGURE risk.
//
// Reference: SVT::Reconstruct (svt.hpp:121-167), PGURE::CalculatePGURE
// (pgure.hpp:120-137) and the lambda search driven by PGURE::Optimize
// (pgure.hpp:197-237).
//
// The risk of one window at lambda is
//   R = (1/N) [ sum (Uh-U)^2 - (a+m) sum U + (2/e1) sum d1 (aU-am+s^2)(U1-Uh)
//               - (2 s^2 a / e2^2) sum d2 (U2p - 2 Uh + U2m) + 2 m sum Uh + m ] - s^2
// (a, m, s are PGURE's alpha, mu, sigma members).  Every term except the first
// is linear in a reconstructed cube, and each reconstructed cube is an
// overlap average Uc = (sum_p scatter(R_p)) / cnt with R_p = sum_i g_i u_i v_i^T.
// Hence  sum_x L(x) Uc(x) = sum_p sum_i g_i (u_i^T G_p v_i)  with the
// lambda-independent field G = L / cnt gathered along patch p's trajectory:
// the SVD epilogue stores h_i = u_i^T G_p v_i once, and a lambda evaluation
// needs only sum_i g_i(lambda) h_i per patch and copy.  Only sum (Uh-U)^2 needs
// the clean reconstruction voxel by voxel: copy 0 is rebuilt and scattered
// into a fixed-point accumulator (int32 at 2^-20, or int64 at 2^-32 when one
// voxel can collect every patch, as with the zero-motion quirk), which makes
// the sums independent of the order of the atomics, so the whole search is
// deterministic.
#include <algorithm>

#include <map>
#include <mutex>
#include <utility>

#include "pgsvt_internal.h"

namespace pgsvt {

namespace {

__device__ __forceinline__ double warp_sum_d(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---- lambda-independent fields and sum(U)
//
// With the integer-delta1 quirk a voxel's fields depend on its coverage and its
// probe code only: k_field_table tabulates them in FP64 for the coverages below
// kFieldTab (the FP64 pipe, at 1/64 of the FP32 rate, was what bounded the
// kernel: a division and ten products per voxel); what is left in FP64 per voxel
// is sum(U).  Two windows of 512 x 512 x 15, GB300: 0.27 -> 0.10 ms.  Without the risk
// there are no fields, and nothing reads sum(U).
constexpr int kFieldTab = 256;

// (field 0, field 2) of a voxel covered n times
__device__ __forceinline__ float2 field_entry(const WinConst& wc, double dl2, int n) {
  const double a = wc.alpha, m = wc.mu, s2 = wc.sigma * wc.sigma;
  const double c2 = 2 * s2 * a / (wc.eps2 * wc.eps2);
  const double ic = n > 0 ? 1.0 / n : 0.0;
  const double l0 = 2 * c2 * dl2 + 2 * m;
  return make_float2((float)(l0 * ic), (float)(-c2 * dl2 * ic));
}

// [window][probe code][coverage]
__global__ void __launch_bounds__(kFieldTab) k_field_table(Problem pb, DeviceBuffers d) {
  const int w = blockIdx.y, code = blockIdx.x;
  d.ftab[((size_t)w * 2 + code) * kFieldTab + threadIdx.x] =
      field_entry(d.wc[w], code ? d.d2neg : d.d2pos, threadIdx.x);
}

__global__ void __launch_bounds__(256) k_fields(Problem pb, DeviceBuffers d) {
  const Geometry& g = pb.g;
  const int w = blockIdx.y;
  const size_t C = g.cube();
  const WinConst& wc = d.wc[w];
  const float* u = d.u + (size_t)w * C;
  const int32_t* cnt = d.cnt + (size_t)w * C;
  const bool intd1 = pb.compat & 0x4;
  const int8_t* d1 = d.d1 + (size_t)w * d.probe_stride;
  const int8_t* d2c = d.d2code + (size_t)w * d.probe_stride;
  const float2* tab = d.ftab + (size_t)w * 2 * kFieldTab;
  double su = 0.0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < C;
       i += (size_t)gridDim.x * blockDim.x) {
    const double uv = u[i];
    su += uv;
    const int n = cnt[i];
    const bool code = d2c[i] != 0;
    if (intd1) {
      const float2 f = n < kFieldTab ? __ldg(tab + code * kFieldTab + n)
                                     : field_entry(wc, code ? d.d2neg : d.d2pos, n);
      d.fld0[(size_t)w * C + i] = f.x;
      d.fld2[(size_t)w * C + i] = f.y;
      continue;
    }
    const double a = wc.alpha, m = wc.mu, s2 = wc.sigma * wc.sigma;
    const double c2 = 2 * s2 * a / (wc.eps2 * wc.eps2);
    const double ic = n > 0 ? 1.0 / n : 0.0;
    const double dl2 = code ? d.d2neg : d.d2pos;
    const double l1 = (2 / wc.eps1) * d1[i] * ((a * uv - a * m) + s2);
    const double l0 = 2 * c2 * dl2 + 2 * m - l1;
    d.fld1[(size_t)w * C + i] = (float)(l1 * ic);
    d.fld0[(size_t)w * C + i] = (float)(l0 * ic);
    d.fld2[(size_t)w * C + i] = (float)(-c2 * dl2 * ic);
  }
  su = warp_sum_d(su);
  __shared__ double sm[32];
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = su;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) t += sm[q];
    d.part_mse[(size_t)w * gridDim.x + blockIdx.x] = t;  // reused as scratch
  }
}
constexpr int kFieldBlocks = 256;  // per window

// ---- search state machine (one block per window, thread 0 decides)
//
// Bracketed batch grid search, identical to the oracle's: round 0 places K
// points geometrically over [lo, hi]; each later round places K/2 points
// evenly inside the bracket formed by the neighbours of the best point so far
// (K points in a narrow search, or when the bracket reaches down to zero).  A
// hint (a given or learned proposal) runs a narrow search first: hint_K
// points over [hint/span, hint*span] and hint_rounds refinements.  When the
// best point of its grid lies on an edge and the neighbouring point's risk
// is more than hint_flat (relative) above it, the plain search runs instead
// and the better of the two results is kept.

struct Sch {
  // grid point j of K from lo to hi
  __device__ static double point(int j, int K, double lo, double hi) {
    return (K == 1) ? hi : lo * pow(hi / lo, (double)j / (double)(K - 1));
  }
  __device__ static void grid(SearchState& s, double lo, double hi) {
    const int K = s.K;
    for (int j = 0; j < K; ++j) s.next[j] = point(j, K, lo, hi);
    s.nnext = K;
    s.first = 1;
  }
  // batch_search's set-up: K shrinks to the evaluation budget
  __device__ static void phase(SearchState& s, int ph, int K0, int max_eval, int rounds,
                               int zero_lo) {
    s.phase = ph;
    s.K = (max_eval < K0) ? max(1, max_eval) : K0;
    s.max_eval = max_eval;
    s.rounds = rounds;
    s.zero_lo = zero_lo;
    s.rd = 0;
    s.evals_phase = 0;
    s.npts = 0;
    s.best = 0;
    s.nsent = 0;
    s.sent_risk = INFINITY;
  }
  __device__ static int best(const SearchState& s) {
    int b = 0;
    for (int i = 1; i < s.npts; ++i)
      if (s.risk[i] < s.risk[b]) b = i;
    return b;
  }
};

// The narrow grid inherits the plain search's bounds: a grid reaching below
// the plain grid's bottom (upper * 1e-4) may refine down to 0 as the plain
// search does, and a grid clipped at `upper` ends there as the plain one
// does; a best point on such a bound is a result, not a miss.  Its first
// round also evaluates the plain grid's ends that it does not reach
// (sentinels, kept out of the point list): one of them below the narrow
// grid's best sends the search to the plain grid.
// Called by the threads of a block; each point's pow() runs in its own thread.
__device__ void start_narrow(SearchState& s, const Problem& pb, double upper, double hint) {
  const double h = fmin(hint, upper);
  const double lo = h / pb.hint_span, hi = fmin(upper, h * pb.hint_span);
  if (threadIdx.x == 0) {
    Sch::phase(s, 1, pb.hint_K, pb.max_evals, pb.hint_rounds, lo <= upper * 1e-4 ? 1 : 0);
    s.nnext = s.K;
    s.first = 1;
    const int room = min(pb.K - s.nnext, pb.max_evals - s.nnext);
    if (room > 0 && lo > upper * 1e-4) s.next[s.nnext + s.nsent++] = upper * 1e-4;
    if (room > s.nsent && hi < upper) s.next[s.nnext + s.nsent++] = upper;
    s.nnext += s.nsent;
  }
  __syncthreads();
  if (threadIdx.x < s.K) s.next[threadIdx.x] = Sch::point(threadIdx.x, s.K, lo, hi);
}

// sum(U) of the window from k_fields' partials (in their order), the search's
// bounds and its first round
__global__ void __launch_bounds__(kFieldBlocks) k_search_init(Problem pb, DeviceBuffers d) {
  const int w = blockIdx.x;
  const Geometry& g = pb.g;
  WinConst& wc = d.wc[w];
  SearchState& s = d.st[w];
  __shared__ double part[kFieldBlocks];
  __shared__ double s_upper;
  part[threadIdx.x] = pb.optimize ? d.part_mse[(size_t)w * kFieldBlocks + threadIdx.x] : 0.0;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    if (pb.optimize) {
#pragma unroll 8
      for (int b = 0; b < kFieldBlocks; ++b) t += part[b];
    }
    wc.sum_u = t;
    s.npts = 0;
    s.nnext = 0;
    s.evals_total = 0;
    s.best = 0;
    s.final_lambda = pb.lambda_user;
    s.final_risk = 0.0;
    s.hint_lambda = s.hint_risk = 0.0;
    s.nsent = 0;
    s.sent_risk = INFINITY;
    s.done = pb.optimize ? 0 : 1;
    if (pb.optimize) {
      // pguresvt.hpp:139-141
      const double OoN = 1.0 / (double)((uint32_t)g.S * (uint32_t)g.S * (uint32_t)g.Ntc);
      double start = (pb.lambda_user >= 0.0) ? pb.lambda_user : t * OoN;
      start = fmax(0.0, start);
      wc.start = start;
      s_upper = wc.upper = fmax(100.0, start);
    }
  }
  __syncthreads();
  if (!pb.optimize) return;
  const double upper = s_upper;
  if (pb.nfixed > 0) {  // a given list: one round, no refinement
    if (threadIdx.x == 0) {
      Sch::phase(s, 0, pb.nfixed, pb.nfixed, 0, 0);
      for (int j = 0; j < pb.nfixed; ++j) s.next[j] = pb.fixed[j];
      s.nnext = pb.nfixed;
      s.first = 1;
    }
  } else if (pb.hint > 0) {
    start_narrow(s, pb, upper, pb.hint);
  } else {
    if (threadIdx.x == 0) {
      Sch::phase(s, 0, pb.K, pb.max_evals, pb.rounds, 1);
      s.nnext = s.K;
      s.first = 1;
    }
    __syncthreads();
    if (threadIdx.x < s.K) s.next[threadIdx.x] = Sch::point(threadIdx.x, s.K, upper * 1e-4, upper);
  }
}

// Narrow searches around the learned proposals y = log10(lambda/upper).
__global__ void __launch_bounds__(32) k_search_hint(Problem pb, DeviceBuffers d) {
  const int w = blockIdx.x;
  SearchState& s = d.st[w];
  if (s.done) return;
  const double upper = d.wc[w].upper;
  const double y = fmin(0.0, fmax(-6.0, (double)d.prop[w]));  // NaN -> -6
  start_narrow(s, pb, upper, upper * pow(10.0, y));
}

__device__ void search_finish(SearchState& s, unsigned long long* counters) {
  atomicAdd(counters + 3, (unsigned long long)s.evals_total);
  const int b = s.best;
  double lam = s.lam[b], risk = s.risk[b];
  if (s.phase == 2 && !(risk < s.hint_risk)) {
    lam = s.hint_lambda;
    risk = s.hint_risk;
  }
  s.final_lambda = lam;
  s.final_risk = risk;
  s.done = 1;
  s.nnext = 0;
}

// Merge the risks of the pending round and schedule the next one.
// One block per window: the partial sums of all its lambda values are reduced
// side by side, in four groups of 256 threads (each sum in the order of a
// 256-thread block: a strided sum per thread, then a tree), and thread 0 advances
// the search state.  Latency-bound: 512 x 512 x 15, 4 to 6 values, GB300: 30 -> 10 us
// (one sum after the other before).
constexpr int kStepGroups = 4;

__global__ void __launch_bounds__(256 * kStepGroups) k_search_step(Problem pb, DeviceBuffers d) {
  const int w = blockIdx.x;
  SearchState& s = d.st[w];
  if (s.done) return;
  __shared__ double red[kStepGroups][256];
  __shared__ double sums[2 * kMaxK];
  __shared__ double risk[kMaxK];
  const Geometry& g = pb.g;
  const WinConst& wc = d.wc[w];
  const int nn = s.nnext;
  const int grp = threadIdx.x >> 8, t = threadIdx.x & 255;
  for (int q0 = 0; q0 < 2 * nn; q0 += kStepGroups) {  // uniform over the block
    const int q = q0 + grp, j = q >> 1;
    if (q < 2 * nn) {
      const int n = (q & 1) ? d.nblk_mse : d.nblk_eval;
      const double* v = ((q & 1) ? d.part_mse : d.part_lin) + ((size_t)w * pb.K + j) * n;
      double x = 0.0;
#pragma unroll 8
      for (int i = t; i < n; i += 256) x += v[i];
      red[grp][t] = x;
    }
    __syncthreads();
    if (q < 2 * nn && t < 32) {
      const double* r = red[grp];
      double x = ((r[t] + r[t + 128]) + (r[t + 64] + r[t + 192])) +
                 ((r[t + 32] + r[t + 160]) + (r[t + 96] + r[t + 224]));
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (t == 0) sums[q] = x;
    }
    __syncthreads();
  }
  if (threadIdx.x < nn) {  // pgure.hpp:136
    const double N = (double)g.S * g.S * g.nwin;
    const double a = wc.alpha, m = wc.mu, s2 = wc.sigma * wc.sigma;
    risk[threadIdx.x] = (1.0 / N) * (sums[2 * threadIdx.x + 1] + sums[2 * threadIdx.x] -
                                     (a + m) * wc.sum_u + m) - s2;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  const double prev_best = s.npts > 0 ? s.risk[s.best] : 0.0;
  for (int j = nn - s.nsent; j < nn; ++j) s.sent_risk = fmin(s.sent_risk, risk[j]);
  for (int j = 0; j < nn - s.nsent; ++j) {
    int pos = s.npts;  // keep lambda ascending, new points after equal ones
    while (pos > 0 && s.lam[pos - 1] > s.next[j]) {
      s.lam[pos] = s.lam[pos - 1];
      s.risk[pos] = s.risk[pos - 1];
      --pos;
    }
    s.lam[pos] = s.next[j];
    s.risk[pos] = risk[j];
    ++s.npts;
  }
  s.evals_phase += s.nnext;
  s.evals_total += s.nnext;
  s.nnext = 0;
  const int b = Sch::best(s);
  s.best = b;
  const bool grid_round = s.first != 0;
  if (s.first) {
    s.first = 0;
    const bool bound = (b == 0 && s.zero_lo) || (b == s.npts - 1 && s.lam[b] >= wc.upper);
    const bool edge = (b == 0 || b == s.npts - 1) && !bound;
    bool steep = edge;
    if (edge && s.npts >= 2) {
      const int nb = (b == 0) ? 1 : s.npts - 2;
      steep = !(s.risk[nb] - s.risk[b] <= pb.hint_flat * fabs(s.risk[b]));
    }
    const bool beaten = s.sent_risk < s.risk[b];  // a plain-grid end does better
    s.nsent = 0;
    if (s.phase == 1 && (steep || beaten)) {  // proposal not bracketed: plain search
      s.hint_lambda = s.lam[b];
      s.hint_risk = s.risk[b];
      const int left = pb.max_evals > s.evals_phase ? pb.max_evals - s.evals_phase : 1;
      Sch::phase(s, 2, pb.K, left, pb.rounds, 1);
      Sch::grid(s, wc.upper * 1e-4, wc.upper);
      return;
    }
  } else {
    ++s.rd;
  }
  const double blo = (b > 0) ? s.lam[b - 1] : (s.zero_lo ? 0.0 : s.lam[b]);
  const double bhi = (b + 1 < s.npts) ? s.lam[b + 1] : s.lam[b];
  if (!grid_round && prev_best - s.risk[b] <= pb.tol * fabs(s.risk[b]) &&
      bhi - blo <= kNarrowBracket * s.lam[b]) {
    search_finish(s, d.counters);  // no progress and a narrow bracket
    return;
  }
  // refinement rounds of the plain search place half the grid's points,
  // unless the bracket reaches down to the zero bound
  const int Kr = (s.phase == 1 || (b == 0 && s.zero_lo)) ? s.K : max(2, s.K / 2);
  if (s.rd >= s.rounds || s.evals_phase + Kr > s.max_eval) {
    search_finish(s, d.counters);
    return;
  }
  if (!(bhi > blo)) {
    search_finish(s, d.counters);
    return;
  }
  for (int i = 0; i < Kr; ++i)
    s.next[i] = blo + (bhi - blo) * (double)(i + 1) / (double)(Kr + 1);
  s.nnext = Kr;
}

// ---- fixed-point accumulators
template <typename T>
struct Acc;
template <>
struct Acc<int> {  // 2^-20: one voxel holds |sum| < 2048
  static constexpr float kScale = 1048576.f;
  __device__ static int fix(float v) { return __float2int_rn(v * kScale); }
  __device__ static float unfix(int a) { return (float)a * (1.f / kScale); }
  __device__ static int from_tile(int t) { return t; }
  __device__ static void add(int* p, int v) { atomicAdd(p, v); }
};
template <>
struct Acc<unsigned long long> {  // 2^-32
  __device__ static long long fix(float v) { return fix32(v); }
  __device__ static float unfix(unsigned long long a) { return unfix32((long long)a); }
  __device__ static long long from_tile(int t) { return (long long)t * 4096; }
  __device__ static void add(unsigned long long* p, long long v) {
    atomicAdd(p, (unsigned long long)v);
  }
};

// ---- overlap sums of rebuilt blocks
//
// A warp holds 32 kept patches (an 8 x 4 half of an 8 x 8 tile of grid positions,
// see the patch order in capi.cu; one per lane).  Their rebuilt blocks in one
// slice overlap heavily, so the warp sums them in a shared-memory tile in
// int32 fixed point (2^-20, order-free) and adds the tile to the accumulator
// with one atomic per touched pixel.
// Its size is a launch's choice (eval_layout.h).
constexpr float kTileBound = 60.f;  // |value| above this bypasses the tile (32 x 60 < 2048)
constexpr float kMagicBound = 4.f;  // and below this value * 2^20 + 1.5 * 2^23 is exact

// The warp's footprint in one slice.  The tile's column stride is padded to 8
// (mod 16) where the footprint allows it, so that the warp's four 8-row lane
// groups (one grid column each) start 0, 8, 16, 24 (or 0, 24, 16, 8) banks apart.
struct Footprint {
  int y0, x0, th, ths, area;  // corner, rows, column stride, pixels
  bool tile;              // it fits the tile
  __device__ __forceinline__ void init(bool live, int y, int x, int nb, int tile_max) {
    // (frame sides are below 0x7fff; without a live lane the products stay in range)
    y0 = __reduce_min_sync(0xffffffffu, live ? y : 0x7fff);
    x0 = __reduce_min_sync(0xffffffffu, live ? x : 0x7fff);
    const int y1 = __reduce_max_sync(0xffffffffu, live ? y : -1);
    const int x1 = __reduce_max_sync(0xffffffffu, live ? x : -1);
    const int tw = x1 - x0 + nb;
    th = y1 - y0 + nb;
    ths = th <= 8 ? 8 : 8 + 16 * ((th - 8 + 15) / 16);
    if (y1 >= 0 && ths * tw > tile_max) ths = th;
    tile = y1 >= 0 && ths * tw <= tile_max;
    area = th * tw;
  }
};

// Add one lane's rebuilt rows e0 .. e0 + CH - 1 (column-major in the nb x nb
// block at (y, x)) to the tile or, where they do not fit, to the accumulator
// slice acc.  A value below kMagicBound becomes its fixed-point integer with
// one FMA (rounding to nearest even, as __float2int_rn rounds it).
template <int BS, int CH, typename AccT>
__device__ __forceinline__ void scatter(const float (&col)[CH], int e0, int nb, const Footprint& f,
                                        int* tile, AccT* acc, int S, int y, int x) {
  const int M = nb * nb;
  float mx = 0.f;
#pragma unroll
  for (int e = 0; e < CH; ++e)  // NaN stays NaN, and takes the second path
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(mx) : "f"(mx), "f"(fabsf(col[e])));
  if (mx == 0.f) return;
  if (f.tile && mx <= kMagicBound) {
    int* t = tile + (y - f.y0) + (x - f.x0) * f.ths;
#pragma unroll
    for (int e = 0; e < CH; ++e) {
      const int ee = e0 + e;
      if (ee >= M) continue;
      const int v = __float_as_int(fmaf(col[e], 1048576.f, 12582912.f)) - 0x4B400000;
      atomicAdd(t + ee % nb + (ee / nb) * f.ths, v);
    }
    return;
  }
#pragma unroll
  for (int e = 0; e < CH; ++e) {
    const int ee = e0 + e;
    const float val = col[e];
    if (ee >= M || val == 0.f) continue;
    const int er = ee % nb, ec = ee / nb;
    if (f.tile && fabsf(val) <= kTileBound)
      atomicAdd(tile + (y - f.y0 + er) + (x - f.x0 + ec) * f.ths, __float2int_rn(val * 1048576.f));
    else
      Acc<AccT>::add(acc + (y + er) + (size_t)(x + ec) * S, Acc<AccT>::fix(val));
  }
}

// Add n <= N tiles (T pixels each) to their accumulator slices (acc, acc +
// jstride) and clear them.
template <int N, typename AccT>
__device__ __forceinline__ void flush(const Footprint& f, int* tile, int T, AccT* acc,
                                      size_t jstride, int n, int S, int lane) {
  // the lane's entries are row r of a column, 32 entries of the footprint apart:
  // divided once, then stepped
  int r = lane % f.th, ti = r + lane / f.th * f.ths;
  AccT* a = acc + (size_t)(f.y0 + r) + (size_t)(f.x0 + lane / f.th) * S;
  const int dr = 32 % f.th, dc = 32 / f.th;
  const int dti = dr + dc * f.ths, da = dr + dc * S;
  const int wti = f.ths - f.th, wa = S - f.th;
  for (int t = lane; t < f.area; t += 32) {
#pragma unroll
    for (int j = 0; j < N; ++j) {
      if (j >= n) break;
      const int v = tile[j * T + ti];
      if (v != 0) {
        tile[j * T + ti] = 0;
        Acc<AccT>::add(a + j * jstride, Acc<AccT>::from_tile(v));
      }
    }
    r += dr;
    ti += dti;
    a += da;
    if (r >= f.th) {
      r -= f.th;
      ti += wti;
      a += wa;
    }
  }
}

// shrunk singular value (svt.hpp:135-143)
__device__ __forceinline__ float shrink(int expw, float s, float smax, float lam) {
  float th;
  if (expw) th = fabsf(smax * expf(-0.5f * lam * (s * s)));  // svt.hpp:137
  else th = lam;                                             // svt.hpp:142
  return fmaxf(fabsf(s) - th, 0.f);
}

// ---- one evaluation round: shrink, linear terms, rebuild + scatter of copy 0
//
// Block = 32 kept patches x nwin warps, small enough (at most about 110 KB of
// shared memory, 64 registers) for two blocks per SM when nwin <= 16.  Phase A
// spreads the (lambda, copy) pairs over all warps: the shrunk singular values
// g_i of copy 0 go to shared memory and sum_i g_i h_i of every copy to per-lane
// partials, over the triplets that can survive (one or two of 15 as a rule; the
// others have g = 0 or h = 0).  Phase B: warp k rebuilds column k (trajectory
// slice k) of its lanes' patches, two lambda values per pass (they share every
// load of the left and right vectors), and scatters them.  What bounds it is
// the instructions and shared-memory atomics of the scatter, 16 per patch,
// slice and lambda, and the flush of the tiles (72% of the shared-memory
// pipe's peak).  GB300, the rounds of one call: 256 x 256 x 100, 4 x 4 patches, 117
// -> 58 ms; 256 x 256 x 24, 8 x 8 patches, 127 -> 34 ms (before: tiles of 256
// pixels, divisions in the flush, conversions on the XU pipe, every triplet
// shrunk, one lambda value per pass for the larger patches).

// Rows of a patch rebuilt per pass: all of a small patch, else whole columns, few
// enough that the left vectors of a pass are loaded together within 64 registers
// (16 rows of an 8 x 8 patch: the loads were made one by one, 62 instead of 34 ms).
template <int BS>
__host__ __device__ constexpr int chunk_rows() {
  return BS >= 1 && BS <= 4 ? BS * BS : (BS == 5 ? 5 : (BS == 6 ? 12 : (BS == 7 ? 7 : 8)));
}

// launch bounds of k_eval: a block is 32 x nwin threads, nwin <= MAXW;
// windows up to 16 frames run two blocks per SM
template <int BS, typename AccT, int MAXW>
__global__ void __launch_bounds__(32 * MAXW, MAXW <= 16 ? 2 : 1)
    k_eval(Problem pb, DeviceBuffers d, int final_pass, int large_rounds) {
  const int nb = BS > 0 ? BS : pb.g.bs;  // BS == 0: any side (9..16)
  const int M = nb * nb;
  constexpr int PB = kEvalPatches;  // patches per block
  const Geometry& g = pb.g;
  const int w = blockIdx.y;
  const SearchState& st = d.st[w];
  const int nl = final_pass ? 1 : st.nnext;
  if (!final_pass && (st.done || nl == 0)) return;
  const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  const int NC = g.NC;
  const size_t NP = g.NP;
  const bool lin_terms = pb.optimize && !final_pass;
  const int ncp = lin_terms ? d.ncopies : 1;
  extern __shared__ __align__(16) float sg[];  // left vectors, g of copy 0 [nl][NC][PB],
                                               // lin [nl][4][PB], tiles
  constexpr bool kStage = BS > 0 && BS * BS <= 16;
  constexpr int US = eval_ustride(BS * BS);
  float* Us = sg;
  float* sgv = sg + eval_staged(BS, NC);
  const int T = eval_tile(BS, sizeof(AccT) == 8, large_rounds, nl);
  float* slin = sgv + (size_t)nl * NC * PB;
  int* tiles = (int*)(sg + eval_tiles_at(BS, NC, nl));
  __shared__ int srmax[kMaxK];
  int* tile = tiles + (size_t)k * (2 * T);
  for (int i = lane * 4; i < 2 * T; i += 128) *reinterpret_cast<int4*>(tile + i) = make_int4(0, 0, 0, 0);
  if (threadIdx.x < kMaxK) srmax[threadIdx.x] = 0;
  __syncthreads();
  const int p = blockIdx.x * PB + lane;
  const bool live = p < g.NP;
  // phase A: (lambda, copy) tasks over all warps
  for (int task = k; task < nl * ncp; task += nwarps) {
    const int j = task / ncp, c = task % ncp;
    const float lam = (float)(final_pass ? st.final_lambda : st.next[j]);
    const float* sv = d.sv + ((size_t)w * 4 + c) * NC * NP;
    const float* hv = d.hv + ((size_t)w * 4 + c) * NC * NP;
    const int nv = live ? d.nlive[((size_t)w * 4 + c) * NP + p] : 0;
    const int nvmax = __reduce_max_sync(0xffffffffu, nv);
    const float smax = live ? sv[p] : 0.f;  // sorted: column 0 is the largest
    float lin = 0.f;
    int r0 = 0;
    for (int i = 0; i < nvmax; ++i) {
      const float s = live ? sv[(size_t)i * NP + p] : 0.f;
      const float gi = shrink(pb.expw, s, smax, lam);
      if (c == 0) {
        sgv[((size_t)j * NC + i) * PB + lane] = gi;
        r0 += gi > 0.f;
      }
      if (lin_terms && live) lin = fmaf(gi, hv[(size_t)i * NP + p], lin);
    }
    slin[((size_t)j * 4 + c) * PB + lane] = lin;
    if (c == 0) {
      r0 = __reduce_max_sync(0xffffffffu, r0);
      if (lane == 0) atomicMax(&srmax[j], r0);
    }
  }
  __syncthreads();
  // patches of at most 16 rows: the left singular vectors of the block's
  // patches, up to the largest rank any lambda of the round keeps, staged in
  // shared memory once; every slice warp and every lambda reads them there
  if constexpr (kStage) {
    int R = 0;
    for (int j = 0; j < nl; ++j) R = max(R, srmax[j]);
    const float* U0p = d.U0 + g.u_at(w, p);
    for (int t = k; t < R * M; t += nwarps)  // t = i * M + e
      Us[((t / M) * PB + lane) * US + t % M] = live ? __ldg(U0p + t * 32) : 0.f;
    __syncthreads();
  }
  if (lin_terms)
    for (int j = k; j < nl; j += nwarps) {
      float lin = 0.f;
      for (int c = 0; c < ncp; ++c) lin += slin[((size_t)j * 4 + c) * PB + lane];
      const double t = warp_sum_d((double)lin);
      if (lane == 0) d.part_lin[((size_t)w * pb.K + j) * d.nblk_eval + blockIdx.x] = t;
    }
  if (k >= g.nwin) return;
  int y = 0, x = 0, nlive = 0;
  if (live) {
    const uint32_t pc = d.pos[((size_t)w * g.nwin + k) * g.P + d.plist[p]];
    y = pc & 0xffffu;
    x = pc >> 16;
    nlive = d.nlive[(size_t)w * 4 * NP + p];
  }
  Footprint f;
  f.init(live, y, x, nb, T);
  const float* U0 = d.U0 + g.u_at(w, p);
  const float* V0 = d.V0 + g.v_at(w, p) + k * 32;
  AccT* accw = (AccT*)d.acc + ((size_t)w * pb.K * g.nwin + k) * g.F();
  const size_t jstride = (size_t)g.nwin * g.F();  // accumulators of one lambda
  constexpr int CH = chunk_rows<BS>();
  for (int j0 = 0; j0 < nl; j0 += 2) {
    const bool two = j0 + 1 < nl;
    const int rm = min(max(srmax[j0], two ? srmax[j0 + 1] : 0), nlive);
    if (rm > 0) {
      const float* sg0 = sgv + (size_t)j0 * NC * PB + lane;
      const float* sg1 = sgv + (size_t)(two ? j0 + 1 : j0) * NC * PB + lane;
#pragma unroll 1
      for (int e0 = 0; e0 < M; e0 += CH) {
        float col[2][CH];
#pragma unroll
        for (int e = 0; e < CH; ++e) col[0][e] = col[1][e] = 0.f;
        for (int i = 0; i < rm; ++i) {
          const float v = V0[i * g.nwin * 32];
          const float c0 = sg0[i * PB] * v;
          const float c1 = two ? sg1[i * PB] * v : 0.f;
          if (c0 == 0.f && c1 == 0.f) continue;
          float u[CH];
          if constexpr (kStage) {
            const float* ui = Us + (i * PB + lane) * US;
            if constexpr (CH % 4 == 0) {
#pragma unroll
              for (int e = 0; e < CH; e += 4)
                *reinterpret_cast<float4*>(u + e) = *reinterpret_cast<const float4*>(ui + e);
            } else {
#pragma unroll
              for (int e = 0; e < CH; ++e) u[e] = ui[e];
            }
          } else {
            const float* ui = U0 + (i * M + e0) * 32;
#pragma unroll
            for (int e = 0; e < CH; ++e) u[e] = e0 + e < M ? __ldg(ui + e * 32) : 0.f;
          }
#pragma unroll
          for (int e = 0; e < CH; ++e) {
            col[0][e] = fmaf(c0, u[e], col[0][e]);
            col[1][e] = fmaf(c1, u[e], col[1][e]);
          }
        }
        scatter<BS, CH>(col[0], e0, nb, f, tile, accw + j0 * jstride, g.S, y, x);
        if (two)
          scatter<BS, CH>(col[1], e0, nb, f, tile + T, accw + (j0 + 1) * jstride, g.S, y, x);
      }
    }
    if (f.tile) {
      __syncwarp();
      flush<2>(f, tile, T, accw + j0 * jstride, jstride, two ? 2 : 1, g.S, lane);
      __syncwarp();
    }
  }
}

// ---- the output slice alone, at the chosen lambda: one warp per 32 patches
// (a block of k_eval would keep one of its nwin warps)
template <int BS, typename AccT>
__global__ void __launch_bounds__(128) k_eval_out(Problem pb, DeviceBuffers d) {
  const int nb = BS > 0 ? BS : pb.g.bs;
  const int M = nb * nb;
  const Geometry& g = pb.g;
  const int w = blockIdx.y;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  constexpr int T = eval_alloc_tile(BS, sizeof(AccT) == 8, 1);
  __shared__ int tiles[4][T];
  int* tile = tiles[wib];
  for (int i = lane; i < T; i += 32) tile[i] = 0;
  __syncwarp();
  const size_t NP = g.NP;
  const int NC = g.NC, k = d.wc[w].out_slice;
  const int p = (blockIdx.x * 4 + wib) * kEvalPatches + lane;
  const bool live = p < g.NP;
  int y = 0, x = 0, nlive = 0;
  if (live) {
    const uint32_t pc = d.pos[((size_t)w * g.nwin + k) * g.P + d.plist[p]];
    y = pc & 0xffffu;
    x = pc >> 16;
    nlive = d.nlive[(size_t)w * 4 * NP + p];
  }
  Footprint f;
  f.init(live, y, x, nb, T);
  const float lam = (float)d.st[w].final_lambda;
  const float* sv = d.sv + (size_t)w * 4 * NC * NP + p;
  const float* U0 = d.U0 + g.u_at(w, p);
  const float* V0 = d.V0 + g.v_at(w, p) + k * 32;
  AccT* acc = (AccT*)d.acc + ((size_t)w * pb.K * g.nwin + k) * g.F();
  constexpr int CH = chunk_rows<BS>();
  if (nlive > 0) {
    const float smax = sv[0];
#pragma unroll 1
    for (int e0 = 0; e0 < M; e0 += CH) {
      float col[CH];
#pragma unroll
      for (int e = 0; e < CH; ++e) col[e] = 0.f;
      for (int i = 0; i < nlive; ++i) {
        const float gi = shrink(pb.expw, sv[(size_t)i * NP], smax, lam);
        const float c0 = gi * V0[i * g.nwin * 32];
        if (c0 == 0.f) continue;
        const float* ui = U0 + (i * M + e0) * 32;
#pragma unroll
        for (int e = 0; e < CH; ++e)
          col[e] = fmaf(c0, e0 + e < M ? __ldg(ui + e * 32) : 0.f, col[e]);
      }
      scatter<BS, CH>(col, e0, nb, f, tile, acc, g.S, y, x);
    }
  }
  if (f.tile) {
    __syncwarp();
    flush<1>(f, tile, T, acc, 0, 1, g.S, lane);
  }
}

// ---- coverage counts (weights in svt.hpp:157-159): as the scatter, a warp
// counts its 32 patches' pixels in a tile and adds it with one atomic per pixel
constexpr int kCountTile = 512;

__global__ void __launch_bounds__(128) k_counts(Problem pb, DeviceBuffers d) {
  const Geometry& g = pb.g;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  const int k = blockIdx.y, w = blockIdx.z;
  const int lane = threadIdx.x & 31;
  __shared__ __align__(16) int tiles[4][kCountTile];
  int* tile = tiles[threadIdx.x >> 5];
  const bool live = p < g.NP;
  int y = 0, x = 0;
  if (live) {
    const uint32_t pc = d.pos[((size_t)w * g.nwin + k) * g.P + d.plist[p]];
    y = pc & 0xffffu;
    x = pc >> 16;
  }
  Footprint f;
  f.init(live, y, x, g.bs, kCountTile);
  if (f.th < g.bs) return;  // no live patch in this warp (warp-uniform)
  int32_t* c = d.cnt + (size_t)w * g.cube() + (size_t)k * g.F();
  if (!f.tile) {  // warp-uniform
    if (live)
      for (int cc = 0; cc < g.bs; ++cc)
        for (int r = 0; r < g.bs; ++r) atomicAdd(c + (y + r) + (size_t)(x + cc) * g.S, 1);
    return;
  }
  for (int i = lane * 4; i < kCountTile; i += 128) *reinterpret_cast<int4*>(tile + i) = make_int4(0, 0, 0, 0);
  __syncwarp();
  if (live) {
    int* t = tile + (y - f.y0) + (x - f.x0) * f.ths;
    for (int cc = 0; cc < g.bs; ++cc, t += f.ths)
      for (int r = 0; r < g.bs; ++r) atomicAdd(t + r, 1);
  }
  __syncwarp();
  flush<1>(f, tile, kCountTile, c, 0, 1, g.S, lane);
}

// The warp's sums of KT values per thread in FP64, each in warp_sum_d's order: while
// more than one value is left, the halves of the lanes go on with half of the values
// each, so 8 values take 9 FP64 additions instead of 40 (an SM needs 16 cycles for
// one).  Value `j` is this lane's; lanes that differ in the last steps' bits agree.
template <int KT>
__device__ __forceinline__ double warp_sums_d(const float (&v)[KT], int n, int& j) {
  const int lane = threadIdx.x & 31;
  double x[KT];
#pragma unroll
  for (int t = 0; t < KT; ++t) x[t] = t < n ? (double)v[t] : 0.0;
  j = 0;
#pragma unroll
  for (int o = 16, m = KT / 2; o > 0; o >>= 1, m >>= 1) {
    if (m > 0) {
      const bool up = lane & o;
      j += up ? m : 0;
#pragma unroll
      for (int t = 0; t < m; ++t) {
        const double give = up ? x[t] : x[t + m];
        x[t] = (up ? x[t + m] : x[t]) + __shfl_xor_sync(0xffffffffu, give, o);
      }
    } else {
      x[0] += __shfl_xor_sync(0xffffffffu, x[0], o);
    }
  }
  return x[0];
}

// ---- sum over voxels of (Uh - U)^2 for every lambda of the round; clears acc.
// Bound by DRAM, so a thread has the loads of two voxels in flight.  Eight windows of
// 256 x 256 x 15, GB300: 166 -> 126 us a round (one voxel at a time, and five FP64
// additions per warp and lambda).
template <typename AccT, int KT>
__global__ void __launch_bounds__(256, sizeof(AccT) * KT <= 32 ? 3 : 1) k_mse(Problem pb, DeviceBuffers d) {
  const Geometry& g = pb.g;
  const int w = blockIdx.y;
  const SearchState& st = d.st[w];
  if (st.done || st.nnext == 0) return;
  const int nl = st.nnext;
  const size_t C = g.cube();
  const float* u = d.u + (size_t)w * C;
  const int32_t* cnt = d.cnt + (size_t)w * C;
  AccT* acc = (AccT*)d.acc + (size_t)w * pb.K * C;
  constexpr int U = sizeof(AccT) * KT <= 64 ? 2 : 1;  // voxels side by side
  const size_t step = (size_t)gridDim.x * blockDim.x;
  float part[KT];  // a thread sees about 16 voxels: FP32 partials, FP64 beyond
#pragma unroll
  for (int j = 0; j < KT; ++j) part[j] = 0.f;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < C; i += U * step) {
    int n[U];
    float uv[U];
    AccT av[U][KT];  // every load first: the clears below could alias them
    const bool two = U > 1 && i + step < C;
#pragma unroll
    for (int v = 0; v < U; ++v) {
      const size_t at = v > 0 && two ? i + step : i;
      n[v] = __ldg(cnt + at);
      uv[v] = __ldg(u + at);
#pragma unroll
      for (int j = 0; j < KT; ++j)
        av[v][j] = (j < nl) ? __ldcs(acc + (size_t)j * C + at) : (AccT)0;
    }
#pragma unroll
    for (int v = 0; v < U; ++v) {
      const size_t at = v > 0 && two ? i + step : i;
      const bool use = v == 0 || two;
      const float inv = n[v] > 0 ? 1.f / (float)n[v] : 0.f;
#pragma unroll
      for (int j = 0; j < KT; ++j) {
        if (j < nl) __stcs(acc + (size_t)j * C + at, (AccT)0);
        const float df = Acc<AccT>::unfix(av[v][j]) * inv - uv[v];
        const float add = fmaf(df, df, part[j]);
        if (j < nl) part[j] = use ? add : part[j];
      }
    }
  }
  __shared__ double sm[KT][8];
  const int wid = threadIdx.x >> 5;
  int jw;
  const double t = warp_sums_d<KT>(part, nl, jw);
  sm[jw][wid] = t;  // the lanes of one value write the same
  __syncthreads();
  if (threadIdx.x < nl) {
    const int j = threadIdx.x;
    double t = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) t += sm[j][q];
    d.part_mse[((size_t)w * pb.K + j) * d.nblk_mse + blockIdx.x] = t;
  }
}

// ---- output slice and estimates (pguresvt.hpp:146-166)
template <typename AccT>
__global__ void k_output(Problem pb, DeviceBuffers d) {
  const Geometry& g = pb.g;
  const int w = blockIdx.y;
  const WinConst& wc = d.wc[w];
  const size_t F = g.F();
  AccT* acc = (AccT*)d.acc + ((size_t)w * pb.K * g.nwin + wc.out_slice) * F;
  const int32_t* cnt = d.cnt + (size_t)w * g.cube() + (size_t)wc.out_slice * F;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < F;
       i += (size_t)gridDim.x * blockDim.x) {
    const AccT a = acc[i];
    acc[i] = 0;
    const int n = cnt[i];
    double v = n > 0 ? (double)Acc<AccT>::unfix(a) / n : 0.0;
    if (!isfinite(v)) v = 0.0;
    d.Y[(size_t)wc.t * F + i] = v * wc.umax;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const int n = g.nimg;
    if (d.risk_out) d.risk_out[wc.t] = d.st[w].final_risk;
    if (pb.fixed_risk) {  // risks of the given list, in its order
      const SearchState& s = d.st[w];
      for (int j = 0; j < pb.nfixed; ++j) {
        double r = NAN;
        for (int i = 0; i < s.npts; ++i)
          if (s.lam[i] == pb.fixed[j]) r = s.risk[i];
        pb.fixed_risk[(size_t)wc.t * pb.nfixed + j] = r;
      }
    }
    if (d.evals_out) d.evals_out[wc.t] = (uint32_t)d.st[w].evals_total;
    d.est[wc.t] = d.st[w].final_lambda;
    d.est[wc.t + n] = wc.est_alpha;
    d.est[wc.t + 2 * (size_t)n] = wc.est_mu;
    d.est[wc.t + 3 * (size_t)n] = wc.est_sigma;
  }
}

// ---- whole reconstructed window v = acc / cnt (svt.hpp:163-164), window 0
template <typename AccT>
__global__ void k_cube_out(Problem pb, DeviceBuffers d, double* v) {
  const Geometry& g = pb.g;
  const size_t C = g.cube();
  AccT* acc = (AccT*)d.acc;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < C;
       i += (size_t)gridDim.x * blockDim.x) {
    const AccT a = acc[i];
    acc[i] = 0;
    const int n = d.cnt[i];
    double q = n > 0 ? (double)Acc<AccT>::unfix(a) / n : 0.0;
    v[i] = isfinite(q) ? q : 0.0;
  }
}

// ---- risks of the pending round without searching (component entry point)
__global__ void k_risk_collect(Problem pb, DeviceBuffers d, double* out) {
  const int w = 0;
  SearchState& s = d.st[w];
  const Geometry& g = pb.g;
  const WinConst& wc = d.wc[w];
  const double N = (double)g.S * g.S * g.nwin;
  const double a = wc.alpha, m = wc.mu, s2 = wc.sigma * wc.sigma;
  const int j = threadIdx.x;
  if (j < s.nnext) {
    double lin = 0.0, mse = 0.0;
    const double* pl = d.part_lin + ((size_t)w * pb.K + j) * d.nblk_eval;
    const double* pm = d.part_mse + ((size_t)w * pb.K + j) * d.nblk_mse;
    for (int b = 0; b < d.nblk_eval; ++b) lin += pl[b];
    for (int b = 0; b < d.nblk_mse; ++b) mse += pm[b];
    out[j] = (1.0 / N) * (mse + lin - (a + m) * wc.sum_u + m) - s2;
  }
}

// Raise, never lower, a kernel's dynamic shared-memory limit on the current
// device.  k_eval's footprint depends on the lambda count of the round, and
// concurrent callers (pgsvt_denoise_batch runs sequences on several host
// threads) must not shrink the limit under another thread's launch.
void allow_dynamic_smem(const void* kernel, size_t shm) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, size_t> limit;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  size_t& cur = limit[{dev, kernel}];
  if (shm > cur && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)shm) == cudaSuccess)
    cur = shm;
}

template <int BS, typename AccT>
void launch_k_eval_bs(dim3 grid, int threads, int nl, cudaStream_t s, const Problem& pb,
                      const DeviceBuffers& d, int final_pass) {
  // (110 KB at most for windows up to 16 frames)
  const size_t shm =
      (size_t)eval_alloc_words(BS, sizeof(AccT) == 8, pb.g.NC, pb.g.nwin, nl) * sizeof(int);
  const int large = eval_large_rounds(BS, sizeof(AccT) == 8, pb.g.NC, pb.g.nwin, nl);
  if constexpr (BS > 0 && BS * BS <= 16) {  // windows of at most 15 frames
    allow_dynamic_smem((const void*)k_eval<BS, AccT, 16>, shm);
    k_eval<BS, AccT, 16><<<grid, threads, shm, s>>>(pb, d, final_pass, large);
  } else if (threads <= 32 * 16) {  // two blocks per SM
    allow_dynamic_smem((const void*)k_eval<BS, AccT, 16>, shm);
    k_eval<BS, AccT, 16><<<grid, threads, shm, s>>>(pb, d, final_pass, large);
  } else {
    allow_dynamic_smem((const void*)k_eval<BS, AccT, 21>, shm);
    k_eval<BS, AccT, 21><<<grid, threads, shm, s>>>(pb, d, final_pass, large);
  }
}

template <typename AccT>
void launch_k_eval_t(int bs, dim3 grid, int threads, int nl, cudaStream_t s,
                     const Problem& pb, const DeviceBuffers& d, int final_pass) {
  switch (bs) {
    case 2: launch_k_eval_bs<2, AccT>(grid, threads, nl, s, pb, d, final_pass); break;
    case 3: launch_k_eval_bs<3, AccT>(grid, threads, nl, s, pb, d, final_pass); break;
    case 4: launch_k_eval_bs<4, AccT>(grid, threads, nl, s, pb, d, final_pass); break;
    case 5: launch_k_eval_bs<5, AccT>(grid, threads, nl, s, pb, d, final_pass); break;
    case 6: launch_k_eval_bs<6, AccT>(grid, threads, nl, s, pb, d, final_pass); break;
    case 7: launch_k_eval_bs<7, AccT>(grid, threads, nl, s, pb, d, final_pass); break;
    case 8: launch_k_eval_bs<8, AccT>(grid, threads, nl, s, pb, d, final_pass); break;
    default: launch_k_eval_bs<0, AccT>(grid, threads, nl, s, pb, d, final_pass); break;
  }
}

void launch_k_eval(const Problem& pb, const DeviceBuffers& d, int final_pass, int nl,
                   cudaStream_t s) {
  const Geometry& g = pb.g;
  const dim3 grid(d.nblk_eval, pb.W);
  if (pb.acc64)
    launch_k_eval_t<unsigned long long>(g.bs, grid, 32 * g.nwin, nl, s, pb, d, final_pass);
  else launch_k_eval_t<int>(g.bs, grid, 32 * g.nwin, nl, s, pb, d, final_pass);
}

template <typename AccT>
void launch_k_eval_out_t(const Problem& pb, const DeviceBuffers& d, cudaStream_t s) {
  const dim3 grid((pb.g.NP + 4 * kEvalPatches - 1) / (4 * kEvalPatches), pb.W);
  switch (pb.g.bs) {
    case 2: k_eval_out<2, AccT><<<grid, 128, 0, s>>>(pb, d); break;
    case 3: k_eval_out<3, AccT><<<grid, 128, 0, s>>>(pb, d); break;
    case 4: k_eval_out<4, AccT><<<grid, 128, 0, s>>>(pb, d); break;
    case 5: k_eval_out<5, AccT><<<grid, 128, 0, s>>>(pb, d); break;
    case 6: k_eval_out<6, AccT><<<grid, 128, 0, s>>>(pb, d); break;
    case 7: k_eval_out<7, AccT><<<grid, 128, 0, s>>>(pb, d); break;
    case 8: k_eval_out<8, AccT><<<grid, 128, 0, s>>>(pb, d); break;
    default: k_eval_out<0, AccT><<<grid, 128, 0, s>>>(pb, d); break;
  }
}

void launch_k_mse(const Problem& pb, const DeviceBuffers& d, cudaStream_t s) {
  const dim3 grid(d.nblk_mse, pb.W);
  if (pb.K <= 8) {
    if (pb.acc64) k_mse<unsigned long long, 8><<<grid, 256, 0, s>>>(pb, d);
    else k_mse<int, 8><<<grid, 256, 0, s>>>(pb, d);
  } else {
    if (pb.acc64) k_mse<unsigned long long, kMaxK><<<grid, 256, 0, s>>>(pb, d);
    else k_mse<int, kMaxK><<<grid, 256, 0, s>>>(pb, d);
  }
}

}  // namespace

int eval_blocks(const Geometry& g) { return (g.NP + kEvalPatches - 1) / kEvalPatches; }
int mse_blocks(const Geometry& g) {
  return (int)std::max<size_t>(32, std::min<size_t>(1024, g.cube() / 4096));
}

cudaError_t launch_fields(const Problem& pb, const DeviceBuffers& d, cudaStream_t s) {
  const Geometry& g = pb.g;
  cudaMemsetAsync(d.cnt, 0, sizeof(int32_t) * g.cube() * pb.W, s);
  dim3 gc((g.NP + 127) / 128, g.nwin, pb.W);
  k_counts<<<gc, 128, 0, s>>>(pb, d);
  if (!pb.optimize) return cudaGetLastError();
  if (pb.compat & 0x4) k_field_table<<<dim3(2, pb.W), kFieldTab, 0, s>>>(pb, d);
  k_fields<<<dim3(kFieldBlocks, pb.W), 256, 0, s>>>(pb, d);
  return cudaGetLastError();
}

cudaError_t launch_search_init(const Problem& pb, const DeviceBuffers& d, cudaStream_t s) {
  k_search_init<<<pb.W, kFieldBlocks, 0, s>>>(pb, d);
  return cudaGetLastError();
}

cudaError_t launch_search_hint(const Problem& pb, const DeviceBuffers& d, cudaStream_t s) {
  k_search_hint<<<pb.W, 32, 0, s>>>(pb, d);
  return cudaGetLastError();
}

cudaError_t launch_eval_round(const Problem& pb, const DeviceBuffers& d, int final_pass,
                              cudaStream_t s) {
  if (final_pass == 1) {  // the output slice alone
    if (pb.acc64) launch_k_eval_out_t<unsigned long long>(pb, d, s);
    else launch_k_eval_out_t<int>(pb, d, s);
    return cudaGetLastError();
  }
  launch_k_eval(pb, d, final_pass, final_pass ? 1 : pb.K, s);
  if (final_pass) return cudaGetLastError();  // 2: every slice
  launch_k_mse(pb, d, s);
  k_search_step<<<pb.W, 256 * kStepGroups, 0, s>>>(pb, d);
  return cudaGetLastError();
}

cudaError_t launch_cube_out(const Problem& pb, const DeviceBuffers& d, double* v,
                            cudaStream_t s) {
  if (pb.acc64) k_cube_out<unsigned long long><<<512, 256, 0, s>>>(pb, d, v);
  else k_cube_out<int><<<512, 256, 0, s>>>(pb, d, v);
  return cudaGetLastError();
}

cudaError_t launch_risk_round(const Problem& pb, const DeviceBuffers& d, double* out,
                              cudaStream_t s) {
  launch_k_eval(pb, d, 0, pb.K, s);
  launch_k_mse(pb, d, s);
  k_risk_collect<<<1, kMaxK, 0, s>>>(pb, d, out);
  return cudaGetLastError();
}

cudaError_t launch_output(const Problem& pb, const DeviceBuffers& d, cudaStream_t s) {
  const Geometry& g = pb.g;
  dim3 go((unsigned)std::min<size_t>((g.F() + 255) / 256, 512), pb.W);
  if (pb.acc64) k_output<unsigned long long><<<go, 256, 0, s>>>(pb, d);
  else k_output<int><<<go, 256, 0, s>>>(pb, d);
  return cudaGetLastError();
}

}  // namespace pgsvt
