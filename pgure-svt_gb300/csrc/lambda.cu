// lambda.cu — learned lambda proposal (not in the reference).
//
// A small MLP maps per-window features (the risk's noise parameters and a
// histogram of log singular values) to y = log10(lambda/upper); the proposal
// starts a narrow PGURE search (eval.cu, phase 1) that falls back to the plain
// search.  The network is tiny (67 -> 128 -> 128 -> 128 -> 1, 41,857
// parameters), far too small to fill a tensor-core tile per step, so every pass
// runs on CUDA cores with FP32 sums.  Training keeps FP32 master weights and a
// bf16 shadow that the passes read.  What bounds a step is latency: 14 MFLOP
// over chains of 128 dependent FMAs per layer.  So it is spread thin: k_mlp_pass
// runs four samples per block (the samples are independent), with the weights in
// shared memory, and k_mlp_update (many rows: k_mlp_chains and k_mlp_sum) forms
// every weight's gradient, sums it in a fixed order (chains of 32 samples, then
// the chains) and applies AdamW in the same thread, so training is deterministic.
#include <cuda_bf16.h>

#include <algorithm>

#include "pgsvt.h"
#include "pgsvt_internal.h"

namespace pgsvt {
namespace lam {

constexpr int NF = PGSVT_LAMBDA_FEATURES;   // 67
constexpr int H = PGSVT_LAMBDA_HIDDEN;      // 128
constexpr int OFF_MEAN = 0, OFF_SCALE = NF, OFF_W1 = 2 * NF;
constexpr int OFF_B1 = OFF_W1 + H * NF, OFF_W2 = OFF_B1 + H, OFF_B2 = OFF_W2 + H * H;
constexpr int OFF_W3 = OFF_B2 + H, OFF_B3 = OFF_W3 + H * H, OFF_W4 = OFF_B3 + H;
constexpr int OFF_B4 = OFF_W4 + H, OFF_YMEAN = OFF_B4 + 1, OFF_YSCALE = OFF_YMEAN + 1;
constexpr int TOTAL = OFF_YSCALE + 1;
constexpr int NPARAM = OFF_YMEAN - OFF_W1;
static_assert(TOTAL == PGSVT_LAMBDA_MODEL_FLOATS, "model layout");
static_assert(NPARAM == PGSVT_LAMBDA_PARAMS, "parameter count");
static_assert(OFF_W1 == PGSVT_LAMBDA_PARAM_OFFSET, "parameter offset");

constexpr int GS = 4;         // samples of a pass at a time
constexpr int PT = 256;       // its threads: one output of two samples each
constexpr int LDA = 132;      // row stride of the activations in shared memory
constexpr int WS1 = 72, WS2 = 136;  // weight row strides (bf16): 16-byte rows that
                                    // start four banks apart
// The bf16 shadow of the model, laid out as the passes hold it in shared memory
// (one straight copy): padded weight rows, then the output row as floats.
struct __align__(16) Shadow {
  __nv_bfloat16 w1[H * WS1], w2[H * WS2], w3[H * WS2];
  float w4[H];
};
static_assert(sizeof(Shadow) <= PGSVT_LAMBDA_SHADOW_BYTES, "shadow allocation");
struct Smem {
  Shadow w;
  float x0[GS * LDA];
  float z[3][GS * LDA];   // pre-activations, then their gradients
  float a[3][GS * LDA];   // activations
  float o[GS], dO[GS];    // network outputs (before y_scale / y_mean), their gradients
};

// Rows of a training pass in device memory, kept for the weight gradients:
// [row][128] each, row r the r-th sample of the batch
enum { ACT_X0, ACT_A1, ACT_A2, ACT_A3, ACT_Z1, ACT_Z2, ACT_Z3, ACT_N };

__device__ __forceinline__ float gelu(float z) {
  return 0.5f * z * (1.f + erff(z * 0.70710678118654752f));
}
__device__ __forceinline__ float gelu_grad(float z) {
  return 0.5f * (1.f + erff(z * 0.70710678118654752f)) +
         z * 0.39894228040143268f * expf(-0.5f * z * z);
}
// Parameter at model offset i (value v) into the shadow, rounded to bf16.
__device__ __forceinline__ void to_shadow(Shadow* sh, int i, float v) {
  const __nv_bfloat16 b = __float2bfloat16_rn(v);
  if (i >= OFF_W1 && i < OFF_B1) sh->w1[(i - OFF_W1) / NF * WS1 + (i - OFF_W1) % NF] = b;
  else if (i >= OFF_W2 && i < OFF_B2) sh->w2[(i - OFF_W2) / H * WS2 + (i - OFF_W2) % H] = b;
  else if (i >= OFF_W3 && i < OFF_B3) sh->w3[(i - OFF_W3) / H * WS2 + (i - OFF_W3) % H] = b;
  else if (i >= OFF_W4 && i < OFF_B4) sh->w4[i - OFF_W4] = __bfloat162float(b);
}

// The weights into shared memory.
__device__ void load_weights(const Shadow* __restrict__ sh, Smem& sm) {
  const uint4* g = reinterpret_cast<const uint4*>(sh);
  uint4* o = reinterpret_cast<uint4*>(&sm.w);
  constexpr int N = (int)(sizeof(Shadow) / 16);
#pragma unroll 11
  for (int i = threadIdx.x; i < N; i += PT) o[i] = g[i];
}

__device__ __forceinline__ float bf_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// One dense layer plus GELU: thread (j, h) computes output j of samples 2h
// and 2h + 1, each sum in input order.
template <int KIN, int WS>
__device__ __forceinline__ void dense_gelu(const __nv_bfloat16* W, float bj, const float* in,
                                           float* z, float* a) {
  const int j = threadIdx.x & (H - 1), s0 = (threadIdx.x >> 7) * 2;
  const float* p = in + s0 * LDA;
  const __nv_bfloat16* wr = W + j * WS;
  float c0 = bj, c1 = bj;
  constexpr int K8 = KIN / 8 * 8;
#pragma unroll 4
  for (int k = 0; k < K8; k += 8) {
    const uint4 wv = *reinterpret_cast<const uint4*>(wr + k);
    const uint32_t wu[4] = {wv.x, wv.y, wv.z, wv.w};
    float u[8], v[8];
    *reinterpret_cast<float4*>(u) = *reinterpret_cast<const float4*>(p + k);
    *reinterpret_cast<float4*>(u + 4) = *reinterpret_cast<const float4*>(p + k + 4);
    *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(p + LDA + k);
    *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(p + LDA + k + 4);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float w = (q & 1) ? bf_hi(wu[q >> 1]) : bf_lo(wu[q >> 1]);
      c0 = fmaf(w, u[q], c0);
      c1 = fmaf(w, v[q], c1);
    }
  }
#pragma unroll
  for (int k = K8; k < KIN; ++k) {
    const float w = __bfloat162float(wr[k]);
    c0 = fmaf(w, p[k], c0);
    c1 = fmaf(w, p[LDA + k], c1);
  }
  z[s0 * LDA + j] = c0;
  z[(s0 + 1) * LDA + j] = c1;
  a[s0 * LDA + j] = gelu(c0);
  a[(s0 + 1) * LDA + j] = gelu(c1);
}

// Gradient of a layer's input through the GELU before it: thread (k, h),
// samples 2h and 2h + 1, each sum in output order; zprev holds the previous
// pre-activations and receives their gradients.
__device__ __forceinline__ void dense_back(const __nv_bfloat16* W, const float* dz, float* zprev) {
  const int k = threadIdx.x & (H - 1), s0 = (threadIdx.x >> 7) * 2;
  const float* p = dz + s0 * LDA;
  float c0 = 0.f, c1 = 0.f;
#pragma unroll 4
  for (int j = 0; j < H; j += 4) {
    float u[4], v[4];
    *reinterpret_cast<float4*>(u) = *reinterpret_cast<const float4*>(p + j);
    *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(p + LDA + j);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float w = __bfloat162float(W[(j + q) * WS2 + k]);
      c0 = fmaf(w, u[q], c0);
      c1 = fmaf(w, v[q], c1);
    }
  }
  float* zp = zprev + s0 * LDA + k;
  zp[0] = c0 * gelu_grad(zp[0]);
  zp[LDA] = c1 * gelu_grad(zp[LDA]);
}

// Stage the features of samples [b0, b0 + GS) of [0, n) as (f - mean) * scale,
// the others as zeros.  `rows` maps a sample to a feature row (or null).
__device__ void load_inputs(const float* m, const float* feat, const int32_t* rows, int b0, int n,
                            Smem& sm) {
  for (int i = threadIdx.x; i < GS * NF; i += PT) {
    const int s = i / NF, k = i % NF;
    float v = 0.f;
    if (b0 + s < n) {
      const int r = rows ? rows[b0 + s] : b0 + s;
      v = (feat[(size_t)r * NF + k] - m[OFF_MEAN + k]) * m[OFF_SCALE + k];
    }
    sm.x0[s * LDA + k] = v;
  }
}

// Forward pass of the GS samples in sm.x0; the outputs land in sm.o.
__device__ void forward(const float* m, Smem& sm) {
  const int j = threadIdx.x & (H - 1);
  __syncthreads();
  dense_gelu<NF, WS1>(sm.w.w1, m[OFF_B1 + j], sm.x0, sm.z[0], sm.a[0]);
  __syncthreads();
  dense_gelu<H, WS2>(sm.w.w2, m[OFF_B2 + j], sm.a[0], sm.z[1], sm.a[1]);
  __syncthreads();
  dense_gelu<H, WS2>(sm.w.w3, m[OFF_B3 + j], sm.a[1], sm.z[2], sm.a[2]);
  __syncthreads();
  if (threadIdx.x < GS) {
    const int s = threadIdx.x;
    float acc = m[OFF_B4];
#pragma unroll 16
    for (int k = 0; k < H; ++k) acc = fmaf(sm.w.w4[k], sm.a[2][s * LDA + k], acc);
    sm.o[s] = acc;
  }
  __syncthreads();
}

// Forward pass and the gradients of the pre-activations of the samples of one
// batch (r0 .. n of the permuted order, rows padded to a multiple of 32): the
// activations, gradients, output gradients and errors of every row to device
// memory.  One block per GS rows; a batch of 256 fills 64 SMs, and
// its chains of dependent FMAs, not its 14 MFLOP, are what takes the time.
// One training step (batch 256), GB300: 177 -> 11.7 us here and 8.5 us in
// k_mlp_update (before, one block of 128 threads did everything for 32 samples).
__global__ void __launch_bounds__(PT) k_mlp_pass(const float* __restrict__ m,
                                                 const Shadow* __restrict__ wbf,
                                                 const float* __restrict__ feat,
                                                 const float* __restrict__ target,
                                                 const int32_t* __restrict__ perm,
                                                 const int* __restrict__ epoch, int64_t perm_stride,
                                                 int r0, int n, int rows_pad, float norm,
                                                 float* __restrict__ act, float* __restrict__ dO,
                                                 float* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char smraw[];
  Smem& sm = *reinterpret_cast<Smem*>(smraw);
  const int32_t* rows = perm ? perm + (epoch ? (int64_t)(*epoch) * perm_stride : 0) : nullptr;
  load_weights(wbf, sm);
  const float ym = m[OFF_YMEAN], ysi = 1.f / m[OFF_YSCALE];
  const size_t plane = (size_t)rows_pad * H;
  for (int g0 = blockIdx.x * GS; g0 < rows_pad; g0 += gridDim.x * GS) {
    const int b0 = r0 + g0;
    load_inputs(m, feat, rows, b0, n, sm);
    forward(m, sm);
    if (threadIdx.x < GS) {
      const int s = threadIdx.x;
      float e = 0.f;
      if (b0 + s < n) {
        const int r = rows ? rows[b0 + s] : b0 + s;
        e = sm.o[s] - (target[r] - ym) * ysi;
      }
      sm.dO[s] = 2.f * e * norm;
      dO[g0 + s] = sm.dO[s];
      err[g0 + s] = e;
    }
    __syncthreads();
    // dz3 = dO W4 gelu'(z3)
    const int j = threadIdx.x & (H - 1), s0 = (threadIdx.x >> 7) * 2;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      float* z = &sm.z[2][(s0 + q) * LDA + j];
      *z = sm.dO[s0 + q] * sm.w.w4[j] * gelu_grad(*z);
    }
    __syncthreads();
    dense_back(sm.w.w3, sm.z[2], sm.z[1]);
    __syncthreads();
    dense_back(sm.w.w2, sm.z[1], sm.z[0]);
#pragma unroll
    for (int q = 0; q < 2; ++q) {  // (own elements only: no barrier needed)
      const size_t o = (size_t)(g0 + s0 + q) * H + j;
      const int l = (s0 + q) * LDA + j;
      if (j < NF) act[ACT_X0 * plane + o] = sm.x0[l];
#pragma unroll
      for (int t = 0; t < 3; ++t) {
        act[(ACT_A1 + t) * plane + o] = sm.a[t][l];
        act[(ACT_Z1 + t) * plane + o] = sm.z[t][l];
      }
    }
    __syncthreads();  // the next group overwrites the rows
  }
}

// Network outputs y (after y_scale / y_mean) of n feature rows.
__global__ void __launch_bounds__(PT) k_mlp_forward(const float* __restrict__ m,
                                                    const Shadow* __restrict__ wbf,
                                                    const float* __restrict__ feat, int n,
                                                    float* __restrict__ y, float* __restrict__ y2) {
  extern __shared__ __align__(16) unsigned char smraw[];
  Smem& sm = *reinterpret_cast<Smem*>(smraw);
  load_weights(wbf, sm);
  for (int b0 = blockIdx.x * GS; b0 < n; b0 += gridDim.x * GS) {
    load_inputs(m, feat, nullptr, b0, n, sm);
    forward(m, sm);
    const int r = b0 + threadIdx.x;
    if (threadIdx.x < GS && r < n) {
      const float v = sm.o[threadIdx.x] * m[OFF_YSCALE] + m[OFF_YMEAN];
      y[r] = v;
      if (y2) y2[r] = v;
    }
    __syncthreads();
  }
}

__device__ __forceinline__ bool is_weight(int i) {  // i: offset in the model
  return (i >= OFF_W1 && i < OFF_B1) || (i >= OFF_W2 && i < OFF_B2) ||
         (i >= OFF_W3 && i < OFF_B3) || (i >= OFF_W4 && i < OFF_B4);
}

// bf16 shadow of the weights.
__global__ void k_mlp_shadow(const float* __restrict__ m, Shadow* __restrict__ wbf) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < TOTAL; i += gridDim.x * blockDim.x)
    to_shadow(wbf, i, m[i]);
}

struct AdamCfg {
  float lr, lr_final, wd, b1, b2, eps;
  int steps_per_epoch, total_steps;
};

// AdamW step t (1-based) of parameter i with gradient g: FP32 master and
// moments, bf16 shadow refreshed.
__device__ __forceinline__ void adam(float* m, Shadow* wbf, float* mom1, float* mom2, int i,
                                     float g, int t, const AdamCfg& c) {
  const float prog = (float)(t - 1) / (float)max(1, c.total_steps - 1);
  const float lr = c.lr_final + 0.5f * (c.lr - c.lr_final) * (1.f + cospif(prog));
  const float m1 = c.b1 * mom1[i] + (1.f - c.b1) * g;
  const float m2 = c.b2 * mom2[i] + (1.f - c.b2) * g * g;
  mom1[i] = m1;
  mom2[i] = m2;
  const float bc1 = 1.f - powf(c.b1, (float)t), bc2 = 1.f - powf(c.b2, (float)t);
  const int mi = OFF_W1 + i;
  float w = m[mi];
  if (is_weight(mi)) w -= lr * c.wd * w;
  w -= lr * (m1 / bc1) / (sqrtf(m2 / bc2) + c.eps);
  m[mi] = w;
  to_shadow(wbf, mi, w);
}

// Gradients from the rows of a pass, summed in a fixed order (a chain of FMAs
// over each 32 rows, then the chains in order), and with ADAM the parameter
// update; without it the gradients go to `grad`.  A block of 128 inputs x NCH
// chains takes JB outputs of one layer: the chains run side by side (what
// bounds the kernel is their latency) and are added in order from shared
// memory.  The last blocks take the biases, the output layer and the squared
// errors.
constexpr int JB = 2;                    // outputs per block
constexpr int NCH = 8;                   // chains at a time
constexpr int UB = H / JB;               // blocks of one layer
constexpr int kUpdateBlocks = 3 * UB + 5;

template <bool ADAM>
__global__ void __launch_bounds__(H * NCH) k_mlp_update(
    float* __restrict__ m, Shadow* __restrict__ wbf, float* __restrict__ mom1,
    float* __restrict__ mom2, const float* __restrict__ act, const float* __restrict__ dO,
    const float* __restrict__ err, int rows_pad, const int* __restrict__ epoch, int step,
    AdamCfg c, float* __restrict__ grad, float* __restrict__ loss) {
  __shared__ float part[JB][NCH][H];
  const int bi = blockIdx.x, tid = threadIdx.x & (H - 1), ch = threadIdx.x >> 7;
  const size_t plane = (size_t)rows_pad * H;
  const int t = ADAM ? *epoch * c.steps_per_epoch + step + 1 : 0;  // 1-based step count
  // kinds of block: layer weights, bias, output row, output bias + errors
  const bool weights = bi < 3 * UB;
  const int rest = bi - 3 * UB;
  const int layer = weights ? bi / UB : rest;
  const int j0 = weights ? (bi % UB) * JB : 0;
  const int kin = weights && layer == 0 ? NF : H;
  float g[JB];
#pragma unroll
  for (int q = 0; q < JB; ++q) g[q] = 0.f;
  for (int b0 = 0; b0 < rows_pad; b0 += 32 * NCH) {
    const int r = b0 + 32 * ch;
    float p[JB];
#pragma unroll
    for (int q = 0; q < JB; ++q) p[q] = 0.f;
    if (r < rows_pad && tid < kin) {
      if (weights) {
        const float* in = act + (ACT_X0 + layer) * plane + (size_t)r * H + tid;
        const float* dz = act + (ACT_Z1 + layer) * plane + (size_t)r * H + j0;
        static_assert(JB == 2, "two outputs per thread");
#pragma unroll
        for (int s = 0; s < 32; ++s) {
          const float x = in[s * H];
          const float2 d = *reinterpret_cast<const float2*>(dz + s * H);
          p[0] = fmaf(d.x, x, p[0]);
          p[1] = fmaf(d.y, x, p[1]);
        }
      } else if (rest < 3) {
        const float* dz = act + (ACT_Z1 + layer) * plane + (size_t)r * H + tid;
#pragma unroll
        for (int s = 0; s < 32; ++s) p[0] += dz[s * H];
      } else if (rest == 3) {
        const float* in = act + ACT_A3 * plane + (size_t)r * H + tid;
#pragma unroll
        for (int s = 0; s < 32; ++s) p[0] = fmaf(dO[r + s], in[s * H], p[0]);
      } else {
        if (tid == 0) {
#pragma unroll
          for (int s = 0; s < 32; ++s) p[0] += dO[r + s];
        }
        if (tid < 32) {
          const float e = err[r + tid];
          float sq = e * e;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
          if (tid == 0) loss[r >> 5] = sq;
        }
      }
    }
    if (b0 > 0) __syncthreads();
#pragma unroll
    for (int q = 0; q < JB; ++q) part[q][ch][tid] = p[q];
    __syncthreads();
    if (ch < JB)
      for (int k = 0; k < NCH && b0 + 32 * k < rows_pad; ++k) g[0] += part[ch][k][tid];
  }
  // thread (tid, ch < JB) holds the gradient of output j0 + ch
  int i;
  if (weights) {
    if (ch >= JB || tid >= kin) return;
    i = (layer == 0 ? OFF_W1 : (layer == 1 ? OFF_W2 : OFF_W3)) + (j0 + ch) * kin + tid;
  } else {
    if (ch > 0 || (rest == 4 && tid > 0)) return;
    i = (rest == 0 ? OFF_B1 : rest == 1 ? OFF_B2 : rest == 2 ? OFF_B3 : rest == 3 ? OFF_W4 : OFF_B4) + tid;
  }
  i -= OFF_W1;
  if constexpr (ADAM) adam(m, wbf, mom1, mom2, i, g[0], t, c);
  else grad[i] = g[0];
}

// The same in two kernels for many rows: a block of k_mlp_chains forms the sums of one
// chain of 32 rows for a whole layer, 8 x 8 of them per thread from rows in shared
// memory, and k_mlp_sum adds the chains up in their order.  k_mlp_update walks the
// chains in every block, so its time goes with the rows.  A step's update, GB300:
// 256 rows 8.6 us there, 8.9 + 4.6 us here; 512 rows 12.0 and 9.1 + 2.9; 1,024 rows
// 23.6 and 9.3 + 3.3; 8,192 rows 175 and 35.4 + 9.6, bound by the FMAs of the chains.
constexpr int CT = 256;  // threads of k_mlp_chains

__global__ void __launch_bounds__(CT) k_mlp_chains(const float* __restrict__ act,
                                                   const float* __restrict__ dO,
                                                   const float* __restrict__ err, int rows_pad,
                                                   int ch0, float* __restrict__ part,
                                                   float* __restrict__ loss) {
  __shared__ __align__(16) float xs[32][H], ds[32][H];
  const int ch = ch0 + blockIdx.x, layer = blockIdx.y, tid = threadIdx.x;
  const size_t plane = (size_t)rows_pad * H, row0 = (size_t)ch * 32 * H;
  float* out = part + (size_t)blockIdx.x * NPARAM;
  if (layer == 3) {  // the biases, the output layer and the squared error
    if (tid < H) {
      float b[3] = {0.f, 0.f, 0.f}, w = 0.f;
      for (int s = 0; s < 32; ++s) {
#pragma unroll
        for (int l = 0; l < 3; ++l) b[l] += act[(ACT_Z1 + l) * plane + row0 + s * H + tid];
        w = fmaf(dO[ch * 32 + s], act[ACT_A3 * plane + row0 + s * H + tid], w);
      }
      out[OFF_B1 - OFF_W1 + tid] = b[0];
      out[OFF_B2 - OFF_W1 + tid] = b[1];
      out[OFF_B3 - OFF_W1 + tid] = b[2];
      out[OFF_W4 - OFF_W1 + tid] = w;
    } else if (tid < H + 32) {
      const float e = err[ch * 32 + tid - H];
      float sq = e * e;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
      if (tid == H) {
        float t = 0.f;
        for (int s = 0; s < 32; ++s) t += dO[ch * 32 + s];
        out[OFF_B4 - OFF_W1] = t;
        loss[ch] = sq;
      }
    }
    return;
  }
  // (inputs beyond the features are not set in layer 0, and not stored below)
  const float4* in = reinterpret_cast<const float4*>(act + (ACT_X0 + layer) * plane + row0);
  const float4* dz = reinterpret_cast<const float4*>(act + (ACT_Z1 + layer) * plane + row0);
  for (int i = tid; i < 32 * H / 4; i += CT) {
    reinterpret_cast<float4*>(xs)[i] = in[i];
    reinterpret_cast<float4*>(ds)[i] = dz[i];
  }
  __syncthreads();
  const int k0 = (tid & 15) * 4, j0 = (tid >> 4) * 8;  // inputs k0.., 64 + k0.., outputs j0..
  float g[8][8];
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int k = 0; k < 8; ++k) g[j][k] = 0.f;
#pragma unroll 4
  for (int s = 0; s < 32; ++s) {
    float x[8], d[8];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      *reinterpret_cast<float4*>(x + 4 * h) = *reinterpret_cast<const float4*>(&xs[s][k0 + 64 * h]);
      *reinterpret_cast<float4*>(d + 4 * h) = *reinterpret_cast<const float4*>(&ds[s][j0 + 4 * h]);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int k = 0; k < 8; ++k) g[j][k] = fmaf(d[j], x[k], g[j][k]);
  }
  const int kin = layer == 0 ? NF : H;
  out += (layer == 0 ? OFF_W1 : (layer == 1 ? OFF_W2 : OFF_W3)) - OFF_W1;
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int kk = k0 + (k & 3) + 64 * (k >> 2);
      if (kk < kin) out[(j0 + j) * kin + kk] = g[j][k];
    }
}

// (more: to the sums in grad of the chains before)
template <bool ADAM>
__global__ void __launch_bounds__(128) k_mlp_sum(float* __restrict__ m, Shadow* __restrict__ wbf,
                                                 float* __restrict__ mom1, float* __restrict__ mom2,
                                                 const float* __restrict__ part, int nch, bool more,
                                                 const int* __restrict__ epoch, int step, AdamCfg c,
                                                 float* __restrict__ grad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NPARAM) return;
  float g = !ADAM && more ? grad[i] : 0.f;
#pragma unroll 16
  for (int k = 0; k < nch; ++k) g += part[(size_t)k * NPARAM + i];
  if constexpr (ADAM) adam(m, wbf, mom1, mom2, i, g, *epoch * c.steps_per_epoch + step + 1, c);
  else grad[i] = g;
}

// Mean loss of the epoch; advances the device epoch counter.
__global__ void k_mlp_epoch_end(const float* __restrict__ loss_acc, int nsteps, int nblk, int n,
                                int* __restrict__ epoch, float* __restrict__ epoch_loss) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  float t = 0.f;
  for (int i = 0; i < nsteps * nblk; ++i) t += loss_acc[i];
  epoch_loss[*epoch] = t / (float)max(1, n);
  *epoch += 1;
}

}  // namespace lam

// ---------------------------------------------------------------------------
// Features of every window of a batch: block w histograms the copy-0
// singular values of the sampled patches of window w.  One block per window, so
// what bounds it is the latency of its scattered reads: 1,024 threads with eight
// reads each in flight, a histogram per warp.  4,096 patches x 15, GB300: 244 -> 57 us.
__global__ void __launch_bounds__(1024) k_lambda_features(Problem pb, DeviceBuffers d) {
  const Geometry& g = pb.g;
  const int w = blockIdx.x;
  __shared__ int hist[32][64];
  __shared__ int total[64];
  int* h = hist[threadIdx.x >> 5];
  h[threadIdx.x & 31] = h[32 + (threadIdx.x & 31)] = 0;
  __syncwarp();
  const int ns = d.nfeat_slots, nwin = g.nwin;
  const size_t NP = g.NP;
  const float* sv = d.sv + (size_t)w * 4 * g.NC * NP;  // copy 0
  for (int si = threadIdx.x; si < ns; si += blockDim.x) {
    const float* col = sv + d.feat_slots[si];
#pragma unroll 8
    for (int t = 0; t < nwin; ++t) {
      const float s = col[(size_t)t * NP];
      int b = 0;
      if (s > 0.f && isfinite(s)) {
        const float x = (log10f(s) + 4.f) * (64.f / 6.f);
        b = x <= 0.f ? 0 : (x >= 63.f ? 63 : (int)x);
      }
      atomicAdd(&h[b], 1);
    }
  }
  __syncthreads();
  if (threadIdx.x < 64) {
    int t = 0;
    for (int q = 0; q < 32; ++q) t += hist[q][threadIdx.x];
    total[threadIdx.x] = t;
  }
  __syncthreads();
  float* f = d.feat + (size_t)w * lam::NF;
  const WinConst& wc = d.wc[w];
  if (threadIdx.x < 64) f[3 + threadIdx.x] = (float)total[threadIdx.x] / (float)(ns * nwin);
  if (threadIdx.x == 0) {
    f[0] = asinhf((float)(wc.alpha * 1000.0)) * 0.125f;
    f[1] = asinhf((float)(wc.mu * 1000.0)) * 0.125f;
    f[2] = asinhf((float)(wc.sigma * 1000.0)) * 0.125f;
  }
}

size_t lambda_smem() { return sizeof(lam::Smem); }

cudaError_t launch_lambda_features(const Problem& pb, const DeviceBuffers& d, cudaStream_t s) {
  k_lambda_features<<<pb.W, 1024, 0, s>>>(pb, d);
  return cudaGetLastError();
}

// Proposals of the batch's windows into d.prop; the narrow search of each
// window starts from them (launch_search_hint).
cudaError_t launch_lambda_propose(const Problem& pb, const DeviceBuffers& d, cudaStream_t s) {
  lam::k_mlp_forward<<<(pb.W + lam::GS - 1) / lam::GS, lam::PT, lambda_smem(), s>>>(
      d.model, (const lam::Shadow*)d.model_bf16, d.feat, pb.W, d.prop,
      d.prop_out ? d.prop_out + d.win0 : nullptr);
  return cudaGetLastError();
}

// ---- training / inference launchers (device buffers)
cudaError_t lambda_shadow(const float* m, void* wbf, cudaStream_t s) {
  lam::k_mlp_shadow<<<64, 256, 0, s>>>(m, (lam::Shadow*)wbf);
  return cudaGetLastError();
}

// blocks of a pass over n rows: at most two per SM (their shared memory)
static int pass_blocks(int n) {
  int dev = 0, sms = 1;
  if (cudaGetDevice(&dev) == cudaSuccess)
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return std::min((n + lam::GS - 1) / lam::GS, 2 * sms);
}

size_t lambda_rows(int n) { return ((size_t)n + 31) / 32 * 32; }
size_t lambda_act_floats(int n) { return lambda_rows(n) * (lam::ACT_N * lam::H + 2); }

cudaError_t lambda_forward(const float* m, const void* wbf, const float* feat, int n, float* y,
                           cudaStream_t s) {
  lam::k_mlp_forward<<<pass_blocks(n), lam::PT, lambda_smem(), s>>>(
      m, (const lam::Shadow*)wbf, feat, n, y, nullptr);
  return cudaGetLastError();
}

// Gradients of the rows of a pass into grad, or with ADAM the parameter update.
// By chains from where two launches are faster than one (equal at 512 rows; 4
// epochs of 8 steps of 8,192 rows 9.4 -> 5.5 ms).
static bool by_chains(size_t rows) { return rows > 512; }
// The sums of at most kSlab chains (65,536 rows, 343 MB) are held at a time; a batch of
// training has no more than 256.
constexpr size_t kSlab = 2048;

template <bool ADAM>
static void launch_update(float* m, lam::Shadow* wbf, float* mom1, float* mom2, const float* act,
                          const float* dO, const float* err, int rows_pad, float* part,
                          const int* epoch, int step, const lam::AdamCfg& c, float* grad,
                          float* loss, cudaStream_t s) {
  if (by_chains(rows_pad)) {
    for (int c0 = 0; c0 < rows_pad / 32; c0 += (int)kSlab) {
      const int nch = std::min((int)kSlab, rows_pad / 32 - c0);
      lam::k_mlp_chains<<<dim3(nch, 4), lam::CT, 0, s>>>(act, dO, err, rows_pad, c0, part, loss);
      lam::k_mlp_sum<ADAM><<<(lam::NPARAM + 127) / 128, 128, 0, s>>>(
          m, wbf, mom1, mom2, part, nch, c0 > 0, epoch, step, c, grad);
    }
  } else {
    lam::k_mlp_update<ADAM><<<lam::kUpdateBlocks, lam::H * lam::NCH, 0, s>>>(
        m, wbf, mom1, mom2, act, dO, err, rows_pad, epoch, step, c, grad, loss);
  }
}
// floats of the chains' sums of n rows (0: not needed)
size_t lambda_part_floats(int n) {
  const size_t r = lambda_rows(n);
  return by_chains(r) ? std::min(r / 32, kSlab) * lam::NPARAM : 0;
}
int lambda_update_launches(int n) {
  const size_t r = lambda_rows(n);
  return by_chains(r) ? 2 * (int)((r / 32 + kSlab - 1) / kSlab) : 1;
}

// Gradient over n samples: act holds lambda_act_floats(n) floats, part
// lambda_part_floats(n), part_loss the squared error of each 32 samples.
cudaError_t lambda_grad(const float* m, const void* wbf, const float* feat, const float* target,
                        int n, float* act, float* part, float* part_loss, float* grad,
                        cudaStream_t s) {
  const int rp = (int)lambda_rows(n);
  float* dO = act + (size_t)rp * lam::ACT_N * lam::H;
  lam::k_mlp_pass<<<pass_blocks(rp), lam::PT, lambda_smem(), s>>>(
      m, (const lam::Shadow*)wbf, feat, target, nullptr, nullptr, 0, 0, n, rp, 1.f / (float)n, act,
      dO, dO + rp);
  launch_update<false>(nullptr, nullptr, nullptr, nullptr, act, dO, dO + rp, rp, part, nullptr, 0,
                       lam::AdamCfg{}, grad, part_loss, s);
  return cudaGetLastError();
}

cudaError_t lambda_attrs() {
  const int shm = (int)lambda_smem();
  cudaError_t e = cudaFuncSetAttribute(lam::k_mlp_pass, cudaFuncAttributeMaxDynamicSharedMemorySize, shm);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(lam::k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, shm);
  return e;
}

// One epoch of training (stream-capturable: launches only; lambda_attrs()
// must have run).
cudaError_t lambda_train_epoch(const LambdaTrain& t, cudaStream_t s) {
  const int nblk = t.batch / 32, blocks = pass_blocks(t.batch);
  float* dO = t.act + (size_t)t.batch * lam::ACT_N * lam::H;
  lam::AdamCfg c{t.lr, t.lr_final, t.wd, t.b1, t.b2, t.eps, t.steps, t.total_steps};
  for (int st = 0; st < t.steps; ++st) {
    lam::k_mlp_pass<<<blocks, lam::PT, lambda_smem(), s>>>(
        t.m, (const lam::Shadow*)t.wbf, t.feat, t.target, t.perm, t.epoch, t.n, st * t.batch,
        t.n, t.batch, 1.f / (float)t.batch, t.act, dO, dO + t.batch);
    launch_update<true>(t.m, (lam::Shadow*)t.wbf, t.mom1, t.mom2, t.act, dO, dO + t.batch, t.batch,
                        t.part, t.epoch, st, c, nullptr, t.loss_acc + (size_t)st * nblk, s);
  }
  lam::k_mlp_epoch_end<<<1, 32, 0, s>>>(t.loss_acc, t.steps, nblk, t.steps * t.batch, t.epoch,
                                        t.epoch_loss);
  return cudaGetLastError();
}

}  // namespace pgsvt
