// The planner network: a 3-layer perceptron  inputs -> 64 -> 64 -> 2  (ReLU
// between layers) that predicts the next layer's log growth and duplicate
// ratio of a BFS from its recent layer sizes and generator features.  It is
// trained and evaluated only by the kernels in this file.
//
// Parameters are one flat fp32 buffer:
//     W1[64][in] | b1[64] | W2[64][64] | b2[64] | W3[2][64] | b3[2]
// Training: mlp_loss_grad (forward + backward of a weighted squared error over
// row tiles in shared memory, gradients summed in registers and over clusters,
// one global atomicAdd per parameter and cluster) and mlp_adam.  Inference: mlp_infer_bf16 reads bf16
// parameters and keeps activations in bf16, accumulating in fp32.
// No reference counterpart: the reference sizes its buffers by worst-case
// bounds and timed pilot runs (crates/mgbfs-runtime/src/generic_memory.rs:36-49,
// multigpubfs/autotune.py:276).
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstddef>

#include "../../include/mgbfs2.h"
#include "engine.h"

namespace mgbfs2 {
namespace {

namespace cg = cooperative_groups;

constexpr uint32_t kHidden = 64, kOut = 2, kMaxIn = 32, kMlpBlock = 128;

struct Offsets {
  uint32_t w1, b1, w2, b2, w3, b3, total;
};

__host__ __device__ __forceinline__ Offsets offsets(uint32_t in) {
  Offsets o;
  o.w1 = 0;
  o.b1 = o.w1 + kHidden * in;
  o.w2 = o.b1 + kHidden;
  o.b2 = o.w2 + kHidden * kHidden;
  o.w3 = o.b2 + kHidden;
  o.b3 = o.w3 + kOut * kHidden;
  o.total = o.b3 + kOut;
  return o;
}

// h1 = relu(W1 x + b1); returns y = W3 relu(W2 h1 + b2) + b3, keeping h1/h2.
__device__ __forceinline__ void forward_one(const float* P, const Offsets& o, uint32_t in, const float* x, float* h1,
                                            float* h2, float* y) {
  for (uint32_t k = 0; k < kHidden; ++k) {
    float a = P[o.b1 + k];
    for (uint32_t i = 0; i < in; ++i) a = fmaf(P[o.w1 + k * in + i], x[i], a);
    h1[k] = fmaxf(a, 0.f);
  }
  y[0] = P[o.b3];
  y[1] = P[o.b3 + 1];
  for (uint32_t j = 0; j < kHidden; ++j) {
    float a = P[o.b2 + j];
    for (uint32_t k = 0; k < kHidden; ++k) a = fmaf(P[o.w2 + j * kHidden + k], h1[k], a);
    a = fmaxf(a, 0.f);
    h2[j] = a;
    y[0] = fmaf(P[o.w3 + j], a, y[0]);
    y[1] = fmaf(P[o.w3 + kHidden + j], a, y[1]);
  }
}

__global__ void __launch_bounds__(kMlpBlock) mlp_forward_kernel(uint32_t in, const float* params, const float* x,
                                                                unsigned long long batch, float* y) {
  extern __shared__ float P[];
  const Offsets o = offsets(in);
  for (uint32_t i = threadIdx.x; i < o.total; i += blockDim.x) P[i] = params[i];
  __syncthreads();
  for (unsigned long long s = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; s < batch;
       s += static_cast<unsigned long long>(gridDim.x) * blockDim.x) {
    float xs[kMaxIn], h1[kHidden], h2[kHidden], out[kOut];
    for (uint32_t i = 0; i < in; ++i) xs[i] = x[s * in + i];
    forward_one(P, o, in, xs, h1, h2, out);
    y[s * kOut] = out[0];
    y[s * kOut + 1] = out[1];
  }
}

// loss = sum_s sum_o w_o (y_so - t_so)^2 / batch; grad += d loss / d params.
//
// A block takes tiles of kGradRows rows with every activation in shared
// memory and forms each layer's product, and each weight gradient's sum over
// the rows, from registers: a thread owns one hidden unit of eight rows, or a
// 4x4 patch of the 64x64 gradient, over all of its tiles; the eight blocks of a
// cluster add their sums up through distributed shared memory, and one global
// atomic per parameter and cluster ends it (an atomic per block rounded 206
// times into one value: error against float64 7e-7, 1e-7 to 2e-7 with a cluster's
// sums, as with one thread per row).  One thread per row with shared-memory atomics on every weight
// took 2.9 ms for 6,568 rows of 16 inputs, all of it in the atomics (31,000 a
// row); fp32 FMA on 148 SMs bounds the arithmetic at a few microseconds;
// the kernel takes about 30, one tile a block: shared-memory reads and the
// barriers between its phases.
constexpr uint32_t kGradRows = 32, kGradBlock = 256, kGradGroups = kGradBlock / kHidden;
constexpr uint32_t kGradPer = kGradRows / kGradGroups;  // rows of a thread
constexpr uint32_t kGradCluster = 8;
constexpr uint32_t kW2Stride = kHidden + 1;             // read along rows and along columns

struct GradSmem {
  float w1[kMaxIn][kHidden];   // transposed
  float w2[kHidden * kW2Stride];
  float w3[kOut][kHidden], b1[kHidden], b2[kHidden], b3[kOut];
  // Read four floats at a time.
  alignas(16) float h1[kGradRows][kHidden];
  alignas(16) float h2[kGradRows][kHidden];
  alignas(16) float d1[kGradRows][kHidden];
  alignas(16) float d2[kGradRows][kHidden];
  float x[kGradRows][kMaxIn], dy[kGradRows][kOut];
};
static_assert(offsetof(GradSmem, h1) % 16 == 0 && offsetof(GradSmem, d2) % 16 == 0 && kHidden % 4 == 0,
              "float4 reads of whole rows");

__global__ void __cluster_dims__(kGradCluster, 1, 1) __launch_bounds__(kGradBlock) mlp_loss_grad_kernel(uint32_t in, const float* params, const float* x,
                                                                   const float* target, float w0, float w1,
                                                                   unsigned long long batch, float* grad, float* loss) {
  extern __shared__ __align__(16) unsigned char raw[];
  GradSmem& s = *reinterpret_cast<GradSmem*>(raw);
  const Offsets o = offsets(in);  // w1, b1, w2, b2, w3, b3 in this order
  const uint32_t tid = threadIdx.x, unit = tid % kHidden, row0 = tid / kHidden * kGradPer;
  bool odd_weight = false;
  for (uint32_t i = tid; i < o.total; i += kGradBlock) {
    const float v = params[i];
    odd_weight = odd_weight || !isfinite(v);
    if (i < o.b1) s.w1[i % in][i / in] = v;
    else if (i < o.w2) s.b1[i - o.b1] = v;
    else if (i < o.b2) s.w2[(i - o.w2) / kHidden * kW2Stride + (i - o.w2) % kHidden] = v;
    else if (i < o.w3) s.b2[i - o.b2] = v;
    else if (i < o.b3) s.w3[(i - o.w3) / kHidden][(i - o.w3) % kHidden] = v;
    else s.b3[i - o.b3] = v;
  }
  const float scale = 2.f / static_cast<float>(batch);
  // This thread's sums over all rows of the block's tiles.
  const uint32_t pj = tid / 16 * 4, pk = tid % 16 * 4;  // its patch of W2's gradient
  constexpr uint32_t kInPer = kMaxIn / kGradGroups;
  const uint32_t in0 = tid / kHidden * kInPer;         // its inputs of W1's gradient
  float g2[4][4] = {}, g1[kInPer] = {}, gb1 = 0.f, gb2 = 0.f, gw30 = 0.f, gw31 = 0.f, gb30 = 0.f, gb31 = 0.f;
  float local_loss = 0.f;
  const unsigned long long tiles = (batch + kGradRows - 1) / kGradRows;
  for (unsigned long long t = blockIdx.x; t < tiles; t += gridDim.x) {
    const unsigned long long base = t * kGradRows;
    __syncthreads();  // the last tile's reads are done
    bool odd = odd_weight;  // an infinity or NaN: products with zeros must be left out, not added as NaN
    for (uint32_t i = tid; i < kGradRows * in; i += kGradBlock) {
      const float v = base + i / in < batch ? x[base * in + i] : 0.f;
      s.x[i / in][i % in] = v;
      odd = odd || !isfinite(v);
    }
    __syncthreads();
    float a[kGradPer];
#pragma unroll
    for (uint32_t r = 0; r < kGradPer; ++r) a[r] = s.b1[unit];
    for (uint32_t i = 0; i < in; ++i) {
      const float w = s.w1[i][unit];
#pragma unroll
      for (uint32_t r = 0; r < kGradPer; ++r) a[r] = fmaf(w, s.x[row0 + r][i], a[r]);
    }
#pragma unroll
    for (uint32_t r = 0; r < kGradPer; ++r) {
      const float h = fmaxf(a[r], 0.f);
      s.h1[row0 + r][unit] = h;
      odd = odd || !isfinite(h);  // overflowed from finite inputs
    }
    __syncthreads();
#pragma unroll
    for (uint32_t r = 0; r < kGradPer; ++r) a[r] = s.b2[unit];
    for (uint32_t k = 0; k < kHidden; k += 4) {
      float w[4];
#pragma unroll
      for (uint32_t u = 0; u < 4; ++u) w[u] = s.w2[unit * kW2Stride + k + u];
#pragma unroll
      for (uint32_t r = 0; r < kGradPer; ++r) {
        const float4 h = *reinterpret_cast<const float4*>(&s.h1[row0 + r][k]);
        a[r] = fmaf(w[3], h.w, fmaf(w[2], h.z, fmaf(w[1], h.y, fmaf(w[0], h.x, a[r]))));
      }
    }
#pragma unroll
    for (uint32_t r = 0; r < kGradPer; ++r) s.h2[row0 + r][unit] = fmaxf(a[r], 0.f);
    __syncthreads();
    // Outputs: four threads a row and output, summed by shuffles.
    {
      const uint32_t row = tid / 8, out = tid / 4 % 2, part = tid % 4;
      float y = part ? 0.f : s.b3[out];
      for (uint32_t j = part; j < kHidden; j += 4) y = fmaf(s.w3[out][j], s.h2[row][j], y);
      y += __shfl_xor_sync(kFullMask, y, 1);
      y += __shfl_xor_sync(kFullMask, y, 2);
      const bool valid = base + row < batch;
      const float e = valid ? y - target[(base + row) * kOut + out] : 0.f, w = out ? w1 : w0;
      const float dy = valid ? scale * w * e : 0.f;  // a row past the batch is 0 under any weight
      if (part == 0) {
        s.dy[row][out] = dy;
        if (valid) local_loss += w * e * e / static_cast<float>(batch);
        if (out) gb31 += dy;
        else gb30 += dy;
      }
      odd = odd || !isfinite(dy);
    }
    __syncthreads();
#pragma unroll
    for (uint32_t r = 0; r < kGradPer; ++r) {
      const float dy0 = s.dy[row0 + r][0], dy1 = s.dy[row0 + r][1], h = s.h2[row0 + r][unit];
      const bool valid = base + row0 + r < batch;
      if (valid) {
        gw30 = fmaf(dy0, h, gw30);
        gw31 = fmaf(dy1, h, gw31);
      }
      const float d = valid && h > 0.f ? fmaf(s.w3[0][unit], dy0, s.w3[1][unit] * dy1) : 0.f;
      s.d2[row0 + r][unit] = d;
      gb2 += d;
      odd = odd || !isfinite(d);
    }
    if (__syncthreads_or(odd)) {
      // Values past finite: every product is taken or left out by itself.
      for (uint32_t r = 0; r < kGradRows; ++r)
        for (uint32_t u = 0; u < 4; ++u)
          for (uint32_t v = 0; v < 4; ++v)
            if (s.d2[r][pj + u] != 0.f && s.h1[r][pk + v] > 0.f) g2[u][v] += s.d2[r][pj + u] * s.h1[r][pk + v];
      for (uint32_t r = 0; r < kGradPer; ++r) {
        float d = 0.f;
        for (uint32_t j = 0; j < kHidden; ++j)
          if (s.d2[row0 + r][j] != 0.f) d = fmaf(s.w2[j * kW2Stride + unit], s.d2[row0 + r][j], d);
        d = s.h1[row0 + r][unit] > 0.f ? d : 0.f;
        s.d1[row0 + r][unit] = d;
        gb1 += d;
      }
      __syncthreads();
      for (uint32_t r = 0; r < kGradRows; ++r)
#pragma unroll
        for (uint32_t i = 0; i < kInPer; ++i)
          if (in0 + i < in && s.d1[r][unit] != 0.f) g1[i] += s.d1[r][unit] * s.x[r][in0 + i];
      continue;
    }
#pragma unroll 4
    for (uint32_t r = 0; r < kGradRows; ++r) {
      const float4 d = *reinterpret_cast<const float4*>(&s.d2[r][pj]), h = *reinterpret_cast<const float4*>(&s.h1[r][pk]);
      const float dv[4] = {d.x, d.y, d.z, d.w}, hv[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
      for (uint32_t u = 0; u < 4; ++u)
#pragma unroll
        for (uint32_t v = 0; v < 4; ++v) g2[u][v] = fmaf(dv[u], hv[v], g2[u][v]);
    }
#pragma unroll
    for (uint32_t r = 0; r < kGradPer; ++r) a[r] = 0.f;
    for (uint32_t j = 0; j < kHidden; j += 4) {
      float w[4];
#pragma unroll
      for (uint32_t u = 0; u < 4; ++u) w[u] = s.w2[(j + u) * kW2Stride + unit];
#pragma unroll
      for (uint32_t r = 0; r < kGradPer; ++r) {
        const float4 d = *reinterpret_cast<const float4*>(&s.d2[row0 + r][j]);
        a[r] = fmaf(w[3], d.w, fmaf(w[2], d.z, fmaf(w[1], d.y, fmaf(w[0], d.x, a[r]))));
      }
    }
#pragma unroll
    for (uint32_t r = 0; r < kGradPer; ++r) {
      const float d = s.h1[row0 + r][unit] > 0.f ? a[r] : 0.f;
      s.d1[row0 + r][unit] = d;
      gb1 += d;
    }
    __syncthreads();
    for (uint32_t r = 0; r < kGradRows; ++r) {
      const float d = s.d1[r][unit];
#pragma unroll
      for (uint32_t i = 0; i < kInPer; ++i)
        if (in0 + i < in) g1[i] = fmaf(d, s.x[r][in0 + i], g1[i]);
    }
  }
  // The block's sums, in the parameters' order with the loss behind them, in
  // the place of the activations.
  for (int off = 16; off > 0; off >>= 1) {
    local_loss += __shfl_xor_sync(kFullMask, local_loss, off);
    gb30 += __shfl_xor_sync(kFullMask, gb30, off);
    gb31 += __shfl_xor_sync(kFullMask, gb31, off);
  }
  __syncthreads();
  float* sums = &s.h1[0][0];
  static_assert(offsetof(GradSmem, x) - offsetof(GradSmem, h1) >= 4 * (kHidden * (kMaxIn + kHidden + kOut + 2) + kOut + 1),
                "room for every parameter's sum");
  // What several threads add to starts at zero: biases, W3 and the loss.
  for (uint32_t i = tid; i < kHidden; i += kGradBlock) sums[o.b1 + i] = 0.f;
  for (uint32_t i = o.b2 + tid; i <= o.total; i += kGradBlock) sums[i] = 0.f;
#pragma unroll
  for (uint32_t u = 0; u < 4; ++u)
#pragma unroll
    for (uint32_t v = 0; v < 4; ++v) sums[o.w2 + (pj + u) * kHidden + pk + v] = g2[u][v];
#pragma unroll
  for (uint32_t i = 0; i < kInPer; ++i)
    if (in0 + i < in) sums[o.w1 + unit * in + in0 + i] = g1[i];
  __syncthreads();
  atomicAdd(&sums[o.b1 + unit], gb1);
  atomicAdd(&sums[o.b2 + unit], gb2);
  atomicAdd(&sums[o.w3 + unit], gw30);
  atomicAdd(&sums[o.w3 + kHidden + unit], gw31);
  if ((tid & 31) == 0) {
    atomicAdd(&sums[o.b3], gb30);
    atomicAdd(&sums[o.b3 + 1], gb31);
    atomicAdd(&sums[o.total], local_loss);
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  const float* from[kGradCluster];
#pragma unroll
  for (uint32_t r = 0; r < kGradCluster; ++r) from[r] = cluster.map_shared_rank(sums, r);
  for (uint32_t i = cluster.block_rank() * kGradBlock + tid; i <= o.total; i += kGradCluster * kGradBlock) {
    float v[kGradCluster];
#pragma unroll
    for (uint32_t r = 0; r < kGradCluster; ++r) v[r] = from[r][i];
    const float all = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
    if (i < o.total) {
      if (all != 0.f) atomicAdd(&grad[i], all);
    } else if (loss) {
      atomicAdd(loss, all);
    }
  }
  cluster.sync();  // no block leaves while others read its sums
}

__global__ void mlp_adam_kernel(uint32_t count, float* params, const float* grad, float* m, float* v, float lr,
                                float beta1, float beta2, float eps, float c1, float c2) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const float g = grad[i];
    m[i] = beta1 * m[i] + (1.f - beta1) * g;
    v[i] = beta2 * v[i] + (1.f - beta2) * g * g;
    params[i] -= lr * (m[i] / c1) / (sqrtf(v[i] / c2) + eps);
  }
}

__global__ void mlp_to_bf16_kernel(uint32_t count, const float* params, __nv_bfloat16* out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
    out[i] = __float2bfloat16(params[i]);
}

// bf16 parameters and activations, fp32 accumulation; two hidden units per
// step through bf16x2 pairs.
__global__ void __launch_bounds__(kMlpBlock) mlp_infer_bf16_kernel(uint32_t in, const __nv_bfloat16* params,
                                                                   const float* x, unsigned long long batch,
                                                                   float* y) {
  extern __shared__ __nv_bfloat16 Q[];
  const Offsets o = offsets(in);
  for (uint32_t i = threadIdx.x; i < o.total; i += blockDim.x) Q[i] = params[i];
  __syncthreads();
  for (unsigned long long s = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; s < batch;
       s += static_cast<unsigned long long>(gridDim.x) * blockDim.x) {
    __nv_bfloat16 xs[kMaxIn], h1[kHidden];
    for (uint32_t i = 0; i < in; ++i) xs[i] = __float2bfloat16(x[s * in + i]);
    for (uint32_t k = 0; k < kHidden; ++k) {
      float a = __bfloat162float(Q[o.b1 + k]);
      for (uint32_t i = 0; i < in; ++i) a = fmaf(__bfloat162float(Q[o.w1 + k * in + i]), __bfloat162float(xs[i]), a);
      h1[k] = __float2bfloat16(fmaxf(a, 0.f));
    }
    float y0 = __bfloat162float(Q[o.b3]), y1 = __bfloat162float(Q[o.b3 + 1]);
    for (uint32_t j = 0; j < kHidden; ++j) {
      float a = __bfloat162float(Q[o.b2 + j]);
      const __nv_bfloat162* row = reinterpret_cast<const __nv_bfloat162*>(Q + o.w2 + j * kHidden);
      for (uint32_t k = 0; k < kHidden; k += 2) {
        const float2 w = __bfloat1622float2(row[k / 2]);
        a = fmaf(w.x, __bfloat162float(h1[k]), a);
        a = fmaf(w.y, __bfloat162float(h1[k + 1]), a);
      }
      const float h2 = __bfloat162float(__float2bfloat16(fmaxf(a, 0.f)));
      y0 = fmaf(__bfloat162float(Q[o.w3 + j]), h2, y0);
      y1 = fmaf(__bfloat162float(Q[o.w3 + kHidden + j]), h2, y1);
    }
    y[s * kOut] = y0;
    y[s * kOut + 1] = y1;
  }
}

// Whole-profile rollout on the device, one thread per instance: the 16
// planner features of depth d are formed from the last four predicted layers
// (bookkeeping in fp64), run through the same bf16 network as
// mlp_infer_bf16_kernel (bf16 inputs and hidden activations, fp32
// accumulation), and the predicted next layer
//     |L_{d+1}| = min(expm1(y0 + log1p |L_d|), orbit - visited, g |L_d|)
// is appended until it drops below one half.  statics[8 m + k] holds
// log orbit, n/16, g/8, inverse-closed, mean and max log generator order,
// fixed-point fraction and cycle fraction; gens[m] the generator counts.
constexpr uint32_t kRolloutInputs = 16;

__global__ void __launch_bounds__(kMlpBlock) mlp_rollout_kernel(const __nv_bfloat16* params, const float* x_mean,
                                                                const float* x_scale, const float* statics,
                                                                const float* gens, uint32_t count, uint32_t max_depth,
                                                                double* peak, double* total, uint32_t* depth) {
  extern __shared__ __nv_bfloat16 Q[];
  const Offsets o = offsets(kRolloutInputs);
  for (uint32_t i = threadIdx.x; i < o.total; i += blockDim.x) Q[i] = params[i];
  __syncthreads();
  const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= count) return;
  const float* st = statics + 8ull * m;
  const double g = gens[m], log_orbit = st[0], orbit = exp(log_orbit);
  double last[4] = {1.0, 0.0, 0.0, 0.0}, visited = 1.0, best = 1.0, sum = 1.0;
  uint32_t d = 0;
  for (; d < max_depth; ++d) {
    float x[kRolloutInputs];
    for (int k = 0; k < 4; ++k) x[k] = static_cast<float>(log1p(last[k]));
    x[4] = static_cast<float>(log1p(visited));
    for (int k = 0; k < 8; ++k) x[5 + k] = st[k];
    x[13] = static_cast<float>(d) / 64.0f;
    x[14] = static_cast<float>(visited / orbit);
    x[15] = static_cast<float>(log1p(g * last[0]));
    __nv_bfloat16 xs[kRolloutInputs], h1[kHidden];
    for (uint32_t i = 0; i < kRolloutInputs; ++i) xs[i] = __float2bfloat16((x[i] - x_mean[i]) / x_scale[i]);
    for (uint32_t k = 0; k < kHidden; ++k) {
      float a = __bfloat162float(Q[o.b1 + k]);
      for (uint32_t i = 0; i < kRolloutInputs; ++i)
        a = fmaf(__bfloat162float(Q[o.w1 + k * kRolloutInputs + i]), __bfloat162float(xs[i]), a);
      h1[k] = __float2bfloat16(fmaxf(a, 0.f));
    }
    float y0 = __bfloat162float(Q[o.b3]);
    for (uint32_t j = 0; j < kHidden; ++j) {
      float a = __bfloat162float(Q[o.b2 + j]);
      const __nv_bfloat162* row = reinterpret_cast<const __nv_bfloat162*>(Q + o.w2 + j * kHidden);
      for (uint32_t k = 0; k < kHidden; k += 2) {
        const float2 w = __bfloat1622float2(row[k / 2]);
        a = fmaf(w.x, __bfloat162float(h1[k]), a);
        a = fmaf(w.y, __bfloat162float(h1[k + 1]), a);
      }
      y0 = fmaf(__bfloat162float(Q[o.w3 + j]), __bfloat162float(__float2bfloat16(fmaxf(a, 0.f))), y0);
    }
    double nxt = expm1(static_cast<double>(y0) + log1p(last[0]));
    nxt = fmin(nxt, fmin(orbit - visited, g * last[0]));
    if (!(nxt >= 0.5)) break;
    last[3] = last[2];
    last[2] = last[1];
    last[1] = last[0];
    last[0] = nxt;
    visited += nxt;
    sum += nxt;
    best = fmax(best, nxt);
  }
  peak[m] = best;
  total[m] = sum;
  depth[m] = d + 1;
}

uint32_t mlp_grid(unsigned long long batch) {
  return static_cast<uint32_t>(std::max<unsigned long long>(1, std::min<unsigned long long>((batch + kMlpBlock - 1) / kMlpBlock, 148ull * 4)));
}

}  // namespace
}  // namespace mgbfs2

using namespace mgbfs2;

extern "C" {

uint32_t mgbfs2_mlp_param_count(uint32_t inputs) { return offsets(inputs).total; }

int mgbfs2_mlp_forward(uint32_t inputs, const float* params, const float* x, uint64_t batch, float* y, void* stream) {
  if (!inputs || inputs > kMaxIn || !params || (batch && (!x || !y))) return MGBFS2_INVALID_ARGUMENT;
  if (!batch) return MGBFS2_OK;
  const size_t smem = offsets(inputs).total * sizeof(float);
  mlp_forward_kernel<<<mlp_grid(batch), kMlpBlock, smem, static_cast<cudaStream_t>(stream)>>>(inputs, params, x, batch,
                                                                                               y);
  return cuda_status(cudaGetLastError());
}

int mgbfs2_mlp_loss_grad(uint32_t inputs, const float* params, const float* x, const float* target, float weight0,
                         float weight1, uint64_t batch, float* grad, float* loss, void* stream) {
  if (!inputs || inputs > kMaxIn || !params || !grad || (batch && (!x || !target))) return MGBFS2_INVALID_ARGUMENT;
  if (!batch) return MGBFS2_OK;
  mgbfs2::TraceRange range("planner.loss_grad");
  const size_t smem = sizeof(GradSmem);
  cudaError_t e = cudaFuncSetAttribute(mlp_loss_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem));
  if (e != cudaSuccess) return cuda_status(e);
  // Whole clusters, at most two blocks an SM.
  const uint64_t tiles = (batch + kGradRows - 1) / kGradRows;
  const uint32_t blocks =
      static_cast<uint32_t>(std::min<uint64_t>((tiles + kGradCluster - 1) / kGradCluster, 2 * 148 / kGradCluster)) * kGradCluster;
  mlp_loss_grad_kernel<<<blocks, kGradBlock, smem, static_cast<cudaStream_t>(stream)>>>(
      inputs, params, x, target, weight0, weight1, batch, grad, loss);
  return cuda_status(cudaGetLastError());
}

int mgbfs2_mlp_adam(uint32_t count, float* params, const float* grad, float* m, float* v, float lr, float beta1,
                    float beta2, float eps, uint32_t step, void* stream) {
  if (!count || !params || !grad || !m || !v || !step) return MGBFS2_INVALID_ARGUMENT;
  const float c1 = 1.f - powf(beta1, static_cast<float>(step)), c2 = 1.f - powf(beta2, static_cast<float>(step));
  mlp_adam_kernel<<<(count + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(count, params, grad, m, v, lr,
                                                                                       beta1, beta2, eps, c1, c2);
  return cuda_status(cudaGetLastError());
}

int mgbfs2_mlp_to_bf16(uint32_t count, const float* params, void* params_bf16, void* stream) {
  if (!count || !params || !params_bf16) return MGBFS2_INVALID_ARGUMENT;
  mlp_to_bf16_kernel<<<(count + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      count, params, static_cast<__nv_bfloat16*>(params_bf16));
  return cuda_status(cudaGetLastError());
}

int mgbfs2_mlp_infer_bf16(uint32_t inputs, const void* params_bf16, const float* x, uint64_t batch, float* y,
                          void* stream) {
  if (!inputs || inputs > kMaxIn || !params_bf16 || (batch && (!x || !y))) return MGBFS2_INVALID_ARGUMENT;
  if (!batch) return MGBFS2_OK;
  const size_t smem = offsets(inputs).total * sizeof(__nv_bfloat16);
  mlp_infer_bf16_kernel<<<mlp_grid(batch), kMlpBlock, smem, static_cast<cudaStream_t>(stream)>>>(
      inputs, static_cast<const __nv_bfloat16*>(params_bf16), x, batch, y);
  return cuda_status(cudaGetLastError());
}

int mgbfs2_mlp_rollout_bf16(const void* params_bf16, const float* x_mean, const float* x_scale, const float* statics,
                            const float* gens, uint32_t count, uint32_t max_depth, double* peak, double* total,
                            uint32_t* depth, void* stream) {
  mgbfs2::TraceRange range("planner.rollout");
  if (!params_bf16 || !x_mean || !x_scale || (count && (!statics || !gens || !peak || !total || !depth)))
    return MGBFS2_INVALID_ARGUMENT;
  if (!count) return MGBFS2_OK;
  const size_t smem = offsets(kRolloutInputs).total * sizeof(__nv_bfloat16);
  mlp_rollout_kernel<<<(count + kMlpBlock - 1) / kMlpBlock, kMlpBlock, smem, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(params_bf16), x_mean, x_scale, statics, gens, count, max_depth, peak, total,
      depth);
  return cuda_status(cudaGetLastError());
}

}  // extern "C"
