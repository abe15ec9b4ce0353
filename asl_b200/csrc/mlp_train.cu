// Learned closure, training side: the network's forward and backward passes
// and an Adam update, as the project's own kernels. Parameters are FP32
// (master copy); the inference layout (MlpNet) rounds the weights to BF16.
//
// Parameter vector (MLP_P floats): W1[64][9], b1[64], W2[64][64], b2[64],
// w3[64], b3. The model is
//   x' = (x - shift) * scale,  h1 = relu(W1 x' + b1),  h2 = relu(W2 h1 + b2),
//   y = w3 . h2 + b3,  Cs^2 = out_scale * softplus(y),
// and the loss the mean squared error of Cs^2 against the targets.
//
// k_mlp_grad: a fixed grid of blocks; each block takes chunks of 128 samples,
// keeps the chunk's activations in shared memory, and runs both passes as
// block-wide matrix products with register tiles. Each block writes one row
// of partial sums; k_mlp_reduce adds the rows in a fixed order, so gradients
// are deterministic.
#include <cuda_bf16.h>
#include <cstring>
#include <string>
#include <vector>
#include "aslb.h"
#include "f32x2.cuh"
#include "kernels.h"
#include "mlp.cuh"
#include "per_device.h"

namespace aslb {

constexpr int kIn = kMlpIn, kH = kMlpHidden;
constexpr int oW1 = 0, oB1 = oW1 + kH * kIn, oW2 = oB1 + kH, oB2 = oW2 + kH * kH, oW3 = oB2 + kH, oB3 = oW3 + kH;
constexpr int kParams = oB3 + 1;
constexpr int kChunk = 128;
constexpr int kGradThreads = 512;
constexpr int kLd = kChunk + 4;  // row stride of the activation tiles: consecutive rows start 4 banks apart
constexpr int kWd = kH + 4;      // row stride of the weight tiles

__device__ __forceinline__ float softplus_f(float y) { return y > 20.f ? y : log1pf(expf(y)); }
__device__ __forceinline__ float sigmoid_f(float y) { return 1.f / (1.f + expf(-y)); }

// Shared memory of one block (floats).
struct GradTile {
  float w2[kH * kWd];    // W2[m][j]
  float w2t[kH * kWd];   // W2[m][j] at [j][m]
  float w1t[kIn * kWd];  // W1[k][j] at [j][k]
  float b1[kH], b2[kH], w3[kH];
  float h1[kH * kLd];    // [unit][sample]: activations, then their gradients
  float h2[kH * kLd];
  float x[kIn * kLd];
  float dy[kChunk], e2[kChunk], yp[4 * kChunk];
};

// acc[r][c] += w[r] * v[c] for four rows and four samples (packed in pairs).
__device__ __forceinline__ void outer_4x4(F2 (&acc)[4][2], const float4& w, const float4& va) {
  const F2 v[2] = {F2(va.x, va.y), F2(va.z, va.w)};
  const float ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const F2 wr = F2(ws[r]);
#pragma unroll
    for (int c = 0; c < 2; ++c) acc[r][c] = fma_(wr, v[c], acc[r][c]);
  }
}
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
__device__ __forceinline__ float dot4(const float4& a, const float4& b, float s) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s))));
}

// One chunk is three 64 x 64 x 128 matrix products (layer 2, its weight
// gradient, its input gradient) and two of a seventh of that size, all in
// FP32. The block keeps the chunk's activations unit-major in shared memory
// and every thread accumulates a 4 x 4 register tile with packed FP32
// instructions, eight of them per two 16-byte shared loads (weight gradient:
// 32 per eight loads, half of the samples per half of the block); the weight
// gradients stay in registers across a block's chunks. A batch of 16,384 is
// 128 chunks, one block each, so a chunk's own time counts: bound by the
// FP32 units (7.6 us at their peak) and the latency of ten block-wide phases.
// Gradient and reduction of that batch: 24.6 us, 26.7 with 256 threads and
// 4 x 8 tiles; one sample per thread with a scalar shared load per
// multiply-add took 71 with its Adam step, this 31.
__global__ void __launch_bounds__(kGradThreads)
    k_mlp_grad(const float* __restrict__ params, const float* __restrict__ X, const float* __restrict__ T,
               long long n, const float* __restrict__ norm, float out_scale, float inv_count,
               float* __restrict__ partials) {
  extern __shared__ __align__(16) unsigned char grad_smem_raw[];
  GradTile& S = *reinterpret_cast<GradTile*>(grad_smem_raw);
  const int t = threadIdx.x;
  for (int i = t; i < kH * kH; i += kGradThreads) {
    const float v = params[oW2 + i];
    const int m = i / kH, j = i % kH;
    S.w2[m * kWd + j] = v;
    S.w2t[j * kWd + m] = v;
  }
  for (int i = t; i < kH * kIn; i += kGradThreads) S.w1t[(i % kIn) * kWd + i / kIn] = params[oW1 + i];
  if (t < kH) {
    S.b1[t] = params[oB1 + t];
    S.b2[t] = params[oB2 + t];
    S.w3[t] = params[oW3 + t];
  }
  const float b3 = params[oB3];
  // register tiles: rows 4 rg .. 4 rg + 3, samples sa .. sa + 3 (a warp: two
  // row groups, 64 samples)
  const int rg = (t >> 6) * 2 + ((t >> 4) & 1), sa = 64 * ((t >> 5) & 1) + 4 * (t & 15);
  // per-unit sums: unit m, samples 4 (q + 8 i) .. + 3
  const int m = t >> 3, q = t & 7;
  // W2's gradient: rows gr + 16 r, columns gc + 16 c over half of the samples;
  // the halves of a pair are even and odd samples
  const int gr = (t >> 4) & 15, gc = t & 15, gs = (t >> 8) * (kChunk / 2);
  F2 gw2[4][4];
  float gw1[kIn], gb1 = 0.f, gb2 = 0.f, gw3 = 0.f, gb3 = 0.f, loss = 0.f;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) gw2[r][c] = F2(0.f);
#pragma unroll
  for (int j = 0; j < kIn; ++j) gw1[j] = 0.f;

  const long long nchunks = (n + kChunk - 1) / kChunk;
  for (long long ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
    const long long i0 = ch * kChunk;
    __syncthreads();  // the previous chunk (or the weights) is done with
    for (int e = t; e < kIn * kChunk; e += kGradThreads) {
      const int j = e / kChunk, s = e % kChunk;
      S.x[j * kLd + s] = i0 + s < n ? (X[(long long)j * n + i0 + s] - norm[j]) * norm[kIn + j] : 0.f;
    }
    const bool valid = t < kChunk && i0 + t < n;
    const float target = valid ? T[i0 + t] : 0.f;
    __syncthreads();
    F2 acc[4][2];
    auto bias = [&](const float* b) {
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) acc[r][c] = F2(b[4 * rg + r]);
    };
    auto put_relu = [&](float* h) {
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        float* row = h + (4 * rg + r) * kLd;
        st4(row + sa, fmaxf(acc[r][0].lo(), 0.f), fmaxf(acc[r][0].hi(), 0.f), fmaxf(acc[r][1].lo(), 0.f),
            fmaxf(acc[r][1].hi(), 0.f));
      }
    };
    // h1 = relu(W1 x' + b1), h2 = relu(W2 h1 + b2)
    bias(S.b1);
#pragma unroll
    for (int j = 0; j < kIn; ++j)
      outer_4x4(acc, ld4(S.w1t + j * kWd + 4 * rg), ld4(S.x + j * kLd + sa));
    put_relu(S.h1);
    __syncthreads();
    bias(S.b2);
#pragma unroll 4
    for (int j = 0; j < kH; ++j)
      outer_4x4(acc, ld4(S.w2t + j * kWd + 4 * rg), ld4(S.h1 + j * kLd + sa));
    put_relu(S.h2);
    __syncthreads();
    // y, four quarters of the units per sample; the loss and its derivative
    {
      const int s = t & (kChunk - 1), k0 = (t >> 7) * (kH / 4);
      float a = 0.f;
#pragma unroll 8
      for (int k = 0; k < kH / 4; ++k) a = fmaf(S.w3[k0 + k], S.h2[(k0 + k) * kLd + s], a);
      S.yp[t] = a;
    }
    __syncthreads();
    if (t < kChunk) {
      const float y = b3 + ((S.yp[t] + S.yp[kChunk + t]) + (S.yp[2 * kChunk + t] + S.yp[3 * kChunk + t]));
      const float e = out_scale * softplus_f(y) - target;
      S.dy[t] = valid ? 2.f * e * out_scale * sigmoid_f(y) * inv_count : 0.f;
      S.e2[t] = valid ? e * e : 0.f;
    }
    __syncthreads();
    // w3's gradient, then dh2 = dy w3 [h2 > 0] in place, and b2's gradient
    {
      const float w = S.w3[m];
#pragma unroll
      for (int i = 0; i < kChunk / 32; ++i) {
        float* p = S.h2 + m * kLd + 4 * (q + 8 * i);
        const float4 h = ld4(p), d = ld4(S.dy + 4 * (q + 8 * i));
        gw3 = dot4(h, d, gw3);
        const float a = h.x > 0.f ? d.x * w : 0.f, b = h.y > 0.f ? d.y * w : 0.f, c = h.z > 0.f ? d.z * w : 0.f,
                    f = h.w > 0.f ? d.w * w : 0.f;
        gb2 += (a + b) + (c + f);
        st4(p, a, b, c, f);
      }
      if (t < 32) {
        const float4 d = ld4(S.dy + 4 * t), e = ld4(S.e2 + 4 * t);
        gb3 += (d.x + d.y) + (d.z + d.w);
        loss += (e.x + e.y) + (e.z + e.w);
      }
    }
    __syncthreads();
    // W2's gradient: sum over samples of dh2[m][s] h1[j][s]
#pragma unroll 2
    for (int s = gs; s < gs + kChunk / 2; s += 4) {
      float4 d[4], h[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        d[r] = ld4(S.h2 + (gr + 16 * r) * kLd + s);
        h[r] = ld4(S.h1 + (gc + 16 * r) * kLd + s);
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          gw2[r][c] = fma_(F2(d[r].x, d[r].y), F2(h[c].x, h[c].y), gw2[r][c]);
          gw2[r][c] = fma_(F2(d[r].z, d[r].w), F2(h[c].z, h[c].w), gw2[r][c]);
        }
    }
    // dh1[j][s] = [h1 > 0] sum_m W2[m][j] dh2[m][s], over h1 once nobody reads it
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 2; ++c) acc[r][c] = F2(0.f);
#pragma unroll 4
    for (int k = 0; k < kH; ++k)
      outer_4x4(acc, ld4(S.w2 + k * kWd + 4 * rg), ld4(S.h2 + k * kLd + sa));
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      float* p = S.h1 + (4 * rg + r) * kLd + sa;
      const float4 h = ld4(p);
      st4(p, h.x > 0.f ? acc[r][0].lo() : 0.f, h.y > 0.f ? acc[r][0].hi() : 0.f, h.z > 0.f ? acc[r][1].lo() : 0.f,
          h.w > 0.f ? acc[r][1].hi() : 0.f);
    }
    __syncthreads();
    // W1's and b1's gradients
#pragma unroll 2
    for (int i = 0; i < kChunk / 32; ++i) {
      const int s = 4 * (q + 8 * i);
      const float4 d = ld4(S.h1 + m * kLd + s);
      gb1 += (d.x + d.y) + (d.z + d.w);
#pragma unroll
      for (int j = 0; j < kIn; ++j) gw1[j] = dot4(d, ld4(S.x + j * kLd + s), gw1[j]);
    }
  }
  // this block's row of partial sums
  float* G = partials + (long long)blockIdx.x * (kParams + 1);
  __syncthreads();  // the activations are done with: their memory passes half of W2's gradient
  for (int half = 1; half >= 0; --half) {
    if ((t >> 8) == half) {
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int e = (gr + 16 * r) * kH + gc + 16 * c;
          const float v = gw2[r][c].lo() + gw2[r][c].hi();
          if (half) S.h1[e] = v;
          else G[oW2 + e] = v + S.h1[e];
        }
    }
    __syncthreads();
  }
  auto quad = [](float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    return v + __shfl_xor_sync(0xffffffffu, v, 4);
  };
  gb1 = quad(gb1);
  gb2 = quad(gb2);
  gw3 = quad(gw3);
#pragma unroll
  for (int j = 0; j < kIn; ++j) {
    const float v = quad(gw1[j]);
    if (q == 0) G[oW1 + m * kIn + j] = v;
  }
  if (q == 0) {
    G[oB1 + m] = gb1;
    G[oB2 + m] = gb2;
    G[oW3 + m] = gw3;
  }
  if (t < 32) {
    for (int o = 16; o > 0; o >>= 1) {
      gb3 += __shfl_xor_sync(0xffffffffu, gb3, o);
      loss += __shfl_xor_sync(0xffffffffu, loss, o);
    }
    if (t == 0) {
      G[oB3] = gb3;
      G[kParams] = loss;
    }
  }
}

// Sum of the blocks' rows: 32 columns per block, eight threads per column
// (each every eighth row, in order), then the eight in order.
constexpr int kReduceCols = 32, kReduceWays = 8;
__global__ void __launch_bounds__(kReduceCols * kReduceWays)
    k_mlp_reduce(const float* __restrict__ partials, int rows, float* __restrict__ grad_loss) {
  __shared__ float sh[kReduceWays][kReduceCols];
  const int c = threadIdx.x % kReduceCols, w = threadIdx.x / kReduceCols;
  const int i = blockIdx.x * kReduceCols + c;
  float a = 0.f;
  if (i <= kParams) {
#pragma unroll 8
    for (int r = w; r < rows; r += kReduceWays) a += partials[(long long)r * (kParams + 1) + i];
  }
  sh[w][c] = a;
  __syncthreads();
  if (w == 0 && i <= kParams) {
#pragma unroll
    for (int k = 1; k < kReduceWays; ++k) a += sh[k][c];
    grad_loss[i] = a;
  }
}

__global__ void k_mlp_adam(float* __restrict__ params, const float* __restrict__ grad, float* __restrict__ m,
                           float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kParams) return;
  const float g = grad[i];
  const float mi = b1 * m[i] + (1.f - b1) * g;
  const float vi = b2 * v[i] + (1.f - b2) * g * g;
  m[i] = mi;
  v[i] = vi;
  params[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

}  // namespace aslb

using namespace aslb;

namespace {
constexpr int kGradBlocks = 148;
size_t grad_smem() { return sizeof(GradTile); }
int err(const char* what, cudaError_t e) {
  set_last_error(std::string(what) + ": " + cudaGetErrorString(e));
  return ASLB_ERR_CUDA;
}
int arg_err(const char* what) {
  set_last_error(std::string(what) + ": bad arguments");
  return ASLB_ERR_ARG;
}
}  // namespace

extern "C" {

int aslb_mlp_param_count(void) { return kParams; }

size_t aslb_mlp_grad_scratch_floats(void) { return (size_t)kGradBlocks * (kParams + 1); }

int aslb_mlp_grad(const float* params, const float* x, const float* t, long long n, const float* norm,
                  float out_scale, float* scratch, float* grad_loss, void* stream) {
  if (!params || !x || !t || !norm || !scratch || !grad_loss || n <= 0) return arg_err("aslb_mlp_grad");
  static PerDevice configured;
  int dev = 0, limit = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess)
    e = configured.get(dev, limit, [](int& n) {
      n = (int)grad_smem();
      return cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, n);
    });
  if (e != cudaSuccess) return err("aslb_mlp_grad", e);
  cudaStream_t st = (cudaStream_t)stream;
  const long long chunks = (n + kChunk - 1) / kChunk;
  const int blocks = (int)(chunks < kGradBlocks ? chunks : kGradBlocks);
  k_mlp_grad<<<blocks, kGradThreads, grad_smem(), st>>>(params, x, t, n, norm, out_scale, 1.f / (float)n, scratch);
  k_mlp_reduce<<<(kParams + kReduceCols) / kReduceCols, kReduceCols * kReduceWays, 0, st>>>(scratch, blocks, grad_loss);
  e = cudaGetLastError();
  return e == cudaSuccess ? ASLB_OK : err("aslb_mlp_grad", e);
}

int aslb_mlp_adam(float* params, const float* grad, float* m, float* v, int step, float lr, float beta1,
                  float beta2, float eps, void* stream) {
  if (!params || !grad || !m || !v || step < 1) return arg_err("aslb_mlp_adam");
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  k_mlp_adam<<<(kParams + 255) / 256, 256, 0, (cudaStream_t)stream>>>(params, grad, m, v, lr, beta1, beta2, eps,
                                                                       c1, c2);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? ASLB_OK : err("aslb_mlp_adam", e);
}

int aslb_mlp_pack(const float* params_host, const float* norm_host, float out_scale, void* net_host) {
  if (!params_host || !norm_host || !net_host) return arg_err("aslb_mlp_pack");
  MlpNet net;
  std::memset(&net, 0, sizeof(net));
  for (int j = 0; j < kMlpInPad; ++j) {
    net.in_shift[j] = j < kIn ? norm_host[j] : 0.f;
    net.in_scale[j] = j < kIn ? norm_host[kIn + j] : 0.f;
  }
  for (int k = 0; k < kH; ++k) {
    for (int j = 0; j < kMlpInPad; ++j)
      net.w1[k][j] = __float2bfloat16_rn(j < kIn ? params_host[oW1 + k * kIn + j] : 0.f);
    net.b1[k] = params_host[oB1 + k];
    for (int j = 0; j < kH; ++j) net.w2[k][j] = __float2bfloat16_rn(params_host[oW2 + k * kH + j]);
    net.b2[k] = params_host[oB2 + k];
    net.w3[k] = __float2bfloat16_rn(params_host[oW3 + k]);
  }
  net.b3 = params_host[oB3];
  net.out_scale = out_scale;
  std::memcpy(net_host, &net, sizeof(net));
  return ASLB_OK;
}

}  // extern "C"
