// The boundary MLP of the learned-CDF sort: 16 -> 64 -> 64 -> 1, ReLU,
// BF16 weights with FP32 master copies, FP32 biases and FP32 accumulation.
// Training (forward + backward, FP32 activations) and Adam are hand-written
// for the CUDA cores: a block takes tiles of 64 rows and runs the layers as
// small matrix products in shared memory; the gradient stays in registers over
// a block's tiles and is added to the global one once per block.  Inference runs on the tensor cores
// (mlp.cuh).  No reference counterpart (the reference has no learned
// component).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "internal.hpp"
#include "mlp.cuh"

namespace rwt {

// parameter layout (FP32 master and gradients): W1 [64][16], b1 [64],
// W2 [64][64], b2 [64], W3 [64], b3 [1]
constexpr int kIn = kMlpIn, kH = kMlpHidden;
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kH * kIn, kOffW2 = kOffB1 + kH,
              kOffB2 = kOffW2 + kH * kH, kOffW3 = kOffB2 + kH, kOffB3 = kOffW3 + kH;
static_assert(kOffB3 + 1 == kMlpParams, "parameter layout");

__device__ __forceinline__ float bf16_round(float x) {
  return __bfloat162float(__float2bfloat16_rn(x));
}

// The training kernel: a block of 256 threads takes tiles of 64 rows.  Every
// product of a layer (forward, weight gradient, input gradient) is 64 x 64
// outputs, 4 x 4 per thread (thread = column group tx, row group ty), reduced
// over k with two 16-byte shared loads per 16 multiply-adds; operands that are
// reduced over both of their axes are kept in both orders.  The output layer
// needs no shared memory: 16 lanes hold a row's 64 hidden units.  The gradient
// stays in registers over the block's tiles and is added to the global one
// once per block.
//
// Bound by the FP32 pipe and the shared loads (about 3,600 multiply-adds per
// thread and tile), behind the latency of loading the parameters.  Before, a
// block of 128 threads took 32 rows with one dot product per output (eight
// rows of a warp on one bank) and added 5,313 values to global memory per 32
// rows: 63.6 us for 8,192 rows.
constexpr int kRows = 64, kMlpThreads = 256;
constexpr int kP = 68, kPx = 20;  // row pitches in floats (16-byte multiples)

struct MlpGradSmem {
  float w1t[kIn][kP];   // [k][u]
  float w2t[kH][kP];    // [k][u]
  float w2[kH][kP];     // [u][k]
  float xt[kIn][kP];    // [k][row]
  float xr[kRows][kPx]; // [row][k]
  float h1t[kH][kP];    // [k][row]
  float h1[kRows][kP];  // [row][k]
  float d2t[kH][kP];    // [u][row]
  float d2[kRows][kP];  // [row][u]: dz2, then dz1
  float red[3][kH];     // db1, db2, dW3 over the block
  float sum[2][kMlpThreads / 32];  // db3 and the loss, by warp
};

__device__ __forceinline__ float4 ld4(const float* p) {
  return *reinterpret_cast<const float4*>(p);
}

// acc[i][j] += a[k][i] * b[k][j] over k < N; a and b point at the thread's
// four columns of row 0.
template <int N>
__device__ __forceinline__ void outer_sum(float (&acc)[4][4], const float* a, const float* b) {
#pragma unroll 8
  for (int k = 0; k < N; ++k) {
    const float4 x = ld4(a + k * kP), y = ld4(b + k * kP);
    const float xa[4] = {x.x, x.y, x.z, x.w}, yb[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xa[i], yb[j], acc[i][j]);
  }
}

// grad[0..4) += v; one 16-byte reduction when the gradient is aligned for it.
__device__ __forceinline__ void add4(float* g, const float (&v)[4], bool vec) {
  if (vec) {
    atomicAdd(reinterpret_cast<float4*>(g), make_float4(v[0], v[1], v[2], v[3]));
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) atomicAdd(g + j, v[j]);
  }
}

// Forward + backward over `rows` examples: grad += d(mean squared error)/d
// params for the batch, loss_sum += sum of squared errors.  Weights are used
// rounded to BF16 (the master copy stays FP32).
__global__ void __launch_bounds__(kMlpThreads)
    k_mlp_grad(const float* __restrict__ params, const float* __restrict__ x,
               const float* __restrict__ t, uint32_t rows, float inv_batch,
               float* __restrict__ grad, float* __restrict__ loss_sum) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  MlpGradSmem& sm = *reinterpret_cast<MlpGradSmem*>(smem_raw);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int c0 = tx * 4, r0 = ty * 4;  // this thread's columns and rows of a product
  for (int i = tid; i < kH * kIn; i += kMlpThreads)
    sm.w1t[i % kIn][i / kIn] = bf16_round(params[kOffW1 + i]);
  for (int i = tid; i < kH * kH; i += kMlpThreads) {
    const float w = bf16_round(params[kOffW2 + i]);
    sm.w2[i / kH][i % kH] = w;
    sm.w2t[i % kH][i / kH] = w;
  }
  if (tid < 3 * kH) sm.red[tid / kH][tid % kH] = 0.0f;
  float w3[4], b1[4], b2[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    w3[j] = bf16_round(params[kOffW3 + c0 + j]);
    b1[j] = params[kOffB1 + c0 + j];
    b2[j] = params[kOffB2 + c0 + j];
  }
  const float b3 = params[kOffB3];

  float gw2[4][4] = {}, gw1[4] = {}, gw3[4] = {}, gb1[4] = {}, gb2[4] = {};
  float gb3 = 0.0f, loss = 0.0f;
  const uint32_t tiles = (rows + kRows - 1) / kRows;
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const uint32_t row0 = tile * kRows;
    const int nr = int(min(uint32_t(kRows), rows - row0));
#pragma unroll
    for (int q = 0; q < kRows * kIn / kMlpThreads; ++q) {
      const int i = q * kMlpThreads + tid, r = i / kIn, k = i % kIn;
      const float v = r < nr ? x[size_t(row0 + r) * kIn + k] : 0.0f;
      sm.xr[r][k] = v;
      sm.xt[k][r] = v;
    }
    float tgt[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) tgt[i] = r0 + i < nr ? t[row0 + r0 + i] : 0.0f;
    __syncthreads();

    // h1 = relu(W1 x + b1): rows r0.., units c0..
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = b1[j];
    outer_sum<kIn>(acc, &sm.xt[0][r0], &sm.w1t[0][c0]);
    uint32_t on = 0;  // bit 4 i + j: z1 > 0
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        on |= uint32_t(acc[i][j] > 0.0f) << (4 * i + j);
        acc[i][j] = fmaxf(acc[i][j], 0.0f);
      }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      *reinterpret_cast<float4*>(&sm.h1[r0 + i][c0]) =
          make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
      *reinterpret_cast<float4*>(&sm.h1t[c0 + i][r0]) =
          make_float4(acc[0][i], acc[1][i], acc[2][i], acc[3][i]);
    }
    __syncthreads();

    // z2 = W2 h1 + b2, y = W3 relu(z2) + b3, dz2 = dy w3 [z2 > 0]
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = b2[j];
    outer_sum<kH>(acc, &sm.h1t[0][r0], &sm.w2t[0][c0]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float y = 0.0f;
#pragma unroll
      for (int j = 0; j < 4; ++j) y = fmaf(w3[j], fmaxf(acc[i][j], 0.0f), y);
#pragma unroll
      for (int d = 1; d < 16; d <<= 1) y += __shfl_xor_sync(0xffffffffu, y, d);
      const float e = r0 + i < nr ? y + b3 - tgt[i] : 0.0f;
      const float dy = 2.0f * e * inv_batch;
      if (tx == 0) {
        loss = fmaf(e, e, loss);
        gb3 += dy;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        gw3[j] = fmaf(dy, fmaxf(acc[i][j], 0.0f), gw3[j]);
        acc[i][j] = acc[i][j] > 0.0f ? dy * w3[j] : 0.0f;
        gb2[j] += acc[i][j];
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      *reinterpret_cast<float4*>(&sm.d2[r0 + i][c0]) =
          make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
      *reinterpret_cast<float4*>(&sm.d2t[c0 + i][r0]) =
          make_float4(acc[0][i], acc[1][i], acc[2][i], acc[3][i]);
    }
    __syncthreads();

    // dW2[u][k] += sum over rows of dz2[u] h1[k]: units r0.., inputs c0..
    outer_sum<kRows>(gw2, &sm.d2[0][r0], &sm.h1[0][c0]);
    // dz1 = (W2^T dz2) [z1 > 0]: rows r0.., units c0..
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    outer_sum<kH>(acc, &sm.d2t[0][r0], &sm.w2[0][c0]);
    __syncthreads();  // every read of dz2 is done before dz1 takes its place
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][j] = (on >> (4 * i + j)) & 1u ? acc[i][j] : 0.0f;
        gb1[j] += acc[i][j];
      }
      *reinterpret_cast<float4*>(&sm.d2[r0 + i][c0]) =
          make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    }
    __syncthreads();
    // dW1[u][k] += sum over rows of dz1[u] x[k]: unit tid / 4, four inputs
    {
      const int u = tid >> 2, k0 = (tid & 3) * 4;
#pragma unroll 8
      for (int r = 0; r < kRows; ++r) {
        const float d = sm.d2[r][u];
        const float4 v = ld4(&sm.xr[r][k0]);
        gw1[0] = fmaf(d, v.x, gw1[0]);
        gw1[1] = fmaf(d, v.y, gw1[1]);
        gw1[2] = fmaf(d, v.z, gw1[2]);
        gw1[3] = fmaf(d, v.w, gw1[3]);
      }
    }
    __syncthreads();  // the next tile writes x
  }

  // the block's sums: the bias and output-layer gradients over its row groups
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    gb1[j] += __shfl_xor_sync(0xffffffffu, gb1[j], 16);
    gb2[j] += __shfl_xor_sync(0xffffffffu, gb2[j], 16);
    gw3[j] += __shfl_xor_sync(0xffffffffu, gw3[j], 16);
    if ((tid & 16) == 0) {
      atomicAdd(&sm.red[0][c0 + j], gb1[j]);
      atomicAdd(&sm.red[1][c0 + j], gb2[j]);
      atomicAdd(&sm.red[2][c0 + j], gw3[j]);
    }
  }
  gb3 += __shfl_xor_sync(0xffffffffu, gb3, 16);
  loss += __shfl_xor_sync(0xffffffffu, loss, 16);
  if ((tid & 31) == 0) {
    sm.sum[0][tid / 32] = gb3;
    sm.sum[1][tid / 32] = loss;
  }
  static_assert(kOffW1 % 4 == 0 && kOffW2 % 4 == 0, "four parameters at a time");
  const bool vec = (reinterpret_cast<uintptr_t>(grad) & 15u) == 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) add4(grad + kOffW2 + (r0 + i) * kH + c0, gw2[i], vec);
  add4(grad + kOffW1 + tid * 4, gw1, vec);
  __syncthreads();
  if (tid < kH) atomicAdd(&grad[kOffB1 + tid], sm.red[0][tid]);
  else if (tid < 2 * kH) atomicAdd(&grad[kOffB2 + tid - kH], sm.red[1][tid - kH]);
  else if (tid < 3 * kH) atomicAdd(&grad[kOffW3 + tid - 2 * kH], sm.red[2][tid - 2 * kH]);
  else if (tid < 3 * kH + 2) {
    // one addition per block: every addition to a large sum rounds it (one per
    // warp left the loss of 8,192 rows over 1e-6 off, now 3.6e-7 at most)
    const float* v = sm.sum[tid - 3 * kH];
    const float all = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
    if (tid == 3 * kH) atomicAdd(&grad[kOffB3], all);
    else if (loss_sum) atomicAdd(loss_sum, all);
  }
}

// Adam on the FP32 master parameters (Kingma & Ba 2015, bias-corrected).
__global__ void k_adam(float* __restrict__ params, const float* __restrict__ grad,
                       float* __restrict__ m, float* __restrict__ v, float lr, float beta1,
                       float beta2, float eps, float bc1, float bc2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kMlpParams) return;
  const float g = grad[i];
  const float mi = beta1 * m[i] + (1.0f - beta1) * g;
  const float vi = beta2 * v[i] + (1.0f - beta2) * g * g;
  m[i] = mi;
  v[i] = vi;
  params[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
}

// Forward only (inference on `rows` feature rows) on the tensor cores, 128
// rows per CTA (mlp.cuh); a row whose tensor-core wait ran out gets NaN.
__global__ void __launch_bounds__(kMlpTcThreads)
    k_mlp_forward(const float* __restrict__ params, const float* __restrict__ x, uint32_t rows,
                  float* __restrict__ y) {
  const uint32_t r0 = blockIdx.x * uint32_t(kMlpTcRows);
  mlp_tile_tc(
      params,
      [&](int t, float (&v)[kMlpIn]) {
        const uint32_t row = r0 + uint32_t(t);
        if (row >= rows) return false;
        const float4* src = reinterpret_cast<const float4*>(x + size_t(row) * kMlpIn);
#pragma unroll
        for (int q = 0; q < kMlpIn / 4; ++q) {
          const float4 f = src[q];
          v[4 * q] = f.x;
          v[4 * q + 1] = f.y;
          v[4 * q + 2] = f.z;
          v[4 * q + 3] = f.w;
        }
        return true;
      },
      [&](int t, float out, bool ok) {
        const uint32_t row = r0 + uint32_t(t);
        if (row < rows) y[row] = ok ? out : __int_as_float(0x7fc00000);
      },
      nullptr);
}

}  // namespace rwt

extern "C" {

int rw_tree_mlp_param_count(void) { return rwt::kMlpParams; }

int rw_tree_mlp_grad(const float* d_params, const float* d_x, const float* d_t, uint32_t rows,
                     uint32_t batch, float* d_grad, float* d_loss_sum, rw_stream_t stream) {
  if (!d_params || !d_x || !d_t || !d_grad || rows < 1 || batch < 1) return RW_ERR_ARG;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const uint32_t tiles = (rows + rwt::kRows - 1) / rwt::kRows;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(rwt::k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             int(sizeof(rwt::MlpGradSmem)));
  if (e != cudaSuccess) return RW_ERR_CUDA;
  const uint32_t blocks = tiles < uint32_t(sms) ? tiles : uint32_t(sms);  // one per SM
  rwt::k_mlp_grad<<<blocks, rwt::kMlpThreads, sizeof(rwt::MlpGradSmem), s>>>(
      d_params, d_x, d_t, rows, 1.0f / float(batch), d_grad, d_loss_sum);
  return cudaGetLastError() == cudaSuccess ? RW_OK : RW_ERR_CUDA;
}

int rw_tree_mlp_adam(float* d_params, const float* d_grad, float* d_m, float* d_v, float lr,
                     float beta1, float beta2, float eps, int32_t step, rw_stream_t stream) {
  if (!d_params || !d_grad || !d_m || !d_v || step < 1) return RW_ERR_ARG;
  const float bc1 = 1.0f - powf(beta1, float(step));
  const float bc2 = 1.0f - powf(beta2, float(step));
  rwt::k_adam<<<(rwt::kMlpParams + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      d_params, d_grad, d_m, d_v, lr, beta1, beta2, eps, bc1, bc2);
  return cudaGetLastError() == cudaSuccess ? RW_OK : RW_ERR_CUDA;
}

int rw_tree_mlp_forward(const float* d_params, const float* d_x, uint32_t rows, float* d_y,
                        rw_stream_t stream) {
  if (!d_params || !d_x || !d_y || rows < 1) return RW_ERR_ARG;
  if (reinterpret_cast<uintptr_t>(d_x) & 15u) return RW_ERR_ARG;  // rows are read as float4
  rwt::k_mlp_forward<<<(rows + rwt::kMlpTcRows - 1) / rwt::kMlpTcRows, rwt::kMlpTcThreads, 0,
                       reinterpret_cast<cudaStream_t>(stream)>>>(d_params, d_x, rows, d_y);
  return cudaGetLastError() == cudaSuccess ? RW_OK : RW_ERR_CUDA;
}

}  // extern "C"
