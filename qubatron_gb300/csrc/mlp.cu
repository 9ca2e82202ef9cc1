// Occluder-proposal network: 48 -> 128 -> 128 -> 128 -> 16 (4 used), GELU,
// BF16 weights and activations on the tensor cores with FP32 accumulation,
// trained on the GPU: the loss and its gradient, and Adam.
//
// gradient_kernel does the whole of a gradient for 128 rows on one SM: four
// forward products, the loss, and the seven products of the backward pass, on
// tcgen05. The accumulators of the three hidden layers stay in tensor memory
// (3 x 128 of its 512 columns) and give the pre-activations again on the way
// back, so no activation goes to memory; a layer's columns then take its
// weight gradient. Operands are in shared memory in the K-major core-matrix
// layout (umma.cuh), a weight matrix's transpose replacing it once its
// forward product is done. Every block adds its tiles' weight gradients into
// a buffer of its own, and reduce_kernel (or adam_kernel) sums those in a
// fixed order: equal inputs give equal bits.
//
// What bounds it: the chain of eleven products and epilogues of one tile
// (GELU and its derivative, transposed writes to shared memory). As separate
// products, with activations in memory and atomic sums, 8192 rows took 18
// launches and 497 us; 107 us in 2 now (64 blocks, the other SMs idle).

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "mlp.h"
#include "mlp_device.cuh"
#include "qbc_internal.h"

using qbc::fail;

namespace qbc {
namespace mlp {

// kernels launched by this thread (the context adds the difference to its
// launch count)
thread_local int64_t g_launches = 0;
int64_t launches() { return g_launches; }

namespace {

using bf16 = __nv_bfloat16;

constexpr int kGradWarps = 16;
constexpr int kGradThreads = 32 * kGradWarps;
constexpr uint32_t kGradTmemCols = 512;  // all of an SM's: one block per SM
// accumulator columns of hidden layer l: 128 l; of what is not kept: 384
constexpr uint32_t kWorkCols = 3 * kHidden;

__device__ __forceinline__ float gelu_grad(float x) {
  const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
  const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
  return cdf + x * pdf;
}

struct GradSmem {
  // operand regions, each a multiple of 1024 bytes from a 1024-aligned base
  bf16 w1[kHidden * kIn];
  bf16 w2[kHidden * kHidden];  // then its transpose
  bf16 w3[kHidden * kHidden];  // then its transpose
  bf16 w4[kOutPad * kHidden];
  bf16 w4t[kHidden * kOutPad];
  bf16 x[kUmmaRows * kIn];
  bf16 xt[kIn * kUmmaRows];
  bf16 h[kUmmaRows * kHidden];   // activations, then pre-activation gradients, by row
  bf16 dzt[kHidden * kUmmaRows];  // pre-activation gradients by unit
  bf16 at[kHidden * kUmmaRows];  // activations by unit
  bf16 d_o[kUmmaRows * kOutPad];
  bf16 dot[kOutPad * kUmmaRows];
  float bias[3 * kHidden + kOutPad];
  float loss[4];
  uint64_t bar;
  uint32_t tmem;
  uint32_t fault;
};
constexpr size_t kGradSmemBytes = sizeof(GradSmem) + 1024;  // + alignment slack
static_assert(kGradSmemBytes <= 232448, "gradient shared memory");

__device__ __forceinline__ bf16& at_core(bf16* base, uint32_t r, uint32_t k, uint32_t K) {
  return *reinterpret_cast<bf16*>(reinterpret_cast<char*>(base) + umma::core_offset(r, k, K));
}

// The transpose of a rows x cols matrix (row-major in memory) as a cols x rows
// operand. Consecutive threads take consecutive rows: their 2-byte stores
// meet four to a bank.
__device__ __forceinline__ void stage_transposed(bf16* dst, const bf16* src, int rows, int cols, int tid) {
  for (int e = tid; e < rows * (cols / 8); e += kGradThreads) {
    const int r = e % rows, c = e / rows * 8;
    const uint4 v = *reinterpret_cast<const uint4*>(src + (size_t)r * cols + c);
    const bf16* p = reinterpret_cast<const bf16*>(&v);
#pragma unroll
    for (int k = 0; k < 8; ++k) at_core(dst, c + k, r, rows) = p[k];
  }
}

// D[128 x N] = A[128 x K] * B[N x K]^T into columns `col`.
__device__ __forceinline__ void issue(uint32_t tmem, uint32_t col, const bf16* a, const bf16* b, int K, int N) {
  issue_layer(tmem + col, a, b, K, N);
}

// What is written before is in shared memory for the tensor core, `products`
// issued by one thread, and done when this returns true (false: a wait gave
// up).
template <class F>
__device__ __forceinline__ bool multiply(GradSmem& S, uint32_t& phase, F products) {
  umma::fence_smem_to_async();
  umma::fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0) {
    umma::fence_after_sync();
    products();
    umma::commit(&S.bar);
  }
  if (!umma::mbar_wait(&S.bar, phase, kUmmaWaitLimit)) atomicOr(&S.fault, 1u);
  umma::fence_after_sync();
  __syncthreads();
  if (S.fault) return false;
  phase ^= 1u;
  return true;
}

// One layer's weight gradient [128 out x N in] from its accumulator into the
// block's buffer (added after its first tile). Warp w: rows 32 (w % 4) .. +
// 31, columns 32 (w / 4) .. + 31.
__device__ __forceinline__ void add_weights(uint32_t tmem, uint32_t col, float* dst, int N, bool first, int warp,
                                            int lane) {
  const int q = warp & 3, c0 = 32 * (warp >> 2);
  if (c0 >= N) return;
  float v[32];
  umma::tmem_ld32(tmem + ((uint32_t)(32 * q) << 16) + col + c0, v);
  umma::tmem_ld_wait();
  float4* p = reinterpret_cast<float4*>(dst + (size_t)(32 * q + lane) * N + c0);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (c0 + 4 * k >= N) break;
    float4 g = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    if (!first) {
      const float4 o = p[k];
      g = make_float4(o.x + g.x, o.y + g.y, o.z + g.z, o.w + g.w);
    }
    p[k] = g;
  }
}

// Bias gradients: sums over the tile's rows of dzt.
__device__ __forceinline__ void add_bias(const bf16* dzt, float* dst, bool first, int tid) {
  if (tid >= kHidden) return;
  float s = 0.0f;
  for (int r = 0; r < kUmmaRows; r += 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(dzt) +
                                                    umma::core_offset(tid, r, kUmmaRows));
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 f = __bfloat1622float2(p[k]);
      s += f.x + f.y;
    }
  }
  dst[tid] = first ? s : dst[tid] + s;
}

// Parameter offsets (floats), at compile time: W1 b1 W2 b2 W3 b3 W4 b4.
__host__ __device__ constexpr int off_w(int l) {
  return l == 0 ? 0 : kHidden * kIn + kHidden + (l - 1) * (kHidden * kHidden + kHidden);
}
__host__ __device__ constexpr int off_b(int l) {
  return off_w(l) + (l == 0 ? kHidden * kIn : (l < 3 ? kHidden * kHidden : kOutPad * kHidden));
}
constexpr int kParams = off_b(3) + kOutPad;
constexpr int kPartial = kParams + 16;  // a block's buffer: gradients, then its loss

// Src: load(row, c, v) the features 8 c .. 8 c + 7 of a row as bf16, and
// label(row, t, kind).
template <class Src>
__global__ void __launch_bounds__(kGradThreads, 1)
    gradient_kernel(const FusedParams p, const Src src, uint32_t rows, float scale, float* partial, unsigned* err) {
  extern __shared__ unsigned char grad_smem_raw[];
  GradSmem& S = *reinterpret_cast<GradSmem*>((reinterpret_cast<uintptr_t>(grad_smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int q = warp & 3, c0 = 32 * (warp >> 2), row = 32 * q + lane;  // this thread's accumulator row, columns
  float* out = partial + (size_t)blockIdx.x * kPartial;

  stage_matrix(S.w1, p.w[0], kHidden, kIn, tid, kGradThreads);
  stage_matrix(S.w4, p.w[3], kOutPad, kHidden, tid, kGradThreads);
  stage_transposed(S.w4t, p.w[3], kOutPad, kHidden, tid);
  for (int e = tid; e < 3 * kHidden + kOutPad; e += kGradThreads)
    S.bias[e] = e < 3 * kHidden ? p.b[e / kHidden][e % kHidden] : p.b[3][e - 3 * kHidden];
  if (tid == 0) {
    S.fault = 0u;
    umma::mbar_init(&S.bar, 1);
  }
  if (warp == 0) {
    umma::tmem_alloc(&S.tmem, kGradTmemCols);
    umma::tmem_relinquish();
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = S.tmem, mine = tmem + ((uint32_t)(32 * q) << 16);
  uint32_t phase = 0;

  // this thread's part of a hidden layer's activations (pre-activations from
  // the layer's accumulator): by row into h, or by unit into at
  auto activate = [&](int l, bool by_row, bool by_unit) {
    float v[32];
    umma::tmem_ld32(mine + 128 * l + c0, v);
    umma::tmem_ld_wait();
    const float* b = S.bias + l * kHidden + c0;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      uint4 o;
      bf16* e = reinterpret_cast<bf16*>(&o);
#pragma unroll
      for (int k = 0; k < 8; ++k) e[k] = __float2bfloat16(gelu_f(v[8 * g + k] + b[8 * g + k]));
      if (by_row)
        *reinterpret_cast<uint4*>(reinterpret_cast<char*>(S.h) + umma::core_offset(row, c0 + 8 * g, kHidden)) = o;
      if (by_unit)
#pragma unroll
        for (int k = 0; k < 8; ++k) at_core(S.at, c0 + 8 * g + k, row, kUmmaRows) = e[k];
    }
  };
  // dZ = dA * GELU'(Z) of layer l from the work columns: by unit into dzt,
  // and by row into h
  auto backward = [&](int l, bool by_row) {
    float d[32], v[32];
    umma::tmem_ld32(mine + kWorkCols + c0, d);
    umma::tmem_ld32(mine + 128 * l + c0, v);
    umma::tmem_ld_wait();
    const float* b = S.bias + l * kHidden + c0;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      uint4 o;
      bf16* e = reinterpret_cast<bf16*>(&o);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        e[k] = __float2bfloat16(d[8 * g + k] * gelu_grad(v[8 * g + k] + b[8 * g + k]));
        at_core(S.dzt, c0 + 8 * g + k, row, kUmmaRows) = e[k];
      }
      if (by_row)
        *reinterpret_cast<uint4*>(reinterpret_cast<char*>(S.h) + umma::core_offset(row, c0 + 8 * g, kHidden)) = o;
    }
  };

  bool first = true, good = true;
  const uint32_t tiles = (rows + kUmmaRows - 1) / kUmmaRows;
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, first = false) {
    const uint32_t r0 = tile * kUmmaRows;
    stage_matrix(S.w2, p.w[1], kHidden, kHidden, tid, kGradThreads);
    stage_matrix(S.w3, p.w[2], kHidden, kHidden, tid, kGradThreads);
    for (int e = tid; e < kUmmaRows * (kIn / 8); e += kGradThreads) {
      const int r = e % kUmmaRows, c = e / kUmmaRows;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (r0 + r < rows) src.load(r0 + r, c, v);
      *reinterpret_cast<uint4*>(reinterpret_cast<char*>(S.x) + umma::core_offset(r, 8 * c, kIn)) = v;
      const bf16* f = reinterpret_cast<const bf16*>(&v);
#pragma unroll
      for (int k = 0; k < 8; ++k) at_core(S.xt, 8 * c + k, r, kUmmaRows) = f[k];
    }
    // ---- forward ----
    if (!(good = multiply(S, phase, [&] { issue(tmem, 0, S.x, S.w1, kIn, kHidden); }))) break;
    activate(0, true, false);
    if (!(good = multiply(S, phase, [&] { issue(tmem, kHidden, S.h, S.w2, kHidden, kHidden); }))) break;
    stage_transposed(S.w2, p.w[1], kHidden, kHidden, tid);
    activate(1, true, false);
    if (!(good = multiply(S, phase, [&] { issue(tmem, 2 * kHidden, S.h, S.w3, kHidden, kHidden); }))) break;
    stage_transposed(S.w3, p.w[2], kHidden, kHidden, tid);
    activate(2, true, true);
    if (!(good = multiply(S, phase, [&] { issue(tmem, kWorkCols, S.h, S.w4, kHidden, kOutPad); }))) break;
    // ---- loss and its gradient: one row a thread of warps 0..3 ----
    // kind 1: the plain shadow walk found an occluder at t: the nearest
    // output is pulled to t (winner takes all) and the others weakly. kind 0:
    // the pixel was lit: every output is pushed past 1.1 (no proposal). Both:
    // weighted cross-entropy of the gate.
    if (warp < 4) {
      float v[32];
      umma::tmem_ld32(mine + kWorkCols, v);
      umma::tmem_ld_wait();
      float g[kOutUsed] = {0.0f, 0.0f, 0.0f, 0.0f}, o[kOutUsed], local = 0.0f;
#pragma unroll
      for (int k = 0; k < kOutUsed; ++k) o[k] = v[k] + S.bias[3 * kHidden + k];
      float t = 0.0f;
      int kind = -1;
      if (r0 + row < rows) src.label(r0 + row, t, kind);
      if (kind == 1) {
        int best = 0;
        float bd = fabsf(o[0] - t);
#pragma unroll
        for (int k = 1; k < 3; ++k)
          if (fabsf(o[k] - t) < bd) {
            bd = fabsf(o[k] - t);
            best = k;
          }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float d = o[k] - t;
          const float w = k == best ? 1.0f : 0.02f;
          local += w * d * d;
          g[k] = 2.0f * w * d;
        }
      } else if (kind == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float d = 1.1f - o[k];
          if (d > 0.0f) {
            local += 0.5f * d * d;
            g[k] = -d;
          }
        }
      }
      if (kind == 0 || kind == 1) {
        const float z = o[kGate], y = kind == 1 ? 1.0f : 0.0f;
        local += kGateWeight * (fmaxf(z, 0.0f) - y * z + log1pf(expf(-fabsf(z))));
        g[kGate] = kGateWeight * (1.0f / (1.0f + expf(-z)) - y);
      }
#pragma unroll
      for (int k = 0; k < kOutPad; ++k) {
        const bf16 d = __float2bfloat16(k < kOutUsed ? g[k] * scale : 0.0f);
        at_core(S.d_o, row, k, kOutPad) = d;
        at_core(S.dot, k, row, kUmmaRows) = d;
      }
      local *= scale;
      for (int off = 16; off > 0; off >>= 1) local += __shfl_down_sync(0xFFFFFFFFu, local, off);
      if (lane == 0) S.loss[warp] = first ? local : S.loss[warp] + local;
    }
    // ---- output layer: dW4^T = A3^T dO, then dA3 = dO W4 ----
    if (!(good = multiply(S, phase, [&] { issue(tmem, kWorkCols, S.at, S.dot, kUmmaRows, kOutPad); }))) break;
    if (warp < 4) {
      float v[32];
      umma::tmem_ld32(mine + kWorkCols, v);
      umma::tmem_ld_wait();
#pragma unroll
      for (int k = 0; k < kOutPad; ++k) {
        float* w = out + off_w(3) + k * kHidden + row;
        *w = first ? v[k] : *w + v[k];
      }
    } else if (tid < 128 + kOutPad) {
      float s = 0.0f;
      for (int r = 0; r < kUmmaRows; ++r) s += __bfloat162float(at_core(S.dot, tid - 128, r, kUmmaRows));
      float* b = out + off_b(3) + (tid - 128);
      *b = first ? s : *b + s;
    }
    if (!(good = multiply(S, phase, [&] { issue(tmem, kWorkCols, S.d_o, S.w4t, kOutPad, kHidden); }))) break;
    // ---- hidden layers: dW = dZ^T A (into the layer's columns), dA = dZ W ----
    backward(2, true);
    activate(1, false, true);
    if (!(good = multiply(S, phase, [&] {
            issue(tmem, 2 * kHidden, S.dzt, S.at, kUmmaRows, kHidden);
            issue(tmem, kWorkCols, S.h, S.w3, kHidden, kHidden);
          })))
      break;
    add_weights(tmem, 2 * kHidden, out + off_w(2), kHidden, first, warp, lane);
    add_bias(S.dzt, out + off_b(2), first, tid);
    __syncthreads();
    backward(1, true);
    activate(0, false, true);
    if (!(good = multiply(S, phase, [&] {
            issue(tmem, kHidden, S.dzt, S.at, kUmmaRows, kHidden);
            issue(tmem, kWorkCols, S.h, S.w2, kHidden, kHidden);
          })))
      break;
    add_weights(tmem, kHidden, out + off_w(1), kHidden, first, warp, lane);
    add_bias(S.dzt, out + off_b(1), first, tid);
    __syncthreads();
    backward(0, false);
    if (!(good = multiply(S, phase, [&] { issue(tmem, 0, S.dzt, S.xt, kUmmaRows, kIn); }))) break;
    add_weights(tmem, 0, out + off_w(0), kIn, first, warp, lane);
    add_bias(S.dzt, out + off_b(0), first, tid);
    umma::fence_before_sync();
    __syncthreads();  // the next tile's operands overwrite this one's
  }
  __syncthreads();
  if (good && tid == 0) out[kParams] = S.loss[0] + S.loss[1] + S.loss[2] + S.loss[3];
  if (!good) {
    if (tid == 0) {
      atomicOr(err, kErrMmaTimeout);
      umma::mbar_wait(&S.bar, phase, kUmmaWaitLimit);  // the products in flight
    }
    __syncthreads();
  }
  umma::fence_after_sync();
  if (warp == 0) umma::tmem_dealloc(tmem, kGradTmemCols);
}

// Sum over the blocks' buffers of parameter (or loss) i, in block order.
__device__ __forceinline__ float sum_partials(const float* __restrict__ partial, int blocks, int64_t i) {
  float s = 0.0f;
#pragma unroll 8
  for (int b = 0; b < blocks; ++b) s += partial[(size_t)b * kPartial + i];
  return s;
}

// The gradient, and the loss.
__global__ void reduce_kernel(const float* __restrict__ partial, int blocks, float* __restrict__ grad,
                              float* __restrict__ loss) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > kParams) return;
  const float s = sum_partials(partial, blocks, i);
  if (i < kParams) grad[i] = s;
  else *loss = s;
}

// ---- elementwise kernels ----

__global__ void to_bf16_kernel(const float* __restrict__ src, bf16* __restrict__ dst, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = __float2bfloat16(src[i]);
}

// One step of Adam on the gradient summed from the blocks' buffers, the bf16
// copy of the parameters, and the loss.
__global__ void adam_kernel(const float* __restrict__ partial, int blocks, float* __restrict__ p,
                            bf16* __restrict__ copy, float* __restrict__ m, float* __restrict__ v,
                            float* __restrict__ loss, float lr, float b1, float b2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > kParams) return;
  const float gi = sum_partials(partial, blocks, i);
  if (i == kParams) {
    *loss = gi;
    return;
  }
  m[i] = b1 * m[i] + (1.0f - b1) * gi;
  v[i] = b2 * v[i] + (1.0f - b2) * gi * gi;
  p[i] -= lr * (m[i] / c1) / (sqrtf(v[i] / c2) + eps);
  copy[i] = __float2bfloat16(p[i]);
}

// Rows of 45 floats, as the caller gave them.
struct FloatRows {
  const float* x;
  const float* t;
  const int8_t* kind;
  __device__ __forceinline__ void load(uint32_t r, int c, uint4& v) const { v = float_features(x, r, c); }
  __device__ __forceinline__ void label(uint32_t r, float& tt, int& k) const {
    tt = t[r];
    k = kind[r];
  }
};

// A seeded random minibatch of the training set (bf16 rows of kIn).
struct PickedRows {
  const bf16* x;
  const float* t;
  const int8_t* kind;
  uint64_t n, seed;
  __device__ __forceinline__ uint64_t pick(uint32_t r) const {
    uint64_t z = seed + 0x9E3779B97F4A7C15ull * ((uint64_t)r + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return z % n;
  }
  __device__ __forceinline__ void load(uint32_t r, int c, uint4& v) const {
    v = reinterpret_cast<const uint4*>(x + pick(r) * kIn)[c];
  }
  __device__ __forceinline__ void label(uint32_t r, float& tt, int& k) const {
    const uint64_t j = pick(r);
    tt = t[j];
    k = kind[j];
  }
};

int grid1(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 4096)); }

}  // namespace

// Parameter offsets (floats) in the master array: W1 b1 W2 b2 W3 b3 W4 b4,
// each W as [out][in].
int64_t param_offset(int layer, bool bias) { return bias ? off_b(layer) : off_w(layer); }

int64_t param_count() { return kParams; }

void Net::release() {
  cudaFree(master);
  cudaFree(wb);
  cudaFree(grad);
  cudaFree(m);
  cudaFree(v);
  cudaFree(partial);
  master = grad = m = v = partial = nullptr;
  wb = nullptr;
  ready = false;
}

int Net::init(uint64_t seed, cudaStream_t s) {
  const int64_t n = param_count();
  if (!master) {
    cudaError_t e = cudaMalloc(&master, n * 4);
    if (e == cudaSuccess) e = cudaMalloc(&wb, n * 2);
    if (e == cudaSuccess) e = cudaMalloc(&grad, n * 4);
    if (e == cudaSuccess) e = cudaMalloc(&m, n * 4);
    if (e == cudaSuccess) e = cudaMalloc(&v, n * 4);
    if (e != cudaSuccess) return fail(QBC_E_NOMEM, "mlp parameters: %s", cudaGetErrorString(e));
  }
  // uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) weights from a seeded splitmix64,
  // zero biases; padding rows / columns zero
  std::vector<float> h(n, 0.0f);
  uint64_t st = seed * 0x9E3779B97F4A7C15ull + 77;
  auto u01 = [&]() {
    uint64_t z = (st += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
  };
  const int ins[4] = {kIn, kHidden, kHidden, kHidden}, outs[4] = {kHidden, kHidden, kHidden, kOutPad};
  const int used_in[4] = {kInUsed, kHidden, kHidden, kHidden}, used_out[4] = {kHidden, kHidden, kHidden, kOutUsed};
  for (int l = 0; l < 4; ++l) {
    const double a = 1.0 / std::sqrt((double)used_in[l]);
    float* W = h.data() + param_offset(l, false);
    for (int o = 0; o < outs[l]; ++o)
      for (int i = 0; i < ins[l]; ++i)
        W[o * ins[l] + i] = (o < used_out[l] && i < used_in[l]) ? (float)((2.0 * u01() - 1.0) * a) : 0.0f;
  }
  // output bias: start with "no proposal" (t past the hit)
  float* b4 = h.data() + param_offset(3, true);
  for (int o = 0; o < kOut; ++o) b4[o] = 1.5f;
  cudaError_t e = cudaMemcpyAsync(master, h.data(), n * 4, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(m, 0, n * 4, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(v, 0, n * 4, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return fail(QBC_E_CUDA, "mlp init: %s", cudaGetErrorString(e));
  step_count = 0;
  ready = true;
  return sync_weights(s);
}

int Net::set(const float* host, cudaStream_t s) {
  if (!master) {
    int rc = init(1, s);
    if (rc) return rc;
  }
  cudaError_t e = cudaMemcpyAsync(master, host, param_count() * 4, cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return fail(QBC_E_CUDA, "mlp set: %s", cudaGetErrorString(e));
  ready = true;
  return sync_weights(s);
}

int Net::get(float* host, cudaStream_t s) const {
  if (!master) return fail(QBC_E_STATE, "mlp: no parameters");
  cudaError_t e = cudaMemcpyAsync(host, master, param_count() * 4, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return fail(QBC_E_CUDA, "mlp get: %s", cudaGetErrorString(e));
  return QBC_OK;
}

int Net::sync_weights(cudaStream_t s) {
  const int64_t n = param_count();
  to_bf16_kernel<<<grid1(n), 256, 0, s>>>(master, wb, n);
  ++g_launches;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(QBC_E_CUDA, "mlp weights: %s", cudaGetErrorString(e));
  return QBC_OK;
}

template <class Src>
int Net::partials(const Src& src, int64_t rows, int* blocks, cudaStream_t s) {
  if (!ready) return fail(QBC_E_STATE, "mlp: not initialised");
  // (the interface's limit; rows and tiles are 32-bit in the kernel)
  constexpr int64_t kMostRows = 65535ll * kUmmaRows;
  if (rows > kMostRows)
    return fail(QBC_E_ARG, "mlp gradient: %lld rows, at most %lld a call", (long long)rows, (long long)kMostRows);
  if (!partial) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess) e = cudaMalloc(&partial, (size_t)sms * kPartial * sizeof(float));
    if (e != cudaSuccess) return fail(QBC_E_NOMEM, "mlp gradient buffers: %s", cudaGetErrorString(e));
  }
  FusedParams p;
  for (int l = 0; l < 4; ++l) {
    p.w[l] = wb + param_offset(l, false);
    p.b[l] = master + param_offset(l, true);
    if (reinterpret_cast<uintptr_t>(p.w[l]) % 16) return fail(QBC_E_STATE, "proposal network: unaligned weights");
  }
  const int smem = (int)kGradSmemBytes;
  auto kern = gradient_kernel<Src>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return fail(QBC_E_CUDA, "mlp gradient attribute: %s", cudaGetErrorString(e));
  // one tile a block while there are SMs, then several
  *blocks = (int)std::min<int64_t>(sms, (rows + kUmmaRows - 1) / kUmmaRows);
  kern<<<*blocks, kGradThreads, smem, s>>>(p, src, (uint32_t)rows, 1.0f / (float)rows, partial, err);
  ++g_launches;
  e = cudaGetLastError();
  if (e != cudaSuccess) return fail(QBC_E_CUDA, "mlp gradient: %s", cudaGetErrorString(e));
  return QBC_OK;
}

int Net::gradient(const float* X, const float* tlab, const int8_t* kind, int64_t rows, float* loss, cudaStream_t s) {
  int blocks = 0;
  int rc = partials(FloatRows{X, tlab, kind}, rows, &blocks, s);
  if (rc) return rc;
  reduce_kernel<<<kParams / 128 + 1, 128, 0, s>>>(partial, blocks, grad, loss);
  ++g_launches;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(QBC_E_CUDA, "mlp gradient: %s", cudaGetErrorString(e));
  return QBC_OK;
}

int Net::train_step(const bf16* X, const float* tlab, const int8_t* kind, int64_t samples, uint64_t seed,
                    int64_t rows, float lr, float* loss, cudaStream_t s) {
  int blocks = 0;
  int rc = partials(PickedRows{X, tlab, kind, (uint64_t)samples, seed}, rows, &blocks, s);
  if (rc) return rc;
  ++step_count;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.0f - std::pow(b1, (float)step_count), c2 = 1.0f - std::pow(b2, (float)step_count);
  adam_kernel<<<kParams / 128 + 1, 128, 0, s>>>(partial, blocks, master, wb, m, v, loss, lr, b1, b2, 1e-8f, c1, c2);
  ++g_launches;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(QBC_E_CUDA, "mlp adam: %s", cudaGetErrorString(e));
  return QBC_OK;
}

}  // namespace mlp
}  // namespace qbc
