// Bandwidth-bound kernels of the Llama / GPT-2 trainers (sm_100a): RMSNorm, LayerNorm, RoPE,
// SwiGLU, bias + GELU, fused softmax cross-entropy, embedding, and a flat fused AdamW.  Every one
// makes a single pass over its operands with 16-byte accesses and keeps row statistics
// in registers / shared memory; the torch-eager equivalents (several kernels and
// temporaries each) are the baseline they replace.  The reference trainer gets these
// ops from torch (benchmarks/train_llama7b_dp_pp_lowbit.py:158-165,248).
//
// C linkage, raw pointers + stream, async, cudaError_t returned as int.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "rope_chunks.cuh"
#include "tc_common.cuh"

namespace ew {

typedef __nv_bfloat16 bf16;

struct alignas(16) Bf8 {
  bf16 v[8];
};

__device__ __forceinline__ void load8(const bf16* p, float (&f)[8]) {
  const Bf8 raw = *reinterpret_cast<const Bf8*>(p);
#pragma unroll
  for (int i = 0; i < 8; ++i) f[i] = __bfloat162float(raw.v[i]);
}
__device__ __forceinline__ void store8(bf16* p, const float (&f)[8]) {
  Bf8 raw;
#pragma unroll
  for (int i = 0; i < 8; ++i) raw.v[i] = __float2bfloat16_rn(f[i]);
  *reinterpret_cast<Bf8*>(p) = raw;
}

// eight bf16 values in a 16-byte register group -> fp32 (a bf16 is the upper half of its fp32)
__device__ __forceinline__ void unpack8(const uint4& r, float (&f)[8]) {
  const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// e^x = 2^(x log2 e), x <= 0, for the terms of a sum that is at least 1: rounding the product and
// ex2.approx.ftz leave a relative error below (2 + 1.2 |x|) 2^-23, and what is flushed (results
// below 2^-126) cannot change such a sum.  Where the exponential itself is a result, __expf keeps it
// (both loops with __expf: 130 us at 4096 x 32000 instead of 122).
__device__ __forceinline__ float exp_term(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.4426950408889634f));
  return y;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// block-wide sum for up to 1024 threads; every thread gets the result
__device__ __forceinline__ float block_sum(float v, float* scratch /*[33]*/) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float t = lane < (blockDim.x + 31) / 32 ? scratch[lane] : 0.0f;
    t = warp_sum(t);
    if (lane == 0) scratch[32] = t;
  }
  __syncthreads();
  return scratch[32];
}
__device__ __forceinline__ float block_max(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float t = lane < (blockDim.x + 31) / 32 ? scratch[lane] : -INFINITY;
    t = warp_max(t);
    if (lane == 0) scratch[32] = t;
  }
  __syncthreads();
  return scratch[32];
}

// ---------------------------------------------------------------------------
// RMSNorm: y = x * rsqrt(mean(x^2) + eps) * w        (H % 8 == 0)
// ---------------------------------------------------------------------------
// A row is read once and stays in registers between the sum of squares and the output; the next
// row of the CTA is requested before the reduction, which costs one barrier (see the backward
// kernel).  Read twice, with three barriers per row, 4096 x 4096 took 15.4 us; now 14.0 us (128 x
// 4096: 3.3 -> 2.3 us).
// Rows of more than 16384 elements: two reads, any H.
__global__ void __launch_bounds__(256)
rmsnorm_fwd_wide_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w,
                        bf16* __restrict__ y, float* __restrict__ rstd_out, int rows, int H,
                        float eps) {
  __shared__ float scratch[33];
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const bf16* xr = x + (size_t)row * H;
    float ss = 0.0f;
    for (int c = threadIdx.x * 8; c < H; c += blockDim.x * 8) {
      float f[8];
      load8(xr + c, f);
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
    }
    ss = block_sum(ss, scratch);
    const float rstd = rsqrtf(ss / (float)H + eps);
    if (threadIdx.x == 0) rstd_out[row] = rstd;
    bf16* yr = y + (size_t)row * H;
    for (int c = threadIdx.x * 8; c < H; c += blockDim.x * 8) {
      float f[8], g[8];
      load8(xr + c, f);
      load8(w + c, g);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = f[i] * rstd * g[i];
      store8(yr + c, f);
    }
  }
}

template <int NV>
__global__ void __launch_bounds__(256)
rmsnorm_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, bf16* __restrict__ y,
                   float* __restrict__ rstd_out, int rows, int H, float eps) {
  __shared__ float partial[2][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  uint4 cur[NV], nxt[NV], wv[NV];
  auto fetch = [&](int row, uint4 (&b)[NV]) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int c = (threadIdx.x + k * blockDim.x) * 8;
      if (c < H) b[k] = *reinterpret_cast<const uint4*>(x + (size_t)row * H + c);
    }
  };
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int c = (threadIdx.x + k * blockDim.x) * 8;
    if (c < H) wv[k] = *reinterpret_cast<const uint4*>(w + c);
  }
  int row = blockIdx.x;
  if (row < rows) fetch(row, cur);
  int parity = 0;
  for (; row < rows; row += gridDim.x, parity ^= 1) {
    if (row + (int)gridDim.x < rows) fetch(row + gridDim.x, nxt);
    float ss = 0.0f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      if ((threadIdx.x + k * blockDim.x) * 8 < H) {
        float f[8];
        unpack8(cur[k], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
      }
    }
    ss = warp_sum(ss);
    if (lane == 0) partial[parity][warp] = ss;
    __syncthreads();  // the other buffer is free again: its readers passed the previous barrier
    float total = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) total += i < nwarps ? partial[parity][i] : 0.0f;
    const float rstd = rsqrtf(total / (float)H + eps);
    if (threadIdx.x == 0) rstd_out[row] = rstd;
    bf16* yr = y + (size_t)row * H;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int c = (threadIdx.x + k * blockDim.x) * 8;
      if (c < H) {
        float f[8], g[8];
        unpack8(cur[k], f);
        unpack8(wv[k], g);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = f[i] * rstd * g[i];
        *reinterpret_cast<uint4*>(yr + c) = pack8(f);
        cur[k] = nxt[k];
      }
    }
  }
}

// dx = rstd * (dy*w - x * rstd^2 * mean(dy*w*x)) [+ dres];  dw += sum_rows dy * x * rstd (fp32)
// Each CTA walks rows blockIdx.x, +gridDim.x, ... and keeps its dw partial in registers
// (thread t owns columns t*8 + k*blockDim*8).  A row is read once: x and dy stay in registers
// (as packed bf16) across the reduction, the next row's loads are issued before the reduction
// of the current one, and the reduction costs one barrier (warp partials in a double-buffered
// scratch, every thread adds them up itself).  At the end a CTA writes its dw partial to its
// row of `partials` ([gridDim.x][H] fp32) and colsum_add_kernel folds the rows into dw: H
// atomic adds per CTA on the same H addresses used to cost a third of the kernel's time.
// `dres` (HAS_RES): the gradient that reaches the same input through the residual connection,
// added to dx here instead of by a separate add kernel.
template <int MAX_ITERS, bool HAS_RES>
__global__ void __launch_bounds__(512)
rmsnorm_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x,
                   const bf16* __restrict__ w, const float* __restrict__ rstd,
                   const bf16* __restrict__ dres, bf16* __restrict__ dx,
                   float* __restrict__ partials, int rows, int H) {
  __shared__ float partial[2][16];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  float acc[MAX_ITERS][8], fw[MAX_ITERS][8];
  Bf8 cx[MAX_ITERS], cg[MAX_ITERS], nx[MAX_ITERS], ng[MAX_ITERS];
#pragma unroll
  for (int k = 0; k < MAX_ITERS; ++k) {
    const int c = (threadIdx.x + k * blockDim.x) * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[k][i] = fw[k][i] = 0.0f;
    if (c < H) load8(w + c, fw[k]);
  }
  auto fetch = [&](int row, Bf8 (&bx)[MAX_ITERS], Bf8 (&bg)[MAX_ITERS]) {
#pragma unroll
    for (int k = 0; k < MAX_ITERS; ++k) {
      const int c = (threadIdx.x + k * blockDim.x) * 8;
      if (c < H) {
        bx[k] = *reinterpret_cast<const Bf8*>(x + (size_t)row * H + c);
        bg[k] = *reinterpret_cast<const Bf8*>(dy + (size_t)row * H + c);
      }
    }
  };
  int row = blockIdx.x;
  if (row < rows) fetch(row, cx, cg);
  int parity = 0;
  for (; row < rows; row += gridDim.x, parity ^= 1) {
    const int next = row + gridDim.x;
    if (next < rows) fetch(next, nx, ng);
    const float rs = rstd[row];
    float dot = 0.0f;
#pragma unroll
    for (int k = 0; k < MAX_ITERS; ++k) {
      const int c = (threadIdx.x + k * blockDim.x) * 8;
      if (c < H) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float fx = __bfloat162float(cx[k].v[i]), fg = __bfloat162float(cg[k].v[i]);
          dot += fg * fw[k][i] * fx;
          acc[k][i] += fg * fx * rs;
        }
      }
    }
    dot = warp_sum(dot);
    if (lane == 0) partial[parity][warp] = dot;
    __syncthreads();  // the other buffer is free again: its readers passed the previous barrier
    float total = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) total += i < nwarps ? partial[parity][i] : 0.0f;
    const float coef = total * rs * rs * rs / (float)H;
    bf16* dr = dx + (size_t)row * H;
#pragma unroll
    for (int k = 0; k < MAX_ITERS; ++k) {
      const int c = (threadIdx.x + k * blockDim.x) * 8;
      if (c < H) {
        float o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float fx = __bfloat162float(cx[k].v[i]), fg = __bfloat162float(cg[k].v[i]);
          o[i] = fg * fw[k][i] * rs - fx * coef;
        }
        if constexpr (HAS_RES) {
          float rr[8];
          load8(dres + (size_t)row * H + c, rr);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] += rr[i];
        }
        store8(dr + c, o);
        cx[k] = nx[k];
        cg[k] = ng[k];
      }
    }
  }
#pragma unroll
  for (int k = 0; k < MAX_ITERS; ++k) {
    const int c = (threadIdx.x + k * blockDim.x) * 8;
    if (c < H) {
      float* dst = partials + (size_t)blockIdx.x * H + c;
      *reinterpret_cast<float4*>(dst) = make_float4(acc[k][0], acc[k][1], acc[k][2], acc[k][3]);
      *reinterpret_cast<float4*>(dst + 4) = make_float4(acc[k][4], acc[k][5], acc[k][6], acc[k][7]);
    }
  }
}

// out[c] += sum over p < nparts of partials[p * width + c] for the `width` columns of a
// partial row; columns [0, split) belong to out_a, columns [split, width) to out_b (at
// out_b[c - split]).  blockDim = (32, 32): a CTA owns 32 columns, its 32 thread rows split
// the partial rows (a few loads each, all in flight at once), shared memory folds them.
__global__ void __launch_bounds__(1024)
colsum_add_kernel(const float* __restrict__ partials, float* __restrict__ out_a,
                  float* __restrict__ out_b, int nparts, int width, int split) {
  __shared__ float fold[32][33];
  const int c = blockIdx.x * 32 + threadIdx.x;
  float s = 0.0f;
  if (c < width) {
    int p = threadIdx.y;
    for (; p + 96 < nparts; p += 128) {
      const float a0 = partials[(size_t)p * width + c];
      const float a1 = partials[(size_t)(p + 32) * width + c];
      const float a2 = partials[(size_t)(p + 64) * width + c];
      const float a3 = partials[(size_t)(p + 96) * width + c];
      s += (a0 + a1) + (a2 + a3);
    }
    for (; p < nparts; p += 32) s += partials[(size_t)p * width + c];
  }
  fold[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && c < width) {
    float t = 0.0f;
#pragma unroll
    for (int i = 0; i < 32; ++i) t += fold[i][threadIdx.x];
    if (c < split) out_a[c] += t;
    else out_b[c - split] += t;
  }
}

// Column sums of a bf16 [rows, C] matrix (bias gradients), first stage: strip blockIdx.y's sums to
// its row of `partials`, folded by colsum_add_kernel.  Four rows in flight per thread.
__global__ void __launch_bounds__(128)
colsum_bf16_kernel(const bf16* __restrict__ x, float* __restrict__ partials, long long rows,
                   int C) {
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (c >= C) return;
  float acc[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] = 0.0f;
  for (long long r0 = blockIdx.y; r0 < rows; r0 += 4LL * gridDim.y) {
    uint4 b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long r = r0 + (long long)j * gridDim.y;
      b[j] = r < rows ? *reinterpret_cast<const uint4*>(x + r * C + c) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float f[8];
      unpack8(b[j], f);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += f[k];
    }
  }
  float* dst = partials + (size_t)blockIdx.y * C + c;
  *reinterpret_cast<float4*>(dst) = make_float4(acc[0], acc[1], acc[2], acc[3]);
  *reinterpret_cast<float4*>(dst + 4) = make_float4(acc[4], acc[5], acc[6], acc[7]);
}

// ---------------------------------------------------------------------------
// LayerNorm (GPT-2): y = (x - mean) * rstd * w + b.  One warp per row, the row held in
// registers between the statistics and the output (one read of x).  H <= 32 * 8 * MAX_ITERS
// (the launchers instantiate 2 and 4: H up to 1024).
// ---------------------------------------------------------------------------
template <int MAX_ITERS>
__global__ void __launch_bounds__(256)
layernorm_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w,
                     const bf16* __restrict__ b, bf16* __restrict__ y,
                     float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows, int H,
                     float eps) {
  const int lane = threadIdx.x & 31;
  const int warps_per_cta = blockDim.x >> 5;
  for (int row = blockIdx.x * warps_per_cta + (threadIdx.x >> 5); row < rows;
       row += gridDim.x * warps_per_cta) {
    const bf16* xr = x + (size_t)row * H;
    float f[MAX_ITERS][8];
    float sum = 0.0f;
#pragma unroll
    for (int k = 0; k < MAX_ITERS; ++k) {
      const int c = (lane + k * 32) * 8;
      if (c < H) {
        load8(xr + c, f[k]);
#pragma unroll
        for (int i = 0; i < 8; ++i) sum += f[k][i];
      }
    }
    const float mean = warp_sum(sum) / (float)H;
    float var = 0.0f;
#pragma unroll
    for (int k = 0; k < MAX_ITERS; ++k) {
      const int c = (lane + k * 32) * 8;
      if (c < H) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float d = f[k][i] - mean;
          var += d * d;
        }
      }
    }
    const float rstd = rsqrtf(warp_sum(var) / (float)H + eps);
    if (lane == 0) {
      mean_out[row] = mean;
      rstd_out[row] = rstd;
    }
    bf16* yr = y + (size_t)row * H;
#pragma unroll
    for (int k = 0; k < MAX_ITERS; ++k) {
      const int c = (lane + k * 32) * 8;
      if (c < H) {
        float g[8], bb[8], o[8];
        load8(w + c, g);
        load8(b + c, bb);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = (f[k][i] - mean) * rstd * g[i] + bb[i];
        store8(yr + c, o);
      }
    }
  }
}

// LayerNorm backward, two rows per CTA pass (H <= 1024: at most 128 threads, thread t owns
// columns [8t, 8t + 8)).  Same shape as rmsnorm_bwd_kernel: the next rows' x and dy are
// requested before the current rows' reduction, the four row sums cost one barrier (warp
// partials in a double-buffered scratch), dw / db partials stay in registers and leave as one
// [dw | db] row of `partials` per CTA.  What bounds it is the latency chain of a pass (loads,
// shuffles, barrier): two independent rows share it (8192 x 1024: 21.8 -> 18.3 us).
__global__ void __launch_bounds__(128)
layernorm_bwd_row_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x,
                         const bf16* __restrict__ w, const float* __restrict__ mean,
                         const float* __restrict__ rstd, bf16* __restrict__ dx,
                         float* __restrict__ partials, int rows, int H) {
  __shared__ float4 partial[2][4];  // warp sums {s1, s2} of both rows
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  const int c = threadIdx.x * 8;
  const bool live = c < H;
  float aw[8], ab[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) aw[i] = ab[i] = 0.0f;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  const uint4 wv = live ? *reinterpret_cast<const uint4*>(w + c) : zero;
  struct Row {
    uint4 x, g;
    float mu, rs;
  };
  auto fetch = [&](int row, Row& r) {
    r.x = r.g = zero;
    r.mu = r.rs = 0.0f;  // a row past the end contributes nothing
    if (row < rows) {
      r.mu = mean[row];
      r.rs = rstd[row];
      if (live) {
        r.x = *reinterpret_cast<const uint4*>(x + (size_t)row * H + c);
        r.g = *reinterpret_cast<const uint4*>(dy + (size_t)row * H + c);
      }
    }
  };
  const int stride = gridDim.x;
  Row cur[2], nxt[2];
  int row = blockIdx.x;
  fetch(row, cur[0]);
  fetch(row + stride, cur[1]);
  int parity = 0;
  const float inv_h = 1.0f / (float)H;
  for (; row < rows; row += 2 * stride, parity ^= 1) {
    fetch(row + 2 * stride, nxt[0]);
    fetch(row + 3 * stride, nxt[1]);
    float fw[8];
    unpack8(wv, fw);
    float s[2][2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      s[q][0] = s[q][1] = 0.0f;
      float fx[8], fg[8];
      unpack8(cur[q].x, fx);
      unpack8(cur[q].g, fg);
      if (live) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float xh = (fx[i] - cur[q].mu) * cur[q].rs;
          const float g = fg[i] * fw[i];
          s[q][0] += g;
          s[q][1] += g * xh;
          aw[i] += fg[i] * xh;
          ab[i] += fg[i];
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        s[q][0] += __shfl_xor_sync(0xffffffffu, s[q][0], o);
        s[q][1] += __shfl_xor_sync(0xffffffffu, s[q][1], o);
      }
    }
    if (lane == 0) partial[parity][warp] = make_float4(s[0][0], s[0][1], s[1][0], s[1][1]);
    __syncthreads();  // the other buffer is free again: its readers passed the previous barrier
    float t[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i < nwarps) {
        const float4 v = partial[parity][i];
        t[0][0] += v.x; t[0][1] += v.y; t[1][0] += v.z; t[1][1] += v.w;
      }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int r = row + q * stride;
      if (live && r < rows) {
        const float t1 = t[q][0] * inv_h, t2 = t[q][1] * inv_h;
        float fx[8], fg[8], o[8];
        unpack8(cur[q].x, fx);
        unpack8(cur[q].g, fg);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float xh = (fx[i] - cur[q].mu) * cur[q].rs;
          o[i] = cur[q].rs * (fg[i] * fw[i] - t1 - xh * t2);
        }
        *reinterpret_cast<uint4*>(dx + (size_t)r * H + c) = pack8(o);
      }
      cur[q] = nxt[q];
    }
  }
  if (live) {
    float* dst = partials + (size_t)blockIdx.x * 2 * H + c;
    *reinterpret_cast<float4*>(dst) = make_float4(aw[0], aw[1], aw[2], aw[3]);
    *reinterpret_cast<float4*>(dst + 4) = make_float4(aw[4], aw[5], aw[6], aw[7]);
    *reinterpret_cast<float4*>(dst + H) = make_float4(ab[0], ab[1], ab[2], ab[3]);
    *reinterpret_cast<float4*>(dst + H + 4) = make_float4(ab[4], ab[5], ab[6], ab[7]);
  }
}

// ---------------------------------------------------------------------------
// bias + GELU (tanh form) on a [rows, C] GEMM output: y = gelu(x + bias).
// Backward recomputes from x and bias: dx = dy * gelu'(x + bias), dbias += colsum(dx).
// ---------------------------------------------------------------------------
__device__ __forceinline__ float tanh_fast(float v) {
  float r;
  asm("tanh.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
constexpr float kGeluK = 0.7978845608028654f;  // sqrt(2 / pi)
constexpr float kGeluC = 0.044715f;

// Thread t of a column tile owns 8 columns (its bias stays in registers) and walks its strip's
// rows, two in flight; a thread per group with a 64-bit division each and one load in flight took
// 28 us at 8192 x 4096, 23 us now.
__global__ void __launch_bounds__(128)
bias_gelu_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ bias,
                     bf16* __restrict__ y, long long rows, int C) {
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (c >= C) return;
  float bb[8];
  load8(bias + c, bb);
  auto gelu8 = [&](const uint4& raw, bf16* dst) {
    float u[8];
    unpack8(raw, u);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float v = u[k] + bb[k];
      u[k] = 0.5f * v * (1.0f + tanh_fast(kGeluK * (v + kGeluC * v * v * v)));
    }
    *reinterpret_cast<uint4*>(dst) = pack8(u);
  };
  for (long long r = blockIdx.y; r < rows; r += 2LL * gridDim.y) {
    const long long r1 = r + gridDim.y;
    const bool two = r1 < rows;
    const uint4 a = *reinterpret_cast<const uint4*>(x + r * C + c);
    const uint4 b = *reinterpret_cast<const uint4*>(x + (two ? r1 : r) * C + c);
    gelu8(a, y + r * C + c);
    if (two) gelu8(b, y + r1 * C + c);
  }
}

// grid: (C / (8 * blockDim.x) column tiles, row strips).  Thread t of a column tile owns 8
// columns and walks its strip's rows, so the bias gradient needs 8 atomics per thread.
__global__ void __launch_bounds__(256)
bias_gelu_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x,
                     const bf16* __restrict__ bias, bf16* __restrict__ dx,
                     float* __restrict__ dbias, long long rows, int C) {
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (c >= C) return;
  float bb[8], acc[8];
  load8(bias + c, bb);
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] = 0.0f;
  // four rows of loads in flight per thread (one row at a time left the kernel at a third of
  // the copy rate)
  for (long long r0 = blockIdx.y; r0 < rows; r0 += 4LL * gridDim.y) {
    Bf8 bu[4], bd[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long r = r0 + (long long)j * gridDim.y;
      if (r < rows) {
        bu[j] = *reinterpret_cast<const Bf8*>(x + r * C + c);
        bd[j] = *reinterpret_cast<const Bf8*>(dy + r * C + c);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long r = r0 + (long long)j * gridDim.y;
      if (r >= rows) continue;
      float d[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float v = __bfloat162float(bu[j].v[k]) + bb[k];
        const float t = tanh_fast(kGeluK * (v + kGeluC * v * v * v));
        const float dg = 0.5f * (1.0f + t) +
                         0.5f * v * (1.0f - t * t) * kGeluK * (1.0f + 3.0f * kGeluC * v * v);
        d[k] = __bfloat162float(bd[j].v[k]) * dg;
        acc[k] += d[k];
      }
      store8(dx + r * C + c, d);
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) atomicAdd(dbias + c + k, acc[k]);
}

// ---------------------------------------------------------------------------
// RoPE (rotate-half convention), in place on a [tokens, heads, head_dim] slice of a
// wider row: element (t, h, d) sits at x[t * row_stride + h * head_dim + d].
// cos/sin: [seq, head_dim/2] fp32; position of token t is t % seq.
// sign = +1 forward, -1 backward (the transposed rotation).
// ---------------------------------------------------------------------------
// A thread owns one 8 + 8 element pair of a head and walks the tokens (no division per element),
// two tokens in flight.  OUT_OF_PLACE: rows are read from `src` and the columns behind the heads
// ([heads * head_dim, width)) are copied, which replaces a clone of the whole gradient followed
// by an in-place rotation (B2 S2048 H32 D128: 36 + 2 x 13 us -> 38 us; the forward rotation of
// q and k in one launch instead of two: 2 x 13 -> 23 us).
template <bool OUT_OF_PLACE>
__global__ void __launch_bounds__(256)
rope_kernel(const bf16* src, bf16* dst, const float* __restrict__ cos_t,
            const float* __restrict__ sin_t, int tokens, int heads, int head_dim,
            long long row_stride, int width, int seq, int pos0, float sign, bool tables_aligned) {
  const int half = head_dim / 2;
  const int vec_per_head = half / 8;
  const int rotated = heads * vec_per_head;
  const int items = rotated + (OUT_OF_PLACE ? (width - heads * head_dim) / 8 : 0);
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= items) return;
  if (OUT_OF_PLACE && j >= rotated) {
    const long long col = (long long)heads * head_dim + (long long)(j - rotated) * 8;
    for (int t = blockIdx.y; t < tokens; t += 2 * gridDim.y) {
      const int t1 = t + gridDim.y;
      const uint4 a = *reinterpret_cast<const uint4*>(src + t * row_stride + col);
      if (t1 < tokens) {
        const uint4 b = *reinterpret_cast<const uint4*>(src + t1 * row_stride + col);
        *reinterpret_cast<uint4*>(dst + t1 * row_stride + col) = b;
      }
      *reinterpret_cast<uint4*>(dst + t * row_stride + col) = a;
    }
    return;
  }
  const int h = j / vec_per_head, v = j - h * vec_per_head;
  const long long col = (long long)h * head_dim + v * 8;
  auto rotate = [&](int t, const uint4& qa, const uint4& qb) {
    const uint32_t pos = ((uint32_t)t + (uint32_t)pos0) % (uint32_t)seq;
    const float* c = cos_t + (size_t)pos * half + v * 8;
    const float* s = sin_t + (size_t)pos * half + v * 8;
    float cs[8], sn[8];
    if (tables_aligned) {
#pragma unroll
      for (int k = 0; k < 8; k += 4) {
        const float4 c4 = *reinterpret_cast<const float4*>(c + k);
        const float4 s4 = *reinterpret_cast<const float4*>(s + k);
        cs[k] = c4.x; cs[k + 1] = c4.y; cs[k + 2] = c4.z; cs[k + 3] = c4.w;
        sn[k] = s4.x; sn[k + 1] = s4.y; sn[k + 2] = s4.z; sn[k + 3] = s4.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) { cs[k] = c[k]; sn[k] = s[k]; }
    }
    float a[8], b[8], ra[8], rb[8];
    unpack8(qa, a);
    unpack8(qb, b);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float sk = sn[k] * sign;
      ra[k] = a[k] * cs[k] - b[k] * sk;
      rb[k] = b[k] * cs[k] + a[k] * sk;
    }
    *reinterpret_cast<uint4*>(dst + t * row_stride + col) = pack8(ra);
    *reinterpret_cast<uint4*>(dst + t * row_stride + col + half) = pack8(rb);
  };
  for (int t = blockIdx.y; t < tokens; t += 2 * gridDim.y) {
    const int t1 = t + gridDim.y;
    const bool two = t1 < tokens;
    const bf16* p0 = src + t * row_stride + col;
    const bf16* p1 = src + (two ? t1 : t) * row_stride + col;
    const uint4 a0 = *reinterpret_cast<const uint4*>(p0);
    const uint4 b0 = *reinterpret_cast<const uint4*>(p0 + half);
    const uint4 a1 = *reinterpret_cast<const uint4*>(p1);
    const uint4 b1 = *reinterpret_cast<const uint4*>(p1 + half);
    rotate(t, a0, b0);
    if (two) rotate(t1, a1, b1);
  }
}

// ---------------------------------------------------------------------------
// SwiGLU on a fused [tokens, 2F] projection (gate | up): h = silu(gate) * up
// ---------------------------------------------------------------------------
// Two independent 8-element groups per thread and iteration: all loads of both are issued
// before the first result is needed (one group per iteration left the kernels at half the copy
// rate: too few bytes in flight per thread for five streams).
// silu(g) = g / (1 + e^-g) with the IEEE division, as in the backward kernel.  The forward kernel
// waits for it (4096 x 11008: 63 us against 51 with __fdividef), but __fdividef returns 0 for
// a denominator above 2^126, which gates below -87 reach, and is 2 ulp off elsewhere.
__device__ __forceinline__ float silu(float g) { return g / (1.0f + __expf(-g)); }

__global__ void __launch_bounds__(256)
swiglu_fwd_kernel(const bf16* __restrict__ gu, bf16* __restrict__ h, long long tokens, int F) {
  const int vec = F / 8;
  const long long total = tokens * vec;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; i0 < total;
       i0 += 2 * stride) {
    const long long i1 = i0 + stride;
    const bool two = i1 < total;
    const long long t0 = i0 / vec, t1 = two ? i1 / vec : t0;
    const int c0 = (int)(i0 - t0 * vec) * 8, c1 = two ? (int)(i1 - t1 * vec) * 8 : c0;
    Bf8 g0 = *reinterpret_cast<const Bf8*>(gu + t0 * 2 * F + c0);
    Bf8 u0 = *reinterpret_cast<const Bf8*>(gu + t0 * 2 * F + F + c0);
    Bf8 g1 = *reinterpret_cast<const Bf8*>(gu + t1 * 2 * F + c1);
    Bf8 u1 = *reinterpret_cast<const Bf8*>(gu + t1 * 2 * F + F + c1);
    float o[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float g = __bfloat162float(g0.v[k]);
      o[k] = silu(g) * __bfloat162float(u0.v[k]);
    }
    store8(h + t0 * F + c0, o);
    if (two) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float g = __bfloat162float(g1.v[k]);
        o[k] = silu(g) * __bfloat162float(u1.v[k]);
      }
      store8(h + t1 * F + c1, o);
    }
  }
}

__device__ __forceinline__ void swiglu_bwd8(const Bf8& g, const Bf8& u, const Bf8& d,
                                            float (&dg)[8], float (&du)[8]) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float gk = __bfloat162float(g.v[k]), uk = __bfloat162float(u.v[k]);
    const float dk = __bfloat162float(d.v[k]);
    const float sg = 1.0f / (1.0f + __expf(-gk));
    const float silu = gk * sg;
    dg[k] = dk * uk * (sg + silu * (1.0f - sg));
    du[k] = dk * silu;
  }
}

__global__ void __launch_bounds__(256)
swiglu_bwd_kernel(const bf16* __restrict__ gu, const bf16* __restrict__ dh,
                  bf16* __restrict__ dgu, long long tokens, int F) {
  const int vec = F / 8;
  const long long total = tokens * vec;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; i0 < total;
       i0 += 2 * stride) {
    const long long i1 = i0 + stride;
    const bool two = i1 < total;
    const long long t0 = i0 / vec, t1 = two ? i1 / vec : t0;
    const int c0 = (int)(i0 - t0 * vec) * 8, c1 = two ? (int)(i1 - t1 * vec) * 8 : c0;
    const Bf8 g0 = *reinterpret_cast<const Bf8*>(gu + t0 * 2 * F + c0);
    const Bf8 u0 = *reinterpret_cast<const Bf8*>(gu + t0 * 2 * F + F + c0);
    const Bf8 d0 = *reinterpret_cast<const Bf8*>(dh + t0 * F + c0);
    const Bf8 g1 = *reinterpret_cast<const Bf8*>(gu + t1 * 2 * F + c1);
    const Bf8 u1 = *reinterpret_cast<const Bf8*>(gu + t1 * 2 * F + F + c1);
    const Bf8 d1 = *reinterpret_cast<const Bf8*>(dh + t1 * F + c1);
    float dg[8], du[8];
    swiglu_bwd8(g0, u0, d0, dg, du);
    store8(dgu + t0 * 2 * F + c0, dg);
    store8(dgu + t0 * 2 * F + F + c0, du);
    if (two) {
      swiglu_bwd8(g1, u1, d1, dg, du);
      store8(dgu + t1 * 2 * F + c1, dg);
      store8(dgu + t1 * 2 * F + F + c1, du);
    }
  }
}

// ---------------------------------------------------------------------------
// Fused softmax cross-entropy over rows of logits [rows, V] (V % 8 == 0).
// loss_out[row] = logsumexp - logit[target] (0 for ignored rows); the logits are
// overwritten in place by dlogits = (softmax - onehot) * grad_scale[0].
//
// Any V: one CTA per row, three passes over it (maximum, sum, gradient).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(512)
cross_entropy_kernel(bf16* __restrict__ logits, const long long* __restrict__ targets,
                     float* __restrict__ loss_out, const float* __restrict__ grad_scale,
                     int rows, int V, long long ignore_index) {
  __shared__ float scratch[33];
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    bf16* lr = logits + (size_t)row * V;
    const long long tgt = targets[row];
    float m = -INFINITY;
    for (int c = threadIdx.x * 8; c < V; c += blockDim.x * 8) {
      float f[8];
      load8(lr + c, f);
#pragma unroll
      for (int i = 0; i < 8; ++i) m = fmaxf(m, f[i]);
    }
    m = block_max(m, scratch);
    float s = 0.0f;
    for (int c = threadIdx.x * 8; c < V; c += blockDim.x * 8) {
      float f[8];
      load8(lr + c, f);
#pragma unroll
      for (int i = 0; i < 8; ++i) s += __expf(f[i] - m);
    }
    s = block_sum(s, scratch);
    const bool ignored = tgt == ignore_index || tgt < 0 || tgt >= V;
    const float lse = m + logf(s);
    if (threadIdx.x == 0)
      loss_out[row] = ignored ? 0.0f : lse - __bfloat162float(lr[tgt]);
    __syncthreads();  // the target logit is read before anybody overwrites it
    const float scale = ignored ? 0.0f : grad_scale[0];
    const float inv = 1.0f / s;
    for (int c = threadIdx.x * 8; c < V; c += blockDim.x * 8) {
      float f[8];
      load8(lr + c, f);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float p = __expf(f[i] - m) * inv;
        if (c + i == tgt) p -= 1.0f;
        f[i] = p * scale;
      }
      store8(lr + c, f);
    }
  }
}

// Vocabulary-sized rows.  The loop above reads a row three times from global memory and its CTAs
// drain the memory pipe at every reduction (4096 x 32000: 159 us, 8192 x 50432: 489 us, 0.50 of
// the copy rate).  Here a row is copied into shared memory once by a bulk copy, and two or
// three persistent CTAs per SM work on rows of their own, so that one waits for its copy or for
// its reduction while the others compute: with the special-function unit busy for half of the
// time that the row's bytes take, one row at a time per SM (with the next one prefetched) came
// to 111 / 356 us.  Measured: 113 / 346 us (4.7 / 4.8 TB/s, 0.71 / 0.73 of copy).
constexpr int kCeThreads = 512;
constexpr unsigned long long kCeBudgetNs = 2000000000ull;

__device__ unsigned int g_ce_status;      // 1: a row's copy did not arrive within the budget

struct alignas(128) CeShared {
  float2 part[2][kCeThreads / 32];
  uint64_t full;
  volatile int expired;  // 1 + the number of the CTA's row whose copy did not arrive
};

// (maximum, sum of e^(x - maximum)) of two sets; an empty or fully masked one is (-inf, 0)
__device__ __forceinline__ void ce_merge(float& m, float& s, float m2, float s2) {
  const float top = fmaxf(m, m2);
  s = (m == top ? s : s * __expf(m - top)) + (m2 == top ? s2 : s2 * __expf(m2 - top));
  m = top;
}

template <int CTAS>
__global__ void __launch_bounds__(kCeThreads, CTAS)
cross_entropy_rows_kernel(bf16* __restrict__ logits, const long long* __restrict__ targets,
                          float* __restrict__ loss_out, const float* __restrict__ grad_scale,
                          int rows, int V, long long ignore_index) {
  extern __shared__ __align__(128) uint8_t ce_smem[];
  CeShared* sh = reinterpret_cast<CeShared*>(ce_smem);
  const bf16* br = reinterpret_cast<const bf16*>(ce_smem + sizeof(CeShared));
  const int tid = threadIdx.x;
  const uint32_t row_bytes = (uint32_t)V * 2u;
  auto load = [&](long long row) {
    tc::mbar_expect_tx(&sh->full, row_bytes);
    tc::bulk_load(ce_smem + sizeof(CeShared), logits + (size_t)row * V, row_bytes, &sh->full);
  };
  if (tid == 0) {
    tc::mbar_init(&sh->full, 1);
    sh->expired = 0;
    tc::fence_mbar_init();
    if (blockIdx.x < rows) load(blockIdx.x);
  }
  __syncthreads();

  const int vec = V / 8;
  const float gscale = grad_scale[0];
  int it = 0;
  long long tgt = blockIdx.x < rows ? targets[blockIdx.x] : 0;
  for (long long row = blockIdx.x; row < rows; row += gridDim.x, ++it) {
    // the next row's target is requested a row ahead: its latency would stall every row
    const long long next_tgt = row + gridDim.x < rows ? targets[row + gridDim.x] : 0;
    const bool ignored = tgt == ignore_index || tgt < 0 || tgt >= V;
    if (!tc::mbar_wait(&sh->full, (uint32_t)it & 1u, kCeBudgetNs)) {
      // finish the row with what is there: a thread that left would leave the others in a barrier
      atomicCAS(&g_ce_status, 0u, 1u);
      sh->expired = it + 1;
    }
    float m = -INFINITY;
#pragma unroll 4
    for (int c = tid; c < vec; c += kCeThreads) {
      float f[8];
      unpack8(*reinterpret_cast<const uint4*>(br + c * 8), f);
#pragma unroll
      for (int i = 0; i < 8; ++i) m = fmaxf(m, f[i]);
    }
    // Sum relative to the warp's own maximum, so that maximum and sum need one barrier.  A warp
    // whose values are all -inf uses 0 instead: its sum is then 0, not NaN.
    m = warp_max(m);
    const float ref = m == -INFINITY ? 0.0f : m;
    float s4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
    for (int c = tid; c < vec; c += kCeThreads) {
      float f[8];
      unpack8(*reinterpret_cast<const uint4*>(br + c * 8), f);
#pragma unroll
      for (int i = 0; i < 8; ++i) s4[i & 3] += exp_term(f[i] - ref);
    }
    float s = warp_sum((s4[0] + s4[1]) + (s4[2] + s4[3]));
    if ((tid & 31) == 0) sh->part[it & 1][tid >> 5] = make_float2(m, s);
    __syncthreads();
    {
      const float2 p = sh->part[it & 1][tid & (kCeThreads / 32 - 1)];
      m = p.x;
      s = p.y;
#pragma unroll
      for (int o = kCeThreads / 64; o > 0; o >>= 1)
        ce_merge(m, s, __shfl_xor_sync(0xffffffffu, m, o), __shfl_xor_sync(0xffffffffu, s, o));
    }
    const float scale = ignored ? 0.0f : gscale;
    const float factor = 1.0f / s * scale;
    bf16* gr = logits + (size_t)row * V;
#pragma unroll 4
    for (int c = tid; c < vec; c += kCeThreads) {
      float f[8];
      unpack8(*reinterpret_cast<const uint4*>(br + c * 8), f);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = __expf(f[i] - m) * factor;
      *reinterpret_cast<uint4*>(gr + c * 8) = pack8(f);
    }
    // The target's own element is written once more by the thread that owns its group: a test
    // in the loop would make the compiler index the group through local memory.
    if (!ignored && tid == (int)((tgt >> 3) % kCeThreads)) {
      const float logit = __bfloat162float(br[tgt]);
      gr[tgt] = __float2bfloat16_rn((__expf(logit - m) / s - 1.0f) * scale);
      loss_out[row] = m + logf(s) - logit;
    } else if (ignored && tid == 0) {
      loss_out[row] = 0.0f;
    }
    tgt = next_tgt;
    __syncthreads();  // everybody has read the row
    if (sh->expired == it + 1) {  // no further copy; the one under way gets another chance to land
      if (tid == 0) (void)tc::mbar_wait(&sh->full, (uint32_t)it & 1u, kCeBudgetNs);
      break;
    }
    if (tid == 0 && row + gridDim.x < rows) load(row + gridDim.x);
  }
}

// valid = number of targets != ignore_index (at least 1), scale = loss_scale / valid
__global__ void __launch_bounds__(1024)
cross_entropy_scale_kernel(const long long* __restrict__ targets, long long rows,
                           long long ignore_index, float loss_scale, float* __restrict__ valid,
                           float* __restrict__ scale) {
  __shared__ int part[32];
  int n = 0;
  for (long long i = threadIdx.x; i < rows; i += 1024) n += targets[i] != ignore_index;
  n = __reduce_add_sync(0xffffffffu, n);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = n;
  __syncthreads();
  if (threadIdx.x < 32) {
    n = __reduce_add_sync(0xffffffffu, part[threadIdx.x]);
    if (threadIdx.x == 0) {
      const float v = (float)(n > 0 ? n : 1);
      *valid = v;
      *scale = loss_scale / v;
    }
  }
}

// loss = sum(per_row) * scale, one CTA, fixed order
__global__ void __launch_bounds__(1024)
cross_entropy_sum_kernel(const float* __restrict__ per_row, long long rows,
                         const float* __restrict__ scale, float* __restrict__ loss) {
  __shared__ float scratch[33];
  float v = 0.0f;
  for (long long i = threadIdx.x; i < rows; i += 1024) v += per_row[i];
  v = block_sum(v, scratch);
  if (threadIdx.x == 0) *loss = v * *scale;
}

// x *= bf16(s[0]) over n bf16 elements (n % 8 == 0).  The gradient that reaches a loss is almost
// always 1: the factor is looked at on the device and the pass over x is then left away
// (x * 1 == x for every bf16 value).  As a torch multiply by a 0-dim tensor it took 280 us at
// 4096 x 32000 and 880 us at 8192 x 50432, longer than the cross-entropy itself; now 2 us when
// the factor is 1.
__global__ void __launch_bounds__(256)
scale_inplace_kernel(bf16* __restrict__ x, long long vecs, const float* __restrict__ s) {
  const float f = __bfloat162float(__float2bfloat16_rn(s[0]));
  if (f == 1.0f) return;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < vecs;
       i += (long long)gridDim.x * blockDim.x) {
    float v[8];
    load8(x + i * 8, v);
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] *= f;
    store8(x + i * 8, v);
  }
}

// ---------------------------------------------------------------------------
// Embedding lookup and its gradient (fp32 accumulation with atomics)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
embedding_fwd_kernel(const long long* __restrict__ ids, const bf16* __restrict__ table,
                     bf16* __restrict__ out, long long tokens, int H, int vocab) {
  const int vec = H / 8;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < tokens * vec;
       i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / vec;
    const int c = (int)(i - t * vec) * 8;
    long long id = ids[t];
    if (id < 0 || id >= vocab) id = 0;
    *reinterpret_cast<Bf8*>(out + t * H + c) =
        *reinterpret_cast<const Bf8*>(table + id * H + c);
  }
}

__global__ void __launch_bounds__(256)
embedding_bwd_kernel(const long long* __restrict__ ids, const bf16* __restrict__ dout,
                     float* __restrict__ dtable, long long tokens, int H, int vocab,
                     bool aligned) {
  const int vec = H / 8;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < tokens * vec;
       i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / vec;
    const int c = (int)(i - t * vec) * 8;
    const long long id = ids[t];
    if (id < 0 || id >= vocab) continue;
    float f[8];
    load8(dout + t * H + c, f);
    float* dst = dtable + id * H + c;
    if (aligned) {  // two 16-byte atomics instead of eight of 4 (8192 x 1024: 54 -> 17 us)
      atomicAdd(reinterpret_cast<float4*>(dst), make_float4(f[0], f[1], f[2], f[3]));
      atomicAdd(reinterpret_cast<float4*>(dst + 4), make_float4(f[4], f[5], f[6], f[7]));
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) atomicAdd(dst + k, f[k]);
    }
  }
}

// ---------------------------------------------------------------------------
// Flat fused AdamW over fp32 master weights; also refreshes the bf16 working copy and
// (optionally) zeroes the gradient for the next step.  n % 4 == 0 buffers, 16-B aligned.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
adamw_kernel(float* __restrict__ master, bf16* __restrict__ param_bf16, float* __restrict__ grad,
             float* __restrict__ exp_avg, float* __restrict__ exp_avg_sq, long long n, float lr,
             float beta1, float beta2, float eps, float weight_decay, float bias1, float bias2,
             float grad_scale, int zero_grad) {
  const long long vecs = n / 4;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < vecs;
       i += (long long)gridDim.x * blockDim.x) {
    float4 p = reinterpret_cast<float4*>(master)[i];
    float4 g = reinterpret_cast<float4*>(grad)[i];
    float4 m = reinterpret_cast<float4*>(exp_avg)[i];
    float4 v = reinterpret_cast<float4*>(exp_avg_sq)[i];
    float* pp = &p.x; float* gg = &g.x; float* mm = &m.x; float* vv = &v.x;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float gk = gg[k] * grad_scale;
      mm[k] = beta1 * mm[k] + (1.0f - beta1) * gk;
      vv[k] = beta2 * vv[k] + (1.0f - beta2) * gk * gk;
      const float mhat = mm[k] / bias1;
      const float vhat = vv[k] / bias2;
      pp[k] = pp[k] * (1.0f - lr * weight_decay) - lr * mhat / (sqrtf(vhat) + eps);
    }
    reinterpret_cast<float4*>(master)[i] = p;
    reinterpret_cast<float4*>(exp_avg)[i] = m;
    reinterpret_cast<float4*>(exp_avg_sq)[i] = v;
    if (zero_grad) reinterpret_cast<float4*>(grad)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (param_bf16) {
      __nv_bfloat162 lo = __floats2bfloat162_rn(p.x, p.y);
      __nv_bfloat162 hi = __floats2bfloat162_rn(p.z, p.w);
      uint2 packed;
      packed.x = *reinterpret_cast<uint32_t*>(&lo);
      packed.y = *reinterpret_cast<uint32_t*>(&hi);
      reinterpret_cast<uint2*>(param_bf16)[i] = packed;
    }
  }
}

// SGD with momentum over flat fp32 buffers (ResNet DDP trainer)
__global__ void __launch_bounds__(256)
sgd_momentum_kernel(float* __restrict__ param, float* __restrict__ grad, float* __restrict__ mom,
                    long long n, float lr, float momentum, float weight_decay, float grad_scale,
                    int zero_grad) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const float g = grad[i] * grad_scale + weight_decay * param[i];
    const float b = momentum * mom[i] + g;
    mom[i] = b;
    param[i] -= lr * b;
    if (zero_grad) grad[i] = 0.0f;
  }
}

// below this a row does not fill the 512 threads (4096 rows: 21.3 -> 25.5 us at 2048, 29.4 ->
// 29.6 at 4096, 45.9 -> 37.9 at 8192, 88 -> 63 at 16384)
constexpr int kCeMinVocab = 8192;
// 228 KiB per SM, 1 KiB of it taken by each CTA
constexpr int kCeMaxSmem = (228 / 2 - 1) * 1024;
constexpr int kCeMaxSmem3 = (228 / 3 - 1) * 1024;

static int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

static int grid_for(long long work, int threads) {
  const int sms = sm_count();
  long long g = (work + threads - 1) / threads;
  const long long cap = (long long)sms * 8;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

}  // namespace ew

using namespace ew;

extern "C" {

int bcom_rmsnorm_fwd(const void* x, const void* w, void* y, void* rstd, int rows, int H,
                     float eps, void* stream) {
  if (rows <= 0) return 0;
  if (H % 8) return (int)cudaErrorInvalidValue;
  cudaStream_t st = (cudaStream_t)stream;
  // a row is NV x 8 elements of up to 256 threads; few enough CTAs that each has a next row
  const int vecs = H / 8;
  if (vecs > 8 * 256 || vecs == 0) {
    rmsnorm_fwd_wide_kernel<<<rows < 148 * 8 ? rows : 148 * 8, 256, 0, st>>>(
        (const bf16*)x, (const bf16*)w, (bf16*)y, (float*)rstd, rows, H, eps);
    return (int)cudaGetLastError();
  }
  const int nv = vecs <= 256 ? 1 : vecs <= 512 ? 2 : vecs <= 1024 ? 4 : 8;
  const int threads = ((vecs + nv - 1) / nv + 31) / 32 * 32;
  const int per_sm = nv <= 2 ? 6 : nv <= 4 ? 4 : 2;
  const int grid = rows < 148 * per_sm ? rows : 148 * per_sm;
#define BCOM_RMS_FWD(N)                                                                    \
  rmsnorm_fwd_kernel<N><<<grid, threads, 0, st>>>((const bf16*)x, (const bf16*)w, (bf16*)y, \
                                                  (float*)rstd, rows, H, eps)
  if (nv == 1) BCOM_RMS_FWD(1);
  else if (nv == 2) BCOM_RMS_FWD(2);
  else if (nv == 4) BCOM_RMS_FWD(4);
  else BCOM_RMS_FWD(8);
#undef BCOM_RMS_FWD
  return (int)cudaGetLastError();
}

// `partials`: fp32 scratch of at least bcom_norm_bwd_scratch_elems(H, layernorm) elements,
// private to the call until it has run.  `dres`: optional bf16 [rows, H] added to dx.
static const int kRmsBwdMaxCtas = 148 * 2;
static const int kLnBwdMaxCtas = 148 * 4;

long long bcom_norm_bwd_scratch_elems(int H, int layernorm) {
  return layernorm ? (long long)kLnBwdMaxCtas * 2 * H : (long long)kRmsBwdMaxCtas * H;
}

int bcom_rmsnorm_bwd(const void* dy, const void* x, const void* w, const void* rstd,
                     const void* dres, void* dx, void* dw_fp32, void* partials, int rows, int H,
                     void* stream) {
  if (rows <= 0) return 0;
  if (H % 8) return (int)cudaErrorInvalidValue;
  const int grid = rows < kRmsBwdMaxCtas ? rows : kRmsBwdMaxCtas;
  const int iters = (H / 8 + 511) / 512;
  cudaStream_t st = (cudaStream_t)stream;
#define BCOM_RMS_BWD(N)                                                                       \
  do {                                                                                        \
    if (dres)                                                                                 \
      rmsnorm_bwd_kernel<N, true><<<grid, 512, 0, st>>>(                                      \
          (const bf16*)dy, (const bf16*)x, (const bf16*)w, (const float*)rstd,                \
          (const bf16*)dres, (bf16*)dx, (float*)partials, rows, H);                           \
    else                                                                                      \
      rmsnorm_bwd_kernel<N, false><<<grid, 512, 0, st>>>(                                     \
          (const bf16*)dy, (const bf16*)x, (const bf16*)w, (const float*)rstd, nullptr,       \
          (bf16*)dx, (float*)partials, rows, H);                                              \
  } while (0)
  if (iters <= 1) BCOM_RMS_BWD(1);
  else if (iters <= 2) BCOM_RMS_BWD(2);
  else if (iters <= 4) BCOM_RMS_BWD(4);
  else return (int)cudaErrorInvalidValue;  // H up to 16384
#undef BCOM_RMS_BWD
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return (int)err;
  colsum_add_kernel<<<(H + 31) / 32, dim3(32, 32), 0, st>>>(
      (const float*)partials, (float*)dw_fp32, nullptr, grid, H, H);
  return (int)cudaGetLastError();
}

// LayerNorm over rows of H <= 1024 elements (H % 8 == 0; one warp keeps a row in
// registers); mean / rstd: fp32 [rows].
int bcom_layernorm_fwd(const void* x, const void* w, const void* b, void* y, void* mean,
                       void* rstd, int rows, int H, float eps, void* stream) {
  if (rows <= 0) return 0;
  if (H % 8 || H > 1024) return (int)cudaErrorInvalidValue;
  const int warps = 8;
  const int want = (rows + warps - 1) / warps;
  const int grid = want < 148 * 8 ? want : 148 * 8;
  cudaStream_t st = (cudaStream_t)stream;
  const int iters = (H / 8 + 31) / 32;
#define BCOM_LN_FWD(N)                                                                       \
  layernorm_fwd_kernel<N><<<grid, warps * 32, 0, st>>>(                                       \
      (const bf16*)x, (const bf16*)w, (const bf16*)b, (bf16*)y, (float*)mean, (float*)rstd,  \
      rows, H, eps)
  if (iters <= 2) BCOM_LN_FWD(2);
  else BCOM_LN_FWD(4);
#undef BCOM_LN_FWD
  return (int)cudaGetLastError();
}

// dw / db: fp32 [H], accumulated into (not overwritten); `partials`: see bcom_rmsnorm_bwd.
int bcom_layernorm_bwd(const void* dy, const void* x, const void* w, const void* mean,
                       const void* rstd, void* dx, void* dw_fp32, void* db_fp32, void* partials,
                       int rows, int H, void* stream) {
  if (rows <= 0) return 0;
  if (H % 8 || H > 1024) return (int)cudaErrorInvalidValue;
  const int grid = rows < kLnBwdMaxCtas ? rows : kLnBwdMaxCtas;
  const int threads = ((H / 8 + 31) / 32) * 32;
  cudaStream_t st = (cudaStream_t)stream;
  layernorm_bwd_row_kernel<<<grid, threads, 0, st>>>(
      (const bf16*)dy, (const bf16*)x, (const bf16*)w, (const float*)mean, (const float*)rstd,
      (bf16*)dx, (float*)partials, rows, H);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return (int)err;
  // a partial row is [dw | db]
  colsum_add_kernel<<<(2 * H + 31) / 32, dim3(32, 32), 0, st>>>(
      (const float*)partials, (float*)dw_fp32, (float*)db_fp32, grid, 2 * H, H);
  return (int)cudaGetLastError();
}

// out[c] += sum over rows of x[row, c] (bf16 [rows, C], C % 8 == 0, 16-byte aligned; out fp32).
// `partials`: fp32 scratch of bcom_colsum_strips(rows, C) * C elements.
int bcom_colsum_strips(long long rows, int C) {
  if (C <= 0) return 1;
  const int col_tiles = (C / 8 + 127) / 128;
  long long strips = (148LL * 8 + col_tiles - 1) / col_tiles;
  if (strips > (rows + 3) / 4) strips = (rows + 3) / 4;
  return (int)(strips < 1 ? 1 : strips);
}

int bcom_colsum_bf16(const void* x, void* out_fp32, void* partials, long long rows, int C,
                     void* stream) {
  if (rows <= 0 || C <= 0) return 0;
  if ((C % 8) || ((uintptr_t)x & 15)) return (int)cudaErrorInvalidValue;
  const int strips = bcom_colsum_strips(rows, C);
  cudaStream_t st = (cudaStream_t)stream;
  colsum_bf16_kernel<<<dim3((C / 8 + 127) / 128, strips), 128, 0, st>>>(
      (const bf16*)x, (float*)partials, rows, C);
  colsum_add_kernel<<<(C + 31) / 32, dim3(32, 32), 0, st>>>((const float*)partials,
                                                            (float*)out_fp32, nullptr, strips, C, C);
  return (int)cudaGetLastError();
}

int bcom_bias_gelu_fwd(const void* x, const void* bias, void* y, long long rows, int C,
                       void* stream) {
  if (rows <= 0 || C == 0) return 0;
  if (C % 8) return (int)cudaErrorInvalidValue;
  const int col_tiles = (C / 8 + 127) / 128;
  long long strips = (148LL * 16 + col_tiles - 1) / col_tiles;
  if (strips > rows) strips = rows;
  if (strips > 65535) strips = 65535;
  bias_gelu_fwd_kernel<<<dim3(col_tiles, (unsigned)strips), 128, 0, (cudaStream_t)stream>>>(
      (const bf16*)x, (const bf16*)bias, (bf16*)y, rows, C);
  return (int)cudaGetLastError();
}

// dbias: fp32 [C], accumulated into.
int bcom_bias_gelu_bwd(const void* dy, const void* x, const void* bias, void* dx,
                       void* dbias_fp32, long long rows, int C, void* stream) {
  if (rows <= 0 || C == 0) return 0;
  if (C % 8) return (int)cudaErrorInvalidValue;
  const int threads = 128;
  const int col_tiles = (C / 8 + threads - 1) / threads;
  int strips = (148 * 4 + col_tiles - 1) / col_tiles;
  if (strips > rows) strips = (int)rows;
  if (strips > 65535) strips = 65535;
  bias_gelu_bwd_kernel<<<dim3(col_tiles, strips), threads, 0, (cudaStream_t)stream>>>(
      (const bf16*)dy, (const bf16*)x, (const bf16*)bias, (bf16*)dx, (float*)dbias_fp32, rows, C);
  return (int)cudaGetLastError();
}

static int launch_rope(const void* src, void* dst, const void* cos_t, const void* sin_t,
                       long long tokens, int heads, int head_dim, long long row_stride, int width,
                       int seq, int backward, bool out_of_place, void* stream) {
  if (tokens <= 0) return 0;
  // 16-byte accesses: halves of whole 8-element groups, rows and bases aligned
  if (seq <= 0 || head_dim % 16 || row_stride % 8 || width % 8 ||
      (((uintptr_t)src | (uintptr_t)dst) & 15))
    return (int)cudaErrorInvalidValue;
  const bool tables_aligned = (((uintptr_t)cos_t | (uintptr_t)sin_t) & 15) == 0;
  const int items = heads * (head_dim / 16) + (out_of_place ? (width - heads * head_dim) / 8 : 0);
  if (items <= 0) return 0;  // no heads
  const int cols = (items + 255) / 256;
  const long long most_rows = (148LL * 16 + cols - 1) / cols;
  auto kernel = out_of_place ? rope_kernel<true> : rope_kernel<false>;
  for (long long first = 0; first < tokens;) {
    const RopeChunk part = rope_chunk(tokens, seq, first);
    const long long rows = most_rows < part.tokens ? most_rows : part.tokens;
    kernel<<<dim3(cols, (unsigned)rows), 256, 0, (cudaStream_t)stream>>>(
        (const bf16*)src + first * row_stride, (bf16*)dst + first * row_stride,
        (const float*)cos_t, (const float*)sin_t, part.tokens, heads, head_dim, row_stride, width,
        seq, part.position, backward ? -1.0f : 1.0f, tables_aligned);
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return (int)err;
    first += part.tokens;
  }
  return 0;
}

// In place on the first heads * head_dim columns of rows `row_stride` apart.
int bcom_rope(void* x, const void* cos_t, const void* sin_t, long long tokens, int heads,
              int head_dim, long long row_stride, int seq, int backward, void* stream) {
  return launch_rope(x, x, cos_t, sin_t, tokens, heads, head_dim, row_stride, 0, seq, backward,
                     false, stream);
}

// dst = src with the first heads * head_dim of `width` columns rotated and the rest copied (rows
// of both `row_stride` apart).
int bcom_rope_copy(const void* src, void* dst, const void* cos_t, const void* sin_t,
                   long long tokens, int heads, int head_dim, long long row_stride, int width,
                   int seq, int backward, void* stream) {
  return launch_rope(src, dst, cos_t, sin_t, tokens, heads, head_dim, row_stride, width, seq,
                     backward, true, stream);
}

int bcom_swiglu_fwd(const void* gate_up, void* h, long long tokens, int F, void* stream) {
  if (tokens <= 0) return 0;
  if (F % 8) return (int)cudaErrorInvalidValue;
  swiglu_fwd_kernel<<<grid_for(tokens * (F / 8), 256), 256, 0, (cudaStream_t)stream>>>(
      (const bf16*)gate_up, (bf16*)h, tokens, F);
  return (int)cudaGetLastError();
}

int bcom_swiglu_bwd(const void* gate_up, const void* dh, void* dgate_up, long long tokens, int F,
                    void* stream) {
  if (tokens <= 0) return 0;
  if (F % 8) return (int)cudaErrorInvalidValue;
  swiglu_bwd_kernel<<<grid_for(tokens * (F / 8), 256), 256, 0, (cudaStream_t)stream>>>(
      (const bf16*)gate_up, (const bf16*)dh, (bf16*)dgate_up, tokens, F);
  return (int)cudaGetLastError();
}

int bcom_cross_entropy(void* logits, const void* targets, void* loss_out, const void* grad_scale,
                       int rows, int V, long long ignore_index, void* stream) {
  if (rows <= 0) return 0;
  if (V % 8) return (int)cudaErrorInvalidValue;
  const int smem = (int)sizeof(CeShared) + 2 * V;
  if (V >= kCeMinVocab && smem <= kCeMaxSmem && ((uintptr_t)logits & 15) == 0) {
    const bool three = smem <= kCeMaxSmem3;
    auto kernel = three ? cross_entropy_rows_kernel<3> : cross_entropy_rows_kernel<2>;
    if (!tc::ensure_dynamic_smem((const void*)kernel, three ? kCeMaxSmem3 : kCeMaxSmem))
      return (int)cudaErrorInvalidValue;
    const int most = sm_count() * (three ? 3 : 2);
    kernel<<<rows < most ? rows : most, kCeThreads, smem, (cudaStream_t)stream>>>(
        (bf16*)logits, (const long long*)targets, (float*)loss_out, (const float*)grad_scale,
        rows, V, ignore_index);
    return (int)cudaGetLastError();
  }
  const int grid = rows < 148 * 4 ? rows : 148 * 4;
  cross_entropy_kernel<<<grid, 512, 0, (cudaStream_t)stream>>>(
      (bf16*)logits, (const long long*)targets, (float*)loss_out, (const float*)grad_scale, rows,
      V, ignore_index);
  return (int)cudaGetLastError();
}

// valid[0] = max(1, #targets != ignore_index), scale[0] = loss_scale / valid (fp32 each)
int bcom_cross_entropy_scale(const void* targets, long long rows, long long ignore_index,
                             float loss_scale, void* valid, void* scale, void* stream) {
  cross_entropy_scale_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(
      (const long long*)targets, rows, ignore_index, loss_scale, (float*)valid, (float*)scale);
  return (int)cudaGetLastError();
}

int bcom_cross_entropy_sum(const void* per_row, long long rows, const void* scale, void* loss,
                           void* stream) {
  cross_entropy_sum_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(
      (const float*)per_row, rows, (const float*)scale, (float*)loss);
  return (int)cudaGetLastError();
}

// x (bf16, n % 8 == 0, 16-byte aligned) *= bf16(factor[0])
int bcom_scale_bf16(void* x, long long n, const void* factor, void* stream) {
  if (n <= 0) return 0;
  if ((n % 8) || ((uintptr_t)x & 15)) return (int)cudaErrorInvalidValue;
  scale_inplace_kernel<<<grid_for(n / 8, 256), 256, 0, (cudaStream_t)stream>>>(
      (bf16*)x, n / 8, (const float*)factor);
  return (int)cudaGetLastError();
}

// 0, or the wait that ran out in a cross-entropy launch; cleared when `clear` != 0
int bcom_cross_entropy_status(unsigned int* out, int clear) {
  cudaError_t err = cudaMemcpyFromSymbol(out, g_ce_status, sizeof(unsigned int));
  const unsigned int zero = 0;
  if (err == cudaSuccess && clear) err = cudaMemcpyToSymbol(g_ce_status, &zero, sizeof(zero));
  return (int)err;
}

int bcom_embedding_fwd(const void* ids, const void* table, void* out, long long tokens, int H,
                       int vocab, void* stream) {
  if (tokens <= 0) return 0;
  if (H % 8) return (int)cudaErrorInvalidValue;
  embedding_fwd_kernel<<<grid_for(tokens * (H / 8), 256), 256, 0, (cudaStream_t)stream>>>(
      (const long long*)ids, (const bf16*)table, (bf16*)out, tokens, H, vocab);
  return (int)cudaGetLastError();
}

int bcom_embedding_bwd(const void* ids, const void* dout, void* dtable_fp32, long long tokens,
                       int H, int vocab, void* stream) {
  if (tokens <= 0) return 0;
  if (H % 8) return (int)cudaErrorInvalidValue;
  embedding_bwd_kernel<<<grid_for(tokens * (H / 8), 256), 256, 0, (cudaStream_t)stream>>>(
      (const long long*)ids, (const bf16*)dout, (float*)dtable_fp32, tokens, H, vocab,
      ((uintptr_t)dtable_fp32 & 15) == 0);
  return (int)cudaGetLastError();
}

int bcom_adamw(void* master, void* param_bf16, void* grad, void* exp_avg, void* exp_avg_sq,
               long long n, float lr, float beta1, float beta2, float eps, float weight_decay,
               int step, float grad_scale, int zero_grad, void* stream) {
  if (n <= 0) return 0;
  if (n % 4) return (int)cudaErrorInvalidValue;
  const float bias1 = 1.0f - powf(beta1, (float)step);
  const float bias2 = 1.0f - powf(beta2, (float)step);
  adamw_kernel<<<grid_for(n / 4, 256), 256, 0, (cudaStream_t)stream>>>(
      (float*)master, (bf16*)param_bf16, (float*)grad, (float*)exp_avg, (float*)exp_avg_sq, n, lr,
      beta1, beta2, eps, weight_decay, bias1, bias2, grad_scale, zero_grad);
  return (int)cudaGetLastError();
}

int bcom_sgd_momentum(void* param, void* grad, void* mom, long long n, float lr, float momentum,
                      float weight_decay, float grad_scale, int zero_grad, void* stream) {
  if (n <= 0) return 0;
  sgd_momentum_kernel<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(
      (float*)param, (float*)grad, (float*)mom, n, lr, momentum, weight_decay, grad_scale,
      zero_grad);
  return (int)cudaGetLastError();
}

}  // extern "C"
