// Epilogue of the tcgen05 GEMM kernels: one warp moves its 32 accumulator rows (TMEM lanes)
// of a BN-column tile from tensor memory to global memory, as bf16 or fp32, overwriting or
// accumulating.  Shared by the one-CTA kernel (gemm_tcgen05.cu) and the CTA-pair kernel
// (gemm_tcgen05_2cta.cu); thread t of the warp holds row `row0` + t.
//
// The rows leave through shared memory: each thread writes its row of a 128-byte wide chunk
// (64 bf16 or 32 fp32 columns, 128-byte swizzle: no bank conflicts), one lane sends the 32 x 128
// byte box with a bulk tensor store, which also clips it at the edges of C.  Two chunks per
// warp alternate over all its tiles, so the next one is read from tensor memory while the last
// one is on its way.
// An accumulating fp32 C (weight gradients) takes the box as a bulk reduction: the addition is
// done by the L2, C is never read into an SM.  Stores straight from the registers, 16 bytes per
// lane at a row's distance, cost 32 wavefronts per instruction and the accumulating form waited
// on its reads (a gradient of 32000 x 4096 from 128 tokens took 350 us for 1 GB of traffic).
#pragma once

#include "gemm_schedule.cuh"
#include "tc_common.cuh"

namespace gemm {

constexpr int EPI_CHUNK_BYTES = 32 * 128;
constexpr int EPI_WARP_BYTES = 2 * EPI_CHUNK_BYTES;  // two chunks per epilogue warp
constexpr int EPI_BYTES = 4 * EPI_WARP_BYTES;        // four epilogue warps per CTA

// byte offset of the 16-byte unit `u` of row `r` inside a 128-byte swizzled chunk
__device__ __forceinline__ uint32_t epi_swz(int r, int u) {
  return (uint32_t)(r * 128 + ((u ^ (r & 7)) << 4));
}

// taddr: TMEM address of the warp's first lane at the tile's first column.  C rows [row0, row0 +
// 32), columns [n0, n0 + BN) are written where row < M and column < N (N % 8 == 0).
// R (bf16 [M, N] with leading dimension ldr, or null): added to the product before the bf16
// result is rounded (a linear layer whose output joins a residual stream: C = R + A x B in one
// pass instead of a GEMM and an add kernel).  bias (bf16 [N], 16-byte aligned, or null): likewise.
template <int BN, bool OUT_F32, bool ACCUM>
__device__ __forceinline__ void store_accumulator_tma(uint32_t taddr, const CUtensorMap* tmC,
                                                      uint8_t* stage, int row0, int n0, int M,
                                                      int N, const void* R, long long ldr,
                                                      const void* bias, int lane,
                                                      gemm_sched::StagingChunks& chunks) {
  static_assert(OUT_F32 || !ACCUM, "bf16 accumulation reads C: store_accumulator_rows");
  constexpr int COLS = OUT_F32 ? 32 : 64;
  if (row0 >= M) return;
#pragma unroll 1
  for (int c = 0; c < BN / COLS; ++c) {
    const int col0 = n0 + c * COLS;
    if (col0 >= N) break;
    uint8_t* buf = stage + chunks.next() * EPI_CHUNK_BYTES;
    if constexpr (OUT_F32) {
      uint32_t r[32];
      tc::tmem_ld_32x32(taddr + c * COLS, r);
      if (lane == 0) tc::bulk_wait_group_read1();  // the box sent two chunks ago has left `buf`
      __syncwarp();
      tc::tmem_wait_ld();
#pragma unroll
      for (int u = 0; u < 8; ++u)
        *reinterpret_cast<uint4*>(buf + epi_swz(lane, u)) =
            make_uint4(r[4 * u], r[4 * u + 1], r[4 * u + 2], r[4 * u + 3]);
    } else {
      uint32_t r[64];
      tc::tmem_ld_32x32(taddr + c * COLS, reinterpret_cast<uint32_t(&)[32]>(r[0]));
      tc::tmem_ld_32x32(taddr + c * COLS + 32, reinterpret_cast<uint32_t(&)[32]>(r[32]));
      uint4 res[8];
      const bool add = R != nullptr && row0 + lane < M;
      if (add) {  // requested before the wait on the TMEM loads
        const __nv_bfloat16* rrow =
            reinterpret_cast<const __nv_bfloat16*>(R) + (long long)(row0 + lane) * ldr + col0;
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (col0 + u * 8 < N) res[u] = *reinterpret_cast<const uint4*>(rrow + u * 8);
      }
      if (lane == 0) tc::bulk_wait_group_read1();
      __syncwarp();
      tc::tmem_wait_ld();
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        float f[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(r[8 * u + i]);
        if (bias != nullptr && col0 + u * 8 < N) {  // one address for the whole warp
          const uint4 b = __ldg(reinterpret_cast<const uint4*>(
              reinterpret_cast<const __nv_bfloat16*>(bias) + col0 + u * 8));
          const __nv_bfloat16* bh = reinterpret_cast<const __nv_bfloat16*>(&b);
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] += __bfloat162float(bh[i]);
        }
        if (add && col0 + u * 8 < N) {
          const __nv_bfloat16* rh = reinterpret_cast<const __nv_bfloat16*>(&res[u]);
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] += __bfloat162float(rh[i]);
        }
        uint4 o;
        __nv_bfloat162* oh2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int i = 0; i < 4; ++i) oh2[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
        *reinterpret_cast<uint4*>(buf + epi_swz(lane, u)) = o;
      }
    }
    tc::fence_proxy_async();  // the chunk is visible to the copy engine
    __syncwarp();
    if (lane == 0) {
      if constexpr (ACCUM) tc::tma_reduce_add_2d(tmC, buf, col0, row0);
      else tc::tma_store_2d(tmC, buf, col0, row0);
      tc::bulk_commit_group();
    }
  }
}

// bf16 C += A x B: the old values are read, the sum is rounded once.
template <int BN>
__device__ __forceinline__ void accumulate_bf16_rows(uint32_t taddr, void* C, long long ldc,
                                                     int row, int n0, int M, int N) {
#pragma unroll 1
  for (int c = 0; c < BN / 32; ++c) {
    uint32_t r[32];
    tc::tmem_ld_32x32(taddr + c * 32, r);
    const int col0 = n0 + c * 32;
    tc::tmem_wait_ld();
    if (row < M && col0 < N) {
      __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(C) + (long long)row * ldc + col0;
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        if (col0 + v * 8 < N) {
          const uint4 old = *reinterpret_cast<const uint4*>(dst + v * 8);
          const __nv_bfloat16* oh = reinterpret_cast<const __nv_bfloat16*>(&old);
          uint4 o;
          __nv_bfloat162* oh2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            oh2[i] = __floats2bfloat162_rn(
                __uint_as_float(r[8 * v + 2 * i]) + __bfloat162float(oh[2 * i]),
                __uint_as_float(r[8 * v + 2 * i + 1]) + __bfloat162float(oh[2 * i + 1]));
          *reinterpret_cast<uint4*>(dst + v * 8) = o;
        }
      }
    }
  }
}

// What an epilogue warp does with a finished tile.
template <int BN, bool OUT_F32, bool ACCUM>
__device__ __forceinline__ void write_accumulator(uint32_t taddr, const CUtensorMap* tmC,
                                                  uint8_t* stage, void* C, long long ldc, int row0,
                                                  int n0, int M, int N, const void* R,
                                                  long long ldr, const void* bias, int lane,
                                                  gemm_sched::StagingChunks& chunks) {
  if constexpr (!OUT_F32 && ACCUM)
    accumulate_bf16_rows<BN>(taddr, C, ldc, row0 + lane, n0, M, N);
  else
    store_accumulator_tma<BN, OUT_F32, ACCUM>(taddr, tmC, stage, row0, n0, M, N, R, ldr, bias,
                                              lane, chunks);
}

// Tensor map of C for the boxes above.
inline int make_c_map(CUtensorMap* map, const void* C, int M, int N, long long ldc,
                      bool out_fp32) {
  if (M == 1 && ldc < N) ldc = (N + 7) / 8 * 8;  // a single row has no distance to the next
  return out_fp32 ? tc::cached_tensor_map_2d(map, C, 4, M, N, ldc, 32, 32)
                  : tc::cached_tensor_map_2d(map, C, 2, M, N, ldc, 64, 32);
}

}  // namespace gemm
