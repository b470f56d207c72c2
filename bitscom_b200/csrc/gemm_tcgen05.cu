// bf16 GEMM on the 5th-generation tensor cores (sm_100a): C[M,N] (+)= A x B with fp32
// accumulation in tensor memory.
//
//   * persistent grid, one CTA per SM, static round-robin over work items: output tiles of
//     128x256 or 128x128 (grouped along M so that concurrently running CTAs share B tiles in
//     L2), the latter also with K shared out among several items per tile, whose fp32 partial
//     tiles a second kernel adds up;
//   * warp 0: TMA producer (cp.async.bulk.tensor 2-D tiles, 128-byte swizzle) into a
//     192 KiB shared-memory ring (4 stages of 48 KiB or 6 of 32 KiB);
//   * warp 1: allocates two accumulators of TMEM and issues tcgen05.mma (cta_group::1, M=128,
//     N=256 or 128, K=16 per instruction): the whole warp walks the loop, an elected lane
//     issues; tcgen05.commit releases ring stages and publishes finished accumulators;
//   * warps 2-5: epilogue (gemm_epilogue.cuh). The two accumulators alternate, so the epilogue
//     of item i (tcgen05.ld -> registers -> shared memory -> bulk tensor store or reduction)
//     overlaps the main loop of item i+1.
//
// Operand layouts.  Either operand may be K-major (reduction dimension contiguous) or
// MN-major (the other dimension contiguous); this covers forward (x W^T), data
// gradient (dy W) and weight gradient (dy^T x) of a linear layer without transposes:
//
//   K-major  X[rows=MN, cols=K]  one TMA box {64 k, BM|BN rows}; descriptor SBO = 1024
//   MN-major X[rows=K, cols=MN]  boxes {64 mn, 64 k} side by side, 8 KiB each;
//                                descriptor LBO = 8192 (next 64-wide MN chunk), SBO = 1024
//
// Every mbarrier wait is bounded; on expiry the kernel records a code, all roles drain,
// TMEM is released and the kernel returns.  torch.matmul / cuBLAS is the library
// baseline this replaces for the trainer's linear layers (the reference trainer's model
// code is plain nn.Linear, benchmarks/train_llama7b_dp_pp_lowbit.py:222-238).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <mutex>

#include "gemm_epilogue.cuh"
#include "gemm_schedule.cuh"
#include "tc_common.cuh"

namespace gemm {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int A_BYTES = BM * BK * 2;  // 16 KiB
constexpr int CHUNK_BYTES = 64 * BK * 2;  // one MN-major box: 64 mn x 64 k
constexpr int kThreads = 192;
constexpr int MAX_STAGES = 6;
// Output tiles are 128 x 256, or 128 x 128 where that many columns leave SMs without a tile.
template <int BN> struct Tile {
  static constexpr int STAGES = BN == 256 ? 4 : 6;
  static constexpr int B_BYTES = BN * BK * 2;             // 32 or 16 KiB
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;   // 192 KiB of ring in both
  static constexpr uint32_t TMEM_COLS = 2 * BN;
  static constexpr int SMEM_BYTES =
      STAGES * STAGE_BYTES + EPI_BYTES + 1024 /*alignment slack*/ + 256;
};
constexpr int GROUP_M = 8;
constexpr unsigned long long kWaitBudgetNs = 2000000000ull;

enum Status : unsigned int {
  kOk = 0, kProducerTimeout = 1, kMmaTimeout = 2, kEpilogueTimeout = 3, kAccumTimeout = 4
};

__device__ unsigned int g_status[4];

struct Params {
  void* C;
  const void* R;  // optional bf16 residual added in the bf16 epilogue (see gemm_epilogue.cuh)
  const void* bias;  // optional bf16 [N], likewise
  long long ldc, ldr;
  int M, N, K;
  int tiles_m, tiles_n;
  // K shared out among this many work items per tile; item s of a tile writes its fp32 partial
  // tile to rows [s * split_rows, ...) of C, which is then the workspace of the call.
  int splits, split_rows;
};

struct Shared {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  volatile int abort;
};

__device__ __forceinline__ void fail(Shared* sh, unsigned int code) {
  sh->abort = 1;
  if (atomicCAS(&g_status[0], 0u, code) == 0u) {
    g_status[1] = blockIdx.x;
    g_status[2] = threadIdx.x;
  }
}

// One unit of work of a CTA: k-blocks [kb0, kb1) of rows [m0, m0 + BM), columns [n0, n0 + BN).
struct WorkItem {
  int m0, n0, kb0, kb1, split;
};
template <int BN>
__device__ __forceinline__ WorkItem work_item(const Params& p, int w) {
  const int tiles = p.tiles_m * p.tiles_n;
  const int num_kb = (p.K + BK - 1) / BK;
  const int split = p.splits == 1 ? 0 : w / tiles;
  const gemm_sched::WorkItem t =
      gemm_sched::work_item<BM, BN, GROUP_M>(p.tiles_m, p.tiles_n, w - split * tiles);
  return WorkItem{t.m0, t.n0, gemm_sched::split_begin(num_kb, p.splits, split),
                  gemm_sched::split_begin(num_kb, p.splits, split + 1), split};
}

template <int BN, bool A_MN, bool B_MN, bool OUT_F32, bool ACCUM>
__global__ void __launch_bounds__(kThreads, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmC, const Params p) {
  constexpr int STAGES = Tile<BN>::STAGES, STAGE_BYTES = Tile<BN>::STAGE_BYTES;
  constexpr uint32_t TMEM_COLS = Tile<BN>::TMEM_COLS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* epi = smem + STAGES * STAGE_BYTES;
  Shared* sh = reinterpret_cast<Shared*>(epi + EPI_BYTES);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int total_tiles = p.tiles_m * p.tiles_n * p.splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      tc::mbar_init(&sh->full[s], 1);
      tc::mbar_init(&sh->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&sh->acc_full[b], 1);
      tc::mbar_init(&sh->acc_empty[b], 4);
    }
    sh->abort = 0;
    tc::fence_mbar_init();
  }
  if (warp == 1) tc::tmem_alloc(&sh->tmem_base, TMEM_COLS);
  tc::tc_fence_before_sync();
  __syncthreads();
  tc::tc_fence_after_sync();
  const uint32_t tmem_base = sh->tmem_base;

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      tc::tma_prefetch_desc(&tmA);
      tc::tma_prefetch_desc(&tmB);
      int stage = 0;
      uint32_t phase = 0;
      for (int t = blockIdx.x; t < total_tiles && !sh->abort; t += gridDim.x) {
        const WorkItem wi = work_item<BN>(p, t);
        const int m0 = wi.m0, n0 = wi.n0;
        for (int kb = wi.kb0; kb < wi.kb1; ++kb) {
          if (!tc::mbar_wait(&sh->empty[stage], phase ^ 1u, kWaitBudgetNs)) {
            fail(sh, kProducerTimeout);
            break;
          }
          uint8_t* sA = smem + stage * STAGE_BYTES;
          uint8_t* sB = sA + A_BYTES;
          tc::mbar_expect_tx(&sh->full[stage], STAGE_BYTES);
          const int k0 = kb * BK;
          if constexpr (A_MN) {
#pragma unroll
            for (int c = 0; c < BM / 64; ++c)
              tc::tma_load_2d(sA + c * CHUNK_BYTES, &tmA, &sh->full[stage], m0 + c * 64, k0);
          } else {
            tc::tma_load_2d(sA, &tmA, &sh->full[stage], k0, m0);
          }
          if constexpr (B_MN) {
#pragma unroll
            for (int c = 0; c < BN / 64; ++c)
              tc::tma_load_2d(sB + c * CHUNK_BYTES, &tmB, &sh->full[stage], n0 + c * 64, k0);
          } else {
            tc::tma_load_2d(sB, &tmB, &sh->full[stage], k0, n0);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ---------------------------------
    // The whole warp walks the loop and one elected lane issues: with `if (lane == 0)` around
    // the loop every descriptor and address is a per-thread value that has to be moved into the
    // uniform registers the MMA takes, and that issue work, not the tensor pipe, set the pace
    // (the tensor pipe is now active in 0.83 of all cycles here, where the operands' way through
    // shared memory is next, and in 0.90 in the CTA-pair kernel, at 4096^3).
    constexpr uint32_t idesc = tc::make_idesc_bf16(BM, BN, A_MN, B_MN);
    constexpr uint32_t hi = tc::desc_hi(1024);
    constexpr uint32_t a_step = (A_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4;
    constexpr uint32_t b_step = (B_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4;
    const uint32_t a_lo0 = tc::desc_lo(tc::smem_u32(smem), A_MN ? CHUNK_BYTES : 16);
    const uint32_t b_lo0 = tc::desc_lo(tc::smem_u32(smem) + A_BYTES, B_MN ? CHUNK_BYTES : 16);
    int stage = 0;
    uint32_t phase = 0;
    int iter = 0;
    for (int t = blockIdx.x; t < total_tiles && !sh->abort; t += gridDim.x, ++iter) {
      const int buf = iter & 1;
      const uint32_t acc_phase = (uint32_t)(iter >> 1) & 1u;
      if (!tc::mbar_wait_warp(&sh->acc_empty[buf], acc_phase ^ 1u, kWaitBudgetNs)) {
        if (lane == 0) fail(sh, kAccumTimeout);
        break;
      }
      tc::tc_fence_after_sync();
      const uint32_t d_tmem = tmem_base + (uint32_t)buf * BN;
      const WorkItem wi = work_item<BN>(p, t);
      bool ok = true;
      for (int kb = wi.kb0; kb < wi.kb1; ++kb) {
        if (!tc::mbar_wait_warp(&sh->full[stage], phase, kWaitBudgetNs)) {
          if (lane == 0) fail(sh, kMmaTimeout);
          ok = false;
          break;
        }
        tc::tc_fence_after_sync();
        const uint32_t a_lo = a_lo0 + stage * (STAGE_BYTES >> 4);
        const uint32_t b_lo = b_lo0 + stage * (STAGE_BYTES >> 4);
        if (tc::elect_one()) {
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            tc::umma_bf16_lo<1>(d_tmem, a_lo + k * a_step, hi, b_lo + k * b_step, hi, idesc,
                                kb != wi.kb0 || k != 0 ? 1u : 0u);
          tc::umma_commit(&sh->empty[stage]);  // stage reusable once these MMAs are done
          if (kb == wi.kb1 - 1) tc::umma_commit(&sh->acc_full[buf]);
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
      if (!ok) break;
    }
  } else {
    // ------------------------------ epilogue -----------------------------------
    const int quarter = warp & 3;  // TMEM lanes this warp may read: 32*quarter ..
    gemm_sched::StagingChunks chunks;
    int iter = 0;
    for (int t = blockIdx.x; t < total_tiles && !sh->abort; t += gridDim.x, ++iter) {
      const WorkItem wi = work_item<BN>(p, t);
      const int buf = iter & 1;
      const uint32_t acc_phase = (uint32_t)(iter >> 1) & 1u;
      if (!tc::mbar_wait(&sh->acc_full[buf], acc_phase, kWaitBudgetNs)) {
        if (lane == 0) fail(sh, kEpilogueTimeout);
        break;
      }
      tc::tc_fence_after_sync();
      const uint32_t taddr = tmem_base + (uint32_t)buf * BN + ((uint32_t)(quarter * 32) << 16);
      const int row0 = wi.m0 + quarter * 32;
      if (p.splits == 1)
        write_accumulator<BN, OUT_F32, ACCUM>(taddr, &tmC, epi + quarter * EPI_WARP_BYTES, p.C,
                                              p.ldc, row0, wi.n0, p.M, p.N, p.R, p.ldr, p.bias,
                                              lane, chunks);
      else if constexpr (OUT_F32 && !ACCUM)
        write_accumulator<BN, true, false>(taddr, &tmC, epi + quarter * EPI_WARP_BYTES, p.C, p.ldc,
                                           wi.split * p.split_rows + row0, wi.n0,
                                           p.splits * p.split_rows, p.N, nullptr, 0, nullptr, lane,
                                           chunks);
      tc::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&sh->acc_empty[buf]);
    }
    if (lane == 0) tc::bulk_wait_group0();  // C is written before the CTA leaves
  }

  // ------------------------------ teardown -------------------------------------
  tc::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::tc_fence_after_sync();
    tc::tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// 2-D bf16 row-major matrix [rows, cols] with leading dimension ld (elements).
static int make_map(CUtensorMap* map, const void* ptr, long long rows, long long cols,
                    long long ld, int box_cols, int box_rows) {
  return tc::cached_tensor_map_2d(map, ptr, 2, rows, cols, ld, box_cols, box_rows);
}

static int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

typedef void (*Kernel)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const Params);

template <int BN, bool A_MN, bool B_MN>
static Kernel pick_out(bool out_f32, bool accum) {
  if (out_f32) return accum ? gemm_bf16_kernel<BN, A_MN, B_MN, true, true>
                            : gemm_bf16_kernel<BN, A_MN, B_MN, true, false>;
  return accum ? gemm_bf16_kernel<BN, A_MN, B_MN, false, true>
               : gemm_bf16_kernel<BN, A_MN, B_MN, false, false>;
}

template <int BN>
static Kernel pick(bool a_mn, bool b_mn, bool out_f32, bool accum) {
  if (a_mn) return b_mn ? pick_out<BN, true, true>(out_f32, accum)
                        : pick_out<BN, true, false>(out_f32, accum);
  return b_mn ? pick_out<BN, false, true>(out_f32, accum)
              : pick_out<BN, false, false>(out_f32, accum);
}

// C (bf16 or fp32) = sum over splits of the partial tiles, in ascending order (+ bias, + residual or + C).
// Reads what the product kernel has just written (it is still in the L2).
template <bool OUT_F32, bool ACCUM>
__global__ void __launch_bounds__(256)
split_sum_kernel(const float* __restrict__ ws, int splits, long long split_stride, void* C,
                 const __nv_bfloat16* __restrict__ R, const __nv_bfloat16* __restrict__ bias,
                 long long ldc, long long ldr, int M, int N) {
  const int vec = N / 4;
  const long long total = (long long)M * vec;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int row = (int)(i / vec), col = (int)(i - (long long)row * vec) * 4;
    const float* src = ws + (long long)row * N + col;
    float4 v[8];
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < splits) v[s] = __ldcg(reinterpret_cast<const float4*>(src + s * split_stride));
    float4 a = v[0];
#pragma unroll
    for (int s = 1; s < 8; ++s)
      if (s < splits) { a.x += v[s].x; a.y += v[s].y; a.z += v[s].z; a.w += v[s].w; }
    if constexpr (OUT_F32) {
      float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(C) + row * ldc + col);
      if constexpr (ACCUM) {
        const float4 o = *dst;
        a.x += o.x; a.y += o.y; a.z += o.z; a.w += o.w;
      }
      *dst = a;
    } else {
      __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(C) + row * ldc + col;
      if (!ACCUM && bias) {
        const uint2 o = *reinterpret_cast<const uint2*>(bias + col);
        a.x += __uint_as_float(o.x << 16);
        a.y += __uint_as_float(o.x & 0xffff0000u);
        a.z += __uint_as_float(o.y << 16);
        a.w += __uint_as_float(o.y & 0xffff0000u);
      }
      const __nv_bfloat16* add = ACCUM ? dst : R ? R + row * ldr + col : nullptr;
      if (add) {
        const uint2 o = *reinterpret_cast<const uint2*>(add);
        a.x += __uint_as_float(o.x << 16);
        a.y += __uint_as_float(o.x & 0xffff0000u);
        a.z += __uint_as_float(o.y << 16);
        a.w += __uint_as_float(o.y & 0xffff0000u);
      }
      const __nv_bfloat162 lo = __floats2bfloat162_rn(a.x, a.y), h = __floats2bfloat162_rn(a.z, a.w);
      *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo),
                                                  *reinterpret_cast<const uint32_t*>(&h));
    }
  }
}

// One launch of the product kernel; `splits` > 1: `C` is the fp32 workspace.
template <int BN>
static int launch(const void* A, const void* B, void* C, const void* residual, const void* bias,
                  int M, int N, int K,
                  long long lda, long long ldb, long long ldc, long long ldr, bool a_mn, bool b_mn,
                  bool out_fp32, bool accumulate, int splits, int max_ctas, cudaStream_t stream) {
  CUtensorMap tmA, tmB, tmC;
  // the tensor-map encoder is a driver call: make sure this thread (it may be an autograd
  // worker) has the device's primary context bound
  tc::bind_context_once();
  Params p;
  p.C = C;
  p.R = residual;
  p.bias = bias;
  p.ldc = ldc;
  p.ldr = ldr;
  p.M = M;
  p.N = N;
  p.K = K;
  p.tiles_m = (M + BM - 1) / BM;
  p.tiles_n = (N + BN - 1) / BN;
  p.splits = splits;
  p.split_rows = p.tiles_m * BM;
  const long long items = (long long)p.tiles_m * p.tiles_n * splits;
  int grid = sm_count();
  if (grid > items) grid = (int)items;
  if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
  if (a_mn ? make_map(&tmA, A, K, M, lda, 64, BK) : make_map(&tmA, A, M, K, lda, BK, BM))
    return 1003;
  if (b_mn ? make_map(&tmB, B, K, N, ldb, 64, BK) : make_map(&tmB, B, N, K, ldb, BK, BN))
    return 1004;
  if (make_c_map(&tmC, C, splits > 1 ? splits * p.split_rows : M, N, ldc, out_fp32)) return 1008;
  Kernel kernel = pick<BN>(a_mn, b_mn, out_fp32, accumulate);
  if (!tc::ensure_dynamic_smem((const void*)kernel, Tile<BN>::SMEM_BYTES)) return 1005;
  kernel<<<grid, kThreads, Tile<BN>::SMEM_BYTES, stream>>>(tmA, tmB, tmC, p);
  return (int)cudaGetLastError();
}

static int check_args(const void* A, const void* B, const void* C, const void* residual,
                      const void* bias, int N, long long lda, long long ldb, long long ldc, long long ldr, bool out_fp32,
                      bool accumulate) {
  // argument errors get codes of their own (1001..1008) so that they cannot be mistaken
  // for a CUDA error
  if ((lda % 8) || (ldb % 8) || (ldc % (out_fp32 ? 4 : 8)) || (N % 8)) return 1001;
  if (((uintptr_t)A & 15) || ((uintptr_t)B & 15) || ((uintptr_t)C & 15)) return 1002;
  if (residual && (out_fp32 || accumulate || (ldr % 8) || ((uintptr_t)residual & 15))) return 1001;
  if (bias && (out_fp32 || accumulate || ((uintptr_t)bias & 15))) return 1001;
  return 0;
}

}  // namespace gemm

extern "C" {

// C[M,N] (+)= op(A) x op(B), bf16 operands, fp32 accumulation.
//   a_mn_major = 0: A is [M, K] row-major (lda >= K); 1: A is stored [K, M] (lda >= M)
//   b_mn_major = 0: B is [N, K] row-major (ldb >= K); 1: B is stored [K, N] (ldb >= N)
//   out_fp32: C is fp32 instead of bf16; accumulate: add to the existing C
// Leading dimensions are in elements and must keep rows 16-byte aligned.
//   residual (optional, bf16 [M, N], leading dimension ldr): C = residual + A x B; only with a
//   bf16, non-accumulating C
//   bias (optional, bf16 [N], 16-byte aligned): added to every row; same condition
int bcom_gemm_bf16_bias(const void* A, const void* B, void* C, const void* residual,
                        const void* bias, int M, int N, int K, long long lda, long long ldb,
                        long long ldc, long long ldr, int a_mn_major, int b_mn_major, int out_fp32,
                        int accumulate, int max_ctas, void* stream) {
  using namespace gemm;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (const int rc = check_args(A, B, C, residual, bias, N, lda, ldb, ldc, ldr, out_fp32 != 0,
                                accumulate != 0))
    return rc;
  (void)cudaGetLastError();  // do not inherit an error left behind by an earlier call
  return launch<256>(A, B, C, residual, bias, M, N, K, lda, ldb, ldc, ldr, a_mn_major != 0,
                     b_mn_major != 0, out_fp32 != 0, accumulate != 0, 1, max_ctas,
                     (cudaStream_t)stream);
}

// The forms without a bias, and without a residual either, for C callers.
int bcom_gemm_bf16_ex(const void* A, const void* B, void* C, const void* residual, int M, int N,
                      int K, long long lda, long long ldb, long long ldc, long long ldr,
                      int a_mn_major, int b_mn_major, int out_fp32, int accumulate, int max_ctas,
                      void* stream) {
  return bcom_gemm_bf16_bias(A, B, C, residual, nullptr, M, N, K, lda, ldb, ldc, ldr, a_mn_major,
                             b_mn_major, out_fp32, accumulate, max_ctas, stream);
}

// fp32 elements of workspace that bcom_gemm_bf16_split needs (0 for splits <= 1)
long long bcom_gemm_split_workspace(int M, int N, int splits) {
  return splits <= 1 ? 0 : (long long)splits * ((M + 127) / 128 * 128) * N;
}

// The same product on 128x128 tiles with K shared out among `splits` (1..8) work items per tile,
// for shapes with few tiles: 128 tokens through a 4096 x 4096 projection are 16 tiles of 128x256,
// i.e. 16 of 148 SMs fetching the weights in 64 serial k-blocks each.  splits > 1: the partial
// tiles go to `workspace` (private to the call until it has run, 16-byte aligned) and a second
// kernel adds them up in ascending order.  `splits` must not exceed the 64-wide k-blocks.
int bcom_gemm_bf16_split(const void* A, const void* B, void* C, const void* residual,
                         const void* bias, int M, int N, int K, long long lda, long long ldb, long long ldc, long long ldr,
                         int a_mn_major, int b_mn_major, int out_fp32, int accumulate, int splits,
                         void* workspace, void* stream) {
  using namespace gemm;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (const int rc = check_args(A, B, C, residual, bias, N, lda, ldb, ldc, ldr, out_fp32 != 0,
                                accumulate != 0))
    return rc;
  if (splits < 1 || splits > 8 || splits > (K + BK - 1) / BK) return (int)cudaErrorInvalidValue;
  (void)cudaGetLastError();
  cudaStream_t st = (cudaStream_t)stream;
  if (splits == 1)
    return launch<128>(A, B, C, residual, bias, M, N, K, lda, ldb, ldc, ldr, a_mn_major != 0,
                       b_mn_major != 0, out_fp32 != 0, accumulate != 0, 1, 0, st);
  if (!workspace || ((uintptr_t)workspace & 15)) return 1002;
  const int rc = launch<128>(A, B, workspace, nullptr, nullptr, M, N, K, lda, ldb, N, 0, a_mn_major != 0,
                             b_mn_major != 0, true, false, splits, 0, st);
  if (rc) return rc;
  const long long stride = (long long)((M + BM - 1) / BM * BM) * N;
  const long long work = ((long long)M * (N / 4) + 255) / 256;
  const int grid = (int)(work < 4LL * sm_count() ? work : 4LL * sm_count());
  const float* ws = (const float*)workspace;
  const __nv_bfloat16* R = (const __nv_bfloat16*)residual;
  const __nv_bfloat16* b = (const __nv_bfloat16*)bias;
  if (out_fp32) {
    if (accumulate)
      split_sum_kernel<true, true><<<grid, 256, 0, st>>>(ws, splits, stride, C, R, b, ldc, ldr, M,
                                                        N);
    else
      split_sum_kernel<true, false><<<grid, 256, 0, st>>>(ws, splits, stride, C, R, b, ldc, ldr, M,
                                                        N);
  } else {
    if (accumulate)
      split_sum_kernel<false, true><<<grid, 256, 0, st>>>(ws, splits, stride, C, R, b, ldc, ldr, M,
                                                        N);
    else
      split_sum_kernel<false, false><<<grid, 256, 0, st>>>(ws, splits, stride, C, R, b, ldc, ldr, M,
                                                        N);
  }
  return (int)cudaGetLastError();
}

int bcom_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                   long long ldb, long long ldc, int a_mn_major, int b_mn_major, int out_fp32,
                   int accumulate, int max_ctas, void* stream) {
  return bcom_gemm_bf16_ex(A, B, C, nullptr, M, N, K, lda, ldb, ldc, 0, a_mn_major, b_mn_major,
                           out_fp32, accumulate, max_ctas, stream);
}

// Copies the 4-word status record {code, cta, thread, -}; clears it when `clear` != 0.
int bcom_gemm_status(unsigned int out[4], int clear) {
  cudaError_t err = cudaMemcpyFromSymbol(out, gemm::g_status, sizeof(unsigned int) * 4);
  if (err == cudaSuccess && clear) {
    unsigned int zero[4] = {0, 0, 0, 0};
    err = cudaMemcpyToSymbol(gemm::g_status, zero, sizeof(zero));
  }
  return (int)err;
}

}  // extern "C"
