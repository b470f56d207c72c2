// Host check of the GEMM tile scheduler (csrc/gemm_schedule.cuh), built by
// tests/test_gemm_schedule.py with g++: for many (M, N) the tiles of the one-CTA kernel
// (128 x 256) and of the CTA-pair kernel (256 x 256) must cover every element of C exactly
// once, whatever the grouping along M does at the edges.
#include <cstdio>
#include <vector>

#define __host__
#define __device__
#include "attention_schedule.cuh"
#include "gemm_schedule.cuh"
#include "rope_chunks.cuh"

template <int BM, int BN>
static int check(int M, int N) {
  const int tiles_m = (M + BM - 1) / BM, tiles_n = (N + BN - 1) / BN;
  const int tiles = tiles_m * tiles_n;
  std::vector<unsigned char> hit((size_t)M * N, 0);
  for (int w = 0; w < tiles; ++w) {
    const gemm_sched::WorkItem wi = gemm_sched::work_item<BM, BN, 8>(tiles_m, tiles_n, w);
    if (wi.m0 % BM || wi.n0 % BN || wi.m0 < 0 || wi.n0 < 0) return 5;
    for (int r = wi.m0; r < wi.m0 + BM && r < M; ++r)
      for (int c = wi.n0; c < wi.n0 + BN && c < N; ++c)
        if (hit[(size_t)r * N + c]++) return 6;  // produced twice
  }
  for (unsigned char h : hit)
    if (h != 1) return 7;  // never produced
  return 0;
}

// The staging chunks of an epilogue warp.  It waits until at most its newest store is under way
// and then fills a chunk, while that store may still be reading another: over the tiles that each
// of `ctas` CTAs takes, no two stores in a row may use the same chunk.  `cols`: columns per chunk
// (64 bf16, 32 fp32).
template <int BN>
static int check_staging(int M, int N, int ctas, int cols) {
  const int tiles_m = (M + 127) / 128, tiles_n = (N + BN - 1) / BN;
  for (int cta = 0; cta < ctas; ++cta) {
    gemm_sched::StagingChunks chunks;
    int newest = -1;  // chunk that the newest store reads
    for (int w = cta; w < tiles_m * tiles_n; w += ctas) {
      const gemm_sched::WorkItem wi = gemm_sched::work_item<128, BN, 8>(tiles_m, tiles_n, w);
      for (int c = 0; c < BN / cols && wi.n0 + c * cols < N; ++c) {
        const int chunk = chunks.next();
        if (chunk < 0 || chunk > 1 || chunk == newest) return 10;
        newest = chunk;
      }
    }
  }
  return 0;
}

int main() {
  const int shapes[][2] = {{128, 256},  {4096, 4096}, {4096, 12288}, {200, 264},  {77, 8},
                           {1024, 1024}, {2048, 22016}, {8192, 4096}, {1152, 512}, {3000, 1000},
                           {256, 256},  {129, 257},   {9 * 128, 3 * 256}};
  int checked = 0;
  for (auto& s : shapes) {
    if (int rc = check<128, 256>(s[0], s[1])) {
      std::fprintf(stderr, "128x256 tiles: M=%d N=%d: code %d\n", s[0], s[1], rc);
      return 1;
    }
    if (int rc = check<256, 256>(s[0], s[1])) {
      std::fprintf(stderr, "256x256 tiles: M=%d N=%d: code %d\n", s[0], s[1], rc);
      return 1;
    }
    checked += 2;
  }
  for (int N : {8, 64, 96, 192, 264, 320, 352, 960, 1032, 1600, 1728, 4096})
    for (int cols : {64, 32})
      for (int ctas : {1, 2, 5}) {
        int rc = check_staging<256>(3000, N, ctas, cols);
        if (!rc) rc = check_staging<128>(3000, N, ctas, cols);
        if (rc) {
          std::fprintf(stderr, "staging: N=%d, %d columns a chunk: code %d\n", N, cols, rc);
          return 1;
        }
      }
  // persistent attention: every item once, a CTA's items end at the first index past the end
  for (int ctas = 1; ctas <= 150; ctas += 7)
    for (int total = ctas; total <= 1100; total += 37) {
      std::vector<int> taken(total, 0);
      for (int c = 0; c < ctas; ++c)
        for (int j = 0; attn_sched::item_index(c, ctas, j) < total; ++j)
          ++taken[attn_sched::item_index(c, ctas, j)];
      for (int t : taken)
        if (t != 1) return 9;
    }
  // RoPE launches: every token once and in order at its own position, and a thread that steps past
  // the last token by two rows of the largest grid stays within 32 bits
  for (long long tokens : {1LL, 4096LL, 1LL << 30, (1LL << 30) + 1, (1LL << 31) - 1, (1LL << 31) + 5,
                           7000000001LL})
    for (int seq : {1, 127, 2048, 1 << 30, 2147483647}) {
      long long first = 0;
      while (first < tokens) {
        const ew::RopeChunk part = ew::rope_chunk(tokens, seq, first);
        if (part.first != first || part.tokens < 1 || part.position != first % seq) return 11;
        if ((long long)part.tokens + 4 * 65535 > 2147483647LL) return 12;
        if ((long long)part.tokens + part.position > 4294967295LL) return 13;
        first += part.tokens;
      }
      if (first != tokens) return 14;
    }
  // shares of K: in order, without gaps, none empty
  for (int kb = 1; kb <= 200; ++kb)
    for (int splits = 1; splits <= 8 && splits <= kb; ++splits)
      for (int i = 0; i < splits; ++i) {
        const int from = gemm_sched::split_begin(kb, splits, i);
        const int to = gemm_sched::split_begin(kb, splits, i + 1);
        if (from >= to || (i == 0 && from != 0) || (i + 1 == splits && to != kb)) return 8;
      }
  std::printf("ok: %d schedules cover their outputs exactly once\n", checked);
  return 0;
}
