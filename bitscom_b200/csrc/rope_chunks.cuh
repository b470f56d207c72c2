// How a RoPE call over many tokens is divided into launches, as a host function so that the CPU
// test tier can check it.
//
// The kernel counts tokens in 32 bits and steps beyond its last token by up to twice the grid's
// rows (below 2^17) before it stops, so a launch takes at most 2^30 tokens.
#pragma once

namespace ew {

struct RopeChunk {
  long long first;  // first token
  int tokens;
  int position;  // of the first token in its sequence
};

inline RopeChunk rope_chunk(long long tokens, int seq, long long first) {
  const long long rest = tokens - first, most = 1LL << 30;
  return RopeChunk{first, (int)(rest < most ? rest : most), (int)(first % seq)};
}

}  // namespace ew
