// Work distribution of the persistent attention kernels, as a host/device function so that the
// CPU test tier can check that every item is taken exactly once.
//
// Items are numbered by decreasing work.  Round j hands one to each of `ctas` CTAs, forwards in
// even rounds and backwards in odd ones: causal attention's work falls linearly over the items,
// so two neighbouring rounds add up to the same for every CTA (1024 items of 16 .. 1 blocks over
// 148 CTAs: 58 to 60 blocks each; always forwards: 51 to 67).
#pragma once

namespace attn_sched {

__host__ __device__ inline int item_index(int cta, int ctas, int j) {
  return j * ctas + ((j & 1) ? ctas - 1 - cta : cta);
}

}  // namespace attn_sched
