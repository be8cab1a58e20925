// prefetch_plan.h — how many of its first weight blocks (128 rows x 64) a CTA of the few-token GEMM (gemm_skinny.cuh) starts on their
// way to L2 while the previous kernel of the stream still runs.  Plain C++.
#pragma once

namespace bshmem {
namespace skinny {

// Four, and up to 64 tokens half of a CTA's blocks where that is more (the ring is the limit): cold weights, us without / 2 / 3 / 4 / a ring of blocks: 8 tokens 2048 -> 2048 5.12 4.76 4.48 4.45 4.45; 16 tokens 4096 -> 4096 9.37
// 9.16 8.95 8.72 8.92; 16 tokens 3584 -> 8192 13.37 13.13 12.90 12.72 12.68; 96 tokens 4096 -> 4096 11.37 11.11 10.99 10.92 11.51; 128 tokens
// 3584 -> 8192 15.71 15.48 15.41 15.33 16.04.  Weights that are in L2 already cost something: 6.44 6.77 6.90 6.96 7.17 for the
// second of these, 3.99 4.05 4.07 4.07 4.05 for the first.  None
//  - above 128 tokens, where the product is longer than what is gained: 200 tokens 2048 -> 2048 9.40 (9.47 with four, 9.55 with a ring), 160 tokens
//    3584 -> 8192 15.98 (16.07, 16.48);
//  - where rows are not whole 128-byte lines, so that every block touches half as many lines again, unless a CTA has only a few blocks:
//    16 tokens 4104 -> 4096 9.60 (9.76, 10.13), 50 tokens 8200 -> 3592 15.24 (15.63, 15.63), both with eight blocks per CTA and more; 8 tokens
//    1504 -> 3000, six blocks, 5.53 (4.94, 4.87).
inline int prefetch_blocks(int tokens, long long row_bytes, int blocks_per_cta) {
  if (tokens > 128 || (row_bytes % 128 && blocks_per_cta >= 8)) return 0;
  return tokens <= 64 && blocks_per_cta / 2 > 4 ? blocks_per_cta / 2 : 4;
}

}  // namespace skinny
}  // namespace bshmem
