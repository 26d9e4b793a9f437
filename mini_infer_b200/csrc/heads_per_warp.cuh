// How many heads of a token a warp takes in the kernels that norm, rotate and store them (rope_norm.cu, qk_prepare.cu).
#pragma once

#include "common.cuh"

// One while all heads of a step are about a wave of warps (148 SMs of 64), so that they start at once; above, warps that take
// several share a token's angles and its place in the cache.  us with 1, 2 and 4, heads of 128, kernels of rope_norm.cu,
// qk_norm_rope_store and qk_bias_norm_store (which has no values of its own here: 20 and 40 heads a token):
//   tokens x heads      3072 (64 x 48)   6144 (256 x 24)  9216 (384 x 24)  12288 (512 x 24)  18432 (768 x 24)  49152 (2048 x 24)
//   rope_norm          3.5  4.0  5.0     4.3  4.5  5.2    5.5  4.6  5.4    6.6  5.9  5.7     9.1  7.2  7.6    21.2  15.7  14.4
//   qk_norm_rope       3.9  4.0  5.1     4.6  5.2  6.2    5.7  6.2  6.8    6.9  6.3  7.9     9.4  7.9  8.1    21.8  16.7  15.2
//   qk_bias_norm       3.0  3.1  4.3     3.4  4.2  4.1    3.9  4.8  5.5    4.5  4.9  5.5     5.9  5.4  6.6    12.8  11.2  10.8
static inline int heads_per_warp(long long heads) { return heads <= 10240 ? 1 : heads < 24576 ? 2 : 4; }
