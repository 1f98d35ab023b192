// From how many iterations on a run of a strategy repays the spatial sort of
// its points.
//
// The sort costs about what three to five plain iterations do; box pruning
// takes off an iteration what the distances to most of the k clusters take, and
// in the three-stage strategy what the sums of points in no order cost besides.
// Measured as whole loops of 8 and of 30 iterations, plain and sorted, over
// blobs of n = 2^20 to 2^24, d = 2, 4 and 8, k = 4, 10, 20 and 32; the iterations at
// which the two are level, for d = 2, 4, 8 ("-": not below 100):
//   single-stage  n = 2^20: k = 4 42 32 -,  k = 10 15 45 40, k = 20 42 22 14, k = 32 16 14 9
//                 n = 2^21: k = 4 61 -  -,  k = 10 21 31 32, k = 20 20 15 10, k = 32 11 8 6
//                 n = 2^23: k = 4 -  68 -,  k = 10 31 19 24, k = 20 11 8 9,   k = 32 6 5 5
//   three-stage   n = 2^20: k = 4 20 22 23, k = 10 14 7 20,  k = 20 6 8 9,    k = 32 6 7 7
//                 n = 2^22: k = 4 -  -  -,  k = 10 15 12 43, k = 20 7 8 8,    k = 32 6 6 5
//                 n = 2^24: k = 4 -  -  -,  k = 10 32 23 42, k = 20 9 8 8,    k = 32 6 5 5
// Of the products of iterations and clusters these are the lines; over all
// loops measured (8 to 50 iterations) the chosen one is 0.4 % slower than the
// faster of the two on average.
#pragma once

#include <cstdint>

namespace Clustering {

inline bool single_stage_spatial_pays(uint64_t n, uint32_t k, uint32_t iterations) {
    const uint64_t line = n >= (1u << 22) ? 180 : n >= (5u << 18) ? 240 : 320;
    return k > 2 && (uint64_t)iterations * (k - 2) >= line;
}

inline bool three_stage_spatial_pays(uint64_t n, uint32_t k, uint32_t iterations) {
    if (n >= (1u << 22)) return k > 4 && (uint64_t)iterations * (k - 4) >= 110;
    return k > 2 && (uint64_t)iterations * (k - 2) >= 96;
}

}  // namespace Clustering
