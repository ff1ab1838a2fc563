// Division of a bin row's slot by the bins per row and per layer (coarse_cluster.cuh) through a
// product with 2^32 / d, rounded up. Plain C++ as well as device code, so that a host test can
// check where it is exact.
#pragma once
#include <cstdint>

#ifndef CFDG_HD
#ifdef __CUDACC__
#define CFDG_HD __host__ __device__ __forceinline__
#else
#define CFDG_HD inline
#endif
#endif

namespace cfdg {

// 2^32 / d, rounded up (unused for d == 1).
CFDG_HD unsigned bin_magic(int d) { return (unsigned)((((uint64_t)1 << 32) + d - 1) / d); }

// q / d for m = bin_magic(d), exact for q < rows with rows d <= 2^32: m d exceeds 2^32 by less than
// d, which adds less than 1 / d to the quotient.
CFDG_HD int bin_div(int q, unsigned m, int d) {
#ifdef __CUDA_ARCH__
  return d == 1 ? q : (int)__umulhi((unsigned)q, m);
#else
  return d == 1 ? q : (int)((uint64_t)(unsigned)q * m >> 32);
#endif
}

// Whether the slots below `rows` of a level with nbh slots per bin row and nby bin rows per layer
// are taken apart exactly: by nbh, then the quotient by nby.
CFDG_HD bool bin_div_exact(uint64_t rows, int nbh, int nby) {
  const uint64_t most = (uint64_t)1 << 32;
  return rows * nbh <= most && (rows + nbh - 1) / nbh * nby <= most;
}

}  // namespace cfdg
