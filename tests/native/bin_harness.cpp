// Test harness (tests only): takes the slots of a bin level apart as the coarse levels' kernels do
// (cfd-craft_gb300/csrc/bin_div.hpp) and counts the wrong quotients.
#include <cstdint>

#include "bin_div.hpp"

using namespace cfdg;

extern "C" int bin_exact(int64_t rows, int nbh, int nby) { return bin_div_exact((uint64_t)rows, nbh, nby); }

extern "C" int64_t bin_scan(int64_t rows, int nbh, int nby) {
  const unsigned mh = bin_magic(nbh), my = bin_magic(nby);
  int64_t wrong = 0;
  for (int64_t q = 0; q < rows; ++q) {
    const int R = bin_div((int)q, mh, nbh);
    wrong += R != q / nbh || bin_div(R, my, nby) != q / nbh / nby;
  }
  return wrong;
}
