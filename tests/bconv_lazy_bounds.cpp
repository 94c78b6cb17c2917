// CPU check of what the base conversion leaves for a transform (bconv_mma_finish of cerium_b200/csrc/bconv_mma.cuh, built here with
// the CUDA stand-ins): below kFpRaisedIn / 1024 q without a rounding term and kFpLoweredIn / 1024 q with one, from which the
// double-precision butterflies count their bounds, for the largest sums.  TEST INFRASTRUCTURE ONLY.  Prints "OK" or "FAIL ...".
#include <cstdio>
#include <random>

#include "bconv_mma.cuh"

using namespace cerium;

template <int kFinish>
static bool check(uint64_t q, int inputs, uint64_t sub, std::mt19937_64& rng, int kind, uint64_t bound) {
  uint32_t c[8] = {};
  for (int k = 0; k < inputs * 8; k++) {
    const uint64_t g = kind == 0 ? q - 1 : rng() % q;
    const uint32_t y = kind == 2 ? (uint32_t)(rng() & 255) : 255;
    for (int m = 0; m < 8; m++) c[m] += (uint32_t)(g >> (8 * m) & 255) * y;
  }
  const uint64_t got = bconv_mma_finish<kFinish>(c, bconv_mma_constants<uint64_t>(q, sub));
  if ((unsigned __int128)got * 1024 <= (unsigned __int128)bound * q) return true;
  std::printf("FAIL finish %d q %llu inputs %d kind %d: %llu\n", kFinish, (unsigned long long)q, inputs, kind, (unsigned long long)got);
  return false;
}

int main() {
  std::mt19937_64 rng(7);
  const uint64_t one = 1;
  for (uint64_t q : {(one << 48) + 1, (one << 48) + 21, (one << 49) + 9, (one << 50) - 27})  // wide, and on doubles
    for (int n : {1, 5, 13, kMmaPairInputs})
      for (int rep = 0; rep < 2000; rep++) {
        const int kind = rep == 0 ? 0 : 1 + rep % 2;
        if (!check<kMmaLazy>(q, n, 0, rng, kind, kFpRaisedIn)) return 1;
        for (uint64_t sub : {one, q / 2, q - 1})
          if (!check<kMmaLazyAdd>(q, n, sub, rng, kind, kFpLoweredIn)) return 1;
      }
  std::printf("OK\n");
}
