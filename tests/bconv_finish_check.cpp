// CPU check of how the base conversion finishes an output (bconv_mma_finish of cerium_b200/csrc/bconv_mma.cuh, built here
// with the CUDA stand-ins): from the byte-plane sums of sum_k g_k y_k, g_k < q and y_k < 2^8, the exact residue, for every
// class of q, up to the largest number of inputs and the largest sum that these allow, where it passes 64 bits.
// TEST INFRASTRUCTURE ONLY.  Prints "OK" or a line starting with "FAIL".
#include <cstdio>
#include <random>
#include <vector>

#include "bconv_mma.cuh"

using namespace cerium;
typedef unsigned __int128 u128;

static std::mt19937_64 rng(2024);

// kind 0: every factor q - 1 and every byte 255; 1: factors at random, bytes 255; 2: both at random; 3: all zero
template <typename W, int kFinish>
static bool check(uint64_t q, int inputs, int kind, uint64_t sub, uint64_t limit) {
  const int terms = inputs * (int)sizeof(W);
  uint32_t c[sizeof(W)] = {};
  u128 x = 0;
  for (int k = 0; k < terms; k++) {
    const uint64_t g = kind == 0 ? q - 1 : kind == 3 ? 0 : rng() % q;
    const uint32_t y = kind == 2 ? (uint32_t)(rng() & 255) : kind == 3 ? 0 : 255;
    for (unsigned m = 0; m < sizeof(W); m++) c[m] += (uint32_t)(g >> (8 * m) & 255) * y;
    x += (u128)g * y;
  }
  const BconvMmaOut<W> o = bconv_mma_constants<W>(q, sub);
  const uint64_t got = bconv_mma_finish<kFinish>(c, o), want = (uint64_t)((x + q - sub) % q);
  if (got % q == want && got < limit) return true;
  std::printf("FAIL word %d finish %d q %llu inputs %d kind %d: %llu, want %llu\n", (int)sizeof(W) * 8, kFinish,
              (unsigned long long)q, inputs, kind, (unsigned long long)got, (unsigned long long)want);
  return false;
}

template <typename W, int kFinish>
static bool sweep(const std::vector<uint64_t>& moduli, const std::vector<int>& inputs) {
  for (uint64_t q : moduli)
    for (int n : inputs)
      for (int kind = 0; kind < 4; kind++)
        for (int rep = 0; rep < (kind == 1 || kind == 2 ? 200 : 1); rep++)
          for (uint64_t sub : {(uint64_t)0, (uint64_t)1, q / 2, q - 1}) {
            if (kFinish == kMmaLazy && sub != 0) continue;
            if (!check<W, kFinish>(q, n, kind, sub, kFinish <= kMmaLazyAdd ? 4 * q : q)) return false;
          }
  return true;
}

int main() {
  // edges of the classes; the smallest modulus that a transform of 2^16 points has is 786433
  const uint64_t one = 1;
  const std::vector<uint64_t> wide = {(one << 60) - 1, (one << 50) - 27, (one << 48) + 21, (one << 48) + 1};
  std::vector<uint64_t> all = wide;
  for (uint64_t q : {(one << 48) - 59, (one << 48) - 1, (one << 47) + 5, (one << 41) + 27, (one << 40) + 15, (one << 40) - 87, (one << 30) + 3, (one << 20) - 3, (uint64_t)786433}) all.push_back(q);
  const std::vector<uint64_t> small = {(one << 30) - 35, (one << 28) - 57, (one << 20) + 7, 786433};
  const bool ok = sweep<uint64_t, kMmaGeneral>(all, {1, 2, 5, 31, kMmaPairInputs}) &&
                  sweep<uint64_t, kMmaBig>(all, {kMmaPairInputs + 1, 48, kMmaMaxInputs}) &&
                  sweep<uint64_t, kMmaLazy>(wide, {1, 5, kMmaPairInputs}) &&
                  sweep<uint64_t, kMmaLazyAdd>(wide, {1, 5, kMmaPairInputs}) &&
                  sweep<uint32_t, kMmaGeneral>(small, {1, 13, kMmaMaxInputs}) &&
                  sweep<uint32_t, kMmaLazy>(small, {1, 13, kMmaMaxInputs}) &&
                  sweep<uint32_t, kMmaLazyAdd>(small, {1, 13, kMmaMaxInputs});
  if (ok) std::printf("OK\n");
  return ok ? 0 : 1;
}
