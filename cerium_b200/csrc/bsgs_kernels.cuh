// Kernels of the baby-step / giant-step multiply-accumulate (the linear-transform building block of
// bootstrapping): the plaintext multiply-accumulate of a group of giant steps in one pass, and the
// sum of several polynomials read through (different) Galois automorphisms.
//
// The reference lowers BsgsMultiplyAccumulate to one MuP and one Add instruction per diagonal and
// polynomial inside a generated kernel group (cerium/compiler/backend/compiler.cc:2495-2522) and one
// rotation + Add per giant step (:2562-2590).  Here a thread keeps the sums of up to kBsgsGroup giant
// steps in registers while it walks the baby steps, so the rotated copies of the input
// are read once per group and every diagonal exactly once; one reduction per output.
#pragma once
#include "ewise_kernels.cuh"
#include "ntt_kernels.cuh"

namespace cerium {

constexpr int kBsgsMaxBaby = 16;   // baby steps (rotated copies of the input)
constexpr int kBsgsGroup = 8;      // giant steps whose inner sums one launch may produce
constexpr int kBsgsMaxGiant = 32;  // giant steps of one multiply-accumulate

template <typename W>
struct PtMacArgs {
  const W* src0[kBsgsMaxBaby];            // baby step j, polynomial 0: [limbs][N]
  const W* src1[kBsgsMaxBaby];            // baby step j, polynomial 1
  const W* pt[kBsgsGroup][kBsgsMaxBaby];  // diagonal of (giant step of the group, baby step); null = absent
  W* out0[kBsgsGroup];                    // inner sum of the group's giant step, polynomial 0
  W* out1[kBsgsGroup];
  int g;                                  // baby steps
  uint8_t prime[kEwMaxLimbs];
};

// One thread owns kPtMacWords consecutive words of a limb: one 8-byte access per operand for both word
// sizes (a warp still moves whole 256-byte runs).  Wider accesses would double the accumulator
// registers: with four giant steps, two polynomials and two-word sums that costs the occupancy a
// streaming kernel lives on (136 registers and one CTA per SM when measured with 16-byte accesses).
template <typename W>
struct PtMacLanes {
  static constexpr int kWords = 8 / sizeof(W);
};
template <typename W>
__device__ __forceinline__ void ptmac_load(const W* p, W (&v)[PtMacLanes<W>::kWords]) {
  if constexpr (sizeof(W) == 8) {
    v[0] = *p;
  } else {
    const uint2 t = *reinterpret_cast<const uint2*>(p);
    v[0] = t.x;
    v[1] = t.y;
  }
}
template <typename W>
__device__ __forceinline__ void ptmac_store(W* p, const W (&v)[PtMacLanes<W>::kWords]) {
  if constexpr (sizeof(W) == 8) {
    *p = v[0];
  } else {
    *reinterpret_cast<uint2*>(p) = make_uint2(v[0], v[1]);
  }
}

// Sum of products of two residues for one word.  General: two words with carries.  Pieces (64-bit words, primes
// below 2^56): the factors as 28-bit pieces, y = y0 + y1 2^28, so that a product is four wide multiply-adds into three
// column sums and no carry anywhere (16 products: the middle column stays below 2^61): 16 cycles of the integer
// multiply pipe against ~28 and twice the instructions.  Fp (every prime of the launch below 2^50): reduced products of
// doubles (Arith::product, below 7/8 q), eight of them on a reduced sum; one register pair a sum, so a launch serves eight giant
// steps and the rotated inputs are read once where they were read for every four.
enum : int { kPtGeneral = 0, kPtPieces = 1, kPtFp = 2 };
template <typename W, int kKind>
struct PtMacSum {
  static constexpr int kTerms = 1 << 30;  // on a reduced sum
  using Operand = W;
  struct Prime {
    __device__ __forceinline__ explicit Prime(const PrimeConst<W>&) {}
  };
  static __device__ __forceinline__ Operand operand(W x) { return x; }
  Acc2<W> acc;
  __device__ __forceinline__ void clear() { acc.clear(); }
  __device__ __forceinline__ void mad(const Operand& a, const Operand& b, const Prime&) { acc.mad(a, b); }
  __device__ __forceinline__ void reduce(const Prime&) {}
  __device__ __forceinline__ W finish(const Prime&, const PrimeConst<W>& pc) const { return barrett2<W>(acc.hi(), acc.lo(), pc); }
};
template <>
struct PtMacSum<uint64_t, kPtFp> {
  static constexpr int kTerms = 8;
  using Operand = double;
  using Prime = Arith<uint64_t, kArithFp>;
  static __device__ __forceinline__ Operand operand(uint64_t x) { return fp_from_u64(x); }
  double s;
  __device__ __forceinline__ void clear() { s = 0.0; }
  __device__ __forceinline__ void mad(double a, double b, const Prime& p) { s = __dadd_rn(s, p.product(a, b)); }
  __device__ __forceinline__ void reduce(const Prime& p) { s = fp_reduce(s, p.qinv, p.nq); }
  __device__ __forceinline__ uint64_t finish(const Prime& p, const PrimeConst<uint64_t>&) const {
    return p.canonical(fp_reduce(s, p.qinv, p.nq));
  }
};
template <>
struct PtMacSum<uint64_t, kPtPieces> {
  static constexpr int kTerms = 1 << 30;
  using Prime = PtMacSum<uint64_t, kPtGeneral>::Prime;
  struct Operand {
    uint32_t lo, hi;
  };
  static __device__ __forceinline__ Operand operand(uint64_t x) {
    return {(uint32_t)x & 0xfffffffu, (uint32_t)(x >> 28)};
  }
  uint64_t c0, c1, c2;
  __device__ __forceinline__ void clear() { c0 = c1 = c2 = 0; }
  __device__ __forceinline__ void reduce(const Prime&) {}
  __device__ __forceinline__ void mad(const Operand& a, const Operand& b, const Prime&) {
    c0 += (uint64_t)a.lo * b.lo;
    c1 += (uint64_t)a.lo * b.hi;
    c1 += (uint64_t)a.hi * b.lo;
    c2 += (uint64_t)a.hi * b.hi;
  }
  // c0 + c1 2^28 + c2 2^56
  __device__ __forceinline__ uint64_t finish(const Prime&, const PrimeConst<uint64_t>& pc) const {
    const uint64_t m = c1 + (c0 >> 28);             // weight 2^28
    const uint64_t h = c2 + (m >> 28);              // weight 2^56
    const uint64_t lo = (c0 & 0xfffffffu) | (m & 0xfffffffu) << 28 | h << 56;
    return barrett2<uint64_t>(h >> 8, lo, pc);
  }
};

// out[i][p] = sum_j pt[i][j] * src_p[j] for the GI giant steps of a group.  Streams 2 + GI words per baby step and word
// position: bound by memory (8 baby and 4 giant steps at 35 limbs are 1.0 GB, 8 and 8 in one launch 1.8).  A thread copies the operands of
// the next steps into shared memory of its own (cp.async, three steps on their way): 60 to 110 KB of an SM in flight, where one step
// ahead in registers was 25 KB.  8 and 4 steps, 8 and 8 steps at 35 limbs, that -> this: 50-bit primes 318 -> 166 us, 629 -> 282 (one
// launch for two); pieces 312 -> 239, 627 -> 482; general 324 -> 243, 652 -> 490; 32-bit words 122 -> 85, 248 -> 170.  An absent
// diagonal costs a predicate and no branch.
// grid = (N / (kThreads * kWords), limbs), block = kThreads = ptmac_threads(GI).
constexpr int kPtMacStages = 4;
constexpr int ptmac_threads(int gi) { return gi > 4 ? 128 : 256; }
template <typename W, int GI, int kKind>
__global__ void __launch_bounds__(ptmac_threads(GI), GI > 4 ? 4 : 3) pt_mac_kernel(const PtMacArgs<W> a, const PrimeConst<W>* __restrict__ pcs) {
  using Sum = PtMacSum<W, kKind>;
  constexpr int kWords = PtMacLanes<W>::kWords, kThreads = ptmac_threads(GI);
  __shared__ __align__(16) W ring[kPtMacStages][2 + GI][kThreads * kWords];
  grid_dependency_launch();
  grid_dependency_wait();
  const int b = blockIdx.y, mine = threadIdx.x * kWords;
  const PrimeConst<W> pc = pcs[a.prime[b]];
  const typename Sum::Prime prime(pc);
  const size_t off = (size_t)b * kN + (size_t)(blockIdx.x * kThreads + threadIdx.x) * kWords;
  Sum acc[GI][2][kWords];
#pragma unroll
  for (int i = 0; i < GI; i++)
#pragma unroll
    for (int l = 0; l < kWords; l++) {
      acc[i][0][l].clear();
      acc[i][1][l].clear();
    }
  auto fetch = [&](int j) {
    if (j < a.g) {
      auto* to = ring[j % kPtMacStages];
      copy_async<8>(&to[0][mine], a.src0[j] + off);
      copy_async<8>(&to[1][mine], a.src1[j] + off);
#pragma unroll
      for (int i = 0; i < GI; i++)
        if (a.pt[i][j] != nullptr) copy_async<8>(&to[2 + i][mine], a.pt[i][j] + off);
    }
    copy_async_commit();
  };
#pragma unroll
  for (int j = 0; j < kPtMacStages - 1; j++) fetch(j);
#pragma unroll 1
  for (int j = 0; j < a.g; j++) {
    copy_async_wait<kPtMacStages - 2>();
    const auto* from = ring[j % kPtMacStages];
    typename Sum::Operand so[2][kWords], po[GI][kWords];
#pragma unroll
    for (int k = 0; k < 2 + GI; k++) {
      W v[kWords];
      ptmac_load<W>(&from[k][mine], v);
#pragma unroll
      for (int l = 0; l < kWords; l++) {
        if (k < 2) so[k < 2 ? k : 0][l] = Sum::operand(v[l]);
        else po[k < 2 ? 0 : k - 2][l] = Sum::operand(a.pt[k < 2 ? 0 : k - 2][j] != nullptr ? v[l] : (W)0);
      }
    }
    fetch(j + kPtMacStages - 1);  // into the step before this one
    const bool full = j != 0 && j % Sum::kTerms == 0;
#pragma unroll
    for (int i = 0; i < GI; i++)
#pragma unroll
      for (int l = 0; l < kWords; l++)
#pragma unroll
        for (int p = 0; p < 2; p++) {
          if (full) acc[i][p][l].reduce(prime);
          acc[i][p][l].mad(so[p][l], po[i][l], prime);
        }
  }
#pragma unroll
  for (int i = 0; i < GI; i++) {
    W o0[kWords], o1[kWords];
#pragma unroll
    for (int l = 0; l < kWords; l++) {
      o0[l] = acc[i][0][l].finish(prime, pc);
      o1[l] = acc[i][1][l].finish(prime, pc);
    }
    ptmac_store<W>(a.out0[i] + off, o0);
    ptmac_store<W>(a.out1[i] + off, o1);
  }
}

template <typename W>
struct AutoSumArgs {
  const W* in[kBsgsMaxGiant];   // [limbs][N] each
  uint32_t elt[kBsgsMaxGiant];  // Galois element the polynomial is read through (1 = as it is)
  int count;
  W* out;                       // [limbs][N]; must not overlap an input
  uint8_t prime[kEwMaxLimbs];
};

// out[b][i] = sum_k in_k[b][pi_k(i)] mod q.  grid = (N / 256, limbs).
template <typename W>
__global__ void __launch_bounds__(kEwThreads) automorph_sum_kernel(const AutoSumArgs<W> a, const PrimeConst<W>* __restrict__ pcs) {
  grid_dependency_launch();
  grid_dependency_wait();
  const int b = blockIdx.y;
  const W q = pcs[a.prime[b]].q;
  const uint32_t i = blockIdx.x * kEwThreads + threadIdx.x;
  W s = 0;
  for (int k = 0; k < a.count; k++) {
    const uint32_t src = a.elt[k] == 1u ? i : galois_source_index(i, a.elt[k]);
    s = add_mod<W>(s, a.in[k][(size_t)b * kN + src], q);
  }
  a.out[(size_t)b * kN + i] = s;
}

}  // namespace cerium
