// Fast base conversion between RNS bases driven by device-resident tables (the reference launcher's arguments);
// conversions whose primes the host knows run on the tensor cores (bconv_mma.cuh).
//
// Replaces convert<I,O> and its launcher (cerium/compiler/backend/kernels/fhe_bconv.cuh:98-151,
// cerium/compiler/backend/kernels/function.cuh:61-122).
//
//   out_j[c] = ( sum_i x_i[c] * F[j][i] ) mod p_j,         c = 0..N-1
//
// One thread owns one coefficient: it reads the I input residues once (coalesced across the
// warp), keeps them in registers or in its own shared-memory column, and streams over the O output
// primes with the factor matrix and the per-output constants broadcast from shared memory.  Sums are
// reduced once per output (primes below 2^60 leave room for 256 terms), instead of the reference's
// trims at i = 15, 30.
#pragma once
#include "modarith.cuh"

namespace cerium {

// 160 threads: with the kernel's ~70 registers five CTAs fit an SM
constexpr int kBconvThreads = 160;
constexpr int kBconvBlocks = (kN + kBconvThreads - 1) / kBconvThreads;  // the last block is partial
constexpr int kBconvRegInputs = 8;

template <typename W>
struct BconvDesc {
  const W* in;             // I limbs, coefficient form, one after another
  W* out;                  // O limbs
  int I;
  int O;
};

// Per-output constants staged in shared memory next to the factor matrix, so the output loop
// has no dependent global loads.
template <typename W>
struct BconvOut {
  W q, q2, mu_hi, mu_lo;
};

// Generic path (32-bit words, or more than 8 inputs): two-word accumulator, one Barrett
// reduction per output; inputs in registers (kRegI > 0) or in the thread's shared-memory column.
template <typename W, int kRegI>
__device__ __forceinline__ void bconv_body(const BconvDesc<W>& d, const W* sfac, const BconvOut<W>* sout, W* scol, int coeff) {
  const int tid = threadIdx.x;
  const int I = kRegI > 0 ? kRegI : d.I, O = d.O;  // kRegI > 0: exact number of inputs
  W y[kRegI > 0 ? kRegI : 1];
  if (kRegI > 0) {
#pragma unroll
    for (int i = 0; i < kRegI; i++) y[i] = d.in[(size_t)i * kN + coeff];
  } else {
    for (int i = 0; i < I; i++) scol[i * kBconvThreads + tid] = d.in[(size_t)i * kN + coeff];
  }
#pragma unroll 2
  for (int j = 0; j < O; j++) {
    const W* f = sfac + j * I;
    W acc_hi, acc_lo;
    if (sizeof(W) == 4 && kRegI > 0) {
      // 32-bit words, at most 8 terms below 2^60 each: the sum fits one 64-bit register, so a
      // multiply-accumulate is a single wide multiply-add
      uint64_t a64 = 0;
#pragma unroll
      for (int i = 0; i < kRegI; i++) a64 += (uint64_t)y[i] * (uint64_t)f[i];
      acc_hi = (W)(a64 >> 32);
      acc_lo = (W)a64;
    } else {
      Acc2<W> acc;
      acc.clear();
      if (kRegI > 0) {
#pragma unroll
        for (int i = 0; i < kRegI; i++) acc.mad(y[i], f[i]);
      } else {
        for (int i = 0; i < I; i++) acc.mad(scol[i * kBconvThreads + tid], f[i]);
      }
      acc_hi = acc.hi();
      acc_lo = acc.lo();
    }
    const BconvOut<W> o = sout[j];
    PrimeConst<W> pc;
    pc.q = o.q;
    pc.q2 = o.q2;
    pc.mu_hi = o.mu_hi;
    pc.mu_lo = o.mu_lo;
    W r = barrett2<W>(acc_hi, acc_lo, pc);
    d.out[(size_t)j * kN + coeff] = r;
  }
}

// 32-bit words, 9 to 32 inputs (the digits of the reference's 28-bit parameter sets hold 10 to 28 limbs): one
// coefficient per thread, every input in a register, the factor rows padded with zeros to kP = a multiple of
// four words and read as 16-byte vectors (one shared-memory load per four terms, the same address in every
// lane).  Residues and factors are below 2^30 (the widest primes a 32-bit context takes), a product is below
// 2^60, so sixteen of them fit one 64-bit sum: a multiply-accumulate is one wide multiply-add, and an output
// takes one Barrett reduction (two and an addition beyond sixteen inputs) - against a two-word accumulator
// with carries and a shared-memory column of inputs in the generic path.  Like the path for at most eight
// inputs, this one takes canonical residues.
template <int kP>
__device__ __forceinline__ void bconv_body_wide32(const BconvDesc<uint32_t>& d, const uint32_t* sfac, const BconvOut<uint32_t>* sout, int coeff) {
  static_assert(kP % 4 == 0 && kP > 8 && kP <= 32, "padded input count");
  uint32_t y[kP];
#pragma unroll
  for (int i = 0; i < kP; i++) y[i] = i < d.I ? d.in[(size_t)i * kN + coeff] : 0u;
  const int O = d.O;
#pragma unroll 2
  for (int j = 0; j < O; j++) {
    const uint4* f = reinterpret_cast<const uint4*>(sfac + (size_t)j * kP);
    uint64_t a = 0, b = 0;  // inputs 0..15 and 16..31
#pragma unroll
    for (int g = 0; g < kP / 4; g++) {
      const uint4 v = f[g];
      uint64_t t = (uint64_t)y[4 * g] * v.x;
      t += (uint64_t)y[4 * g + 1] * v.y;
      t += (uint64_t)y[4 * g + 2] * v.z;
      t += (uint64_t)y[4 * g + 3] * v.w;
      if (g < 4) a += t; else b += t;
    }
    const BconvOut<uint32_t> o = sout[j];
    PrimeConst<uint32_t> pc;
    pc.q = o.q;
    pc.q2 = o.q2;
    pc.mu_hi = o.mu_hi;
    pc.mu_lo = o.mu_lo;
    uint32_t r = barrett2<uint32_t>((uint32_t)(a >> 32), (uint32_t)a, pc);
    if (kP > 16) r = add_mod<uint32_t>(r, barrett2<uint32_t>((uint32_t)(b >> 32), (uint32_t)b, pc), o.q);
    d.out[(size_t)j * kN + coeff] = r;
  }
}

// The wide path's dispatch on the padded input count.
__device__ __forceinline__ void bconv_wide32(const BconvDesc<uint32_t>& d, const uint32_t* sfac, const BconvOut<uint32_t>* sout, int coeff) {
  switch ((d.I + 3) / 4) {
    case 3: bconv_body_wide32<12>(d, sfac, sout, coeff); break;
    case 4: bconv_body_wide32<16>(d, sfac, sout, coeff); break;
    case 5: bconv_body_wide32<20>(d, sfac, sout, coeff); break;
    case 6: bconv_body_wide32<24>(d, sfac, sout, coeff); break;
    case 7: bconv_body_wide32<28>(d, sfac, sout, coeff); break;
    default: bconv_body_wide32<32>(d, sfac, sout, coeff); break;
  }
}
constexpr int kBconvWideMaxInputs = 32;
template <typename W>
__host__ __device__ inline bool bconv_is_wide32(int I) {
  return sizeof(W) == 4 && I > kBconvRegInputs && I <= kBconvWideMaxInputs;
}

// Shared-memory need of one conversion (bytes): factor matrix, per-output constants and, for
// more than kBconvRegInputs inputs, one column of inputs per thread.
template <typename W>
__host__ __device__ inline size_t bconv_smem_bytes(int I, int O) {
  size_t n = (size_t)O * I * sizeof(W);
  n = (n + 15) / 16 * 16 + ((size_t)O * sizeof(BconvOut<W>) + 15) / 16 * 16;
  if (I > kBconvRegInputs) n += (size_t)I * kBconvThreads * sizeof(W);
  if (bconv_is_wide32<W>(I)) {  // padded factor rows in place of the plain matrix (and no input column)
    const size_t wide = ((size_t)O * ((I + 3) / 4 * 4) * sizeof(W) + 15) / 16 * 16 + ((size_t)O * sizeof(BconvOut<W>) + 15) / 16 * 16;
    if (wide > n) n = wide;
  }
  return n;
}

// The same conversion driven entirely by device-resident tables, the argument layout of the
// reference's launcher (_kernel_bco, cerium/compiler/backend/kernels/function.cuh:61-78, filled by
// Evaluator::fn_bco, cerium/runtime/execution/evaluator.cpp:861-940): conversion j reads
// ins[j] = [n_in[j]][N], writes outs[j] = [n_out[j]][N], with factors[j] = [O][I] residues and
// out_moduli[j] = [O] primes.  The host knows neither shapes nor primes, so the Barrett constants
// are derived here from the moduli (one division per output and CTA).  Lazy conversion only
// (the reference's), canonical outputs.
// The shared memory was sized on the host from the caller's shape bounds; a table entry above them
// (or above the smem_limit bytes the launch has) must not be staged: such a CTA touches no memory,
// records kStatusBconvShape in *status and returns.
// grid = (ceil(N / kBconvThreads), conversions), block = kBconvThreads, dynamic smem >= bconv_smem_bytes(I, O).
constexpr uint32_t kStatusBconvShape = 1u;  // bit of the context's status word
template <typename W>
__global__ void __launch_bounds__(kBconvThreads, 5)
    bconv_ptrs_kernel(W* const* __restrict__ outs, const size_t* __restrict__ n_out, const W* const* __restrict__ ins,
                      const size_t* __restrict__ n_in, const W* const* __restrict__ factors,
                      const W* const* __restrict__ out_moduli, const size_t max_in, const size_t max_out,
                      const size_t smem_limit, uint32_t* __restrict__ status) {
  CERIUM_DYN_SMEM(smem_raw);
  grid_dependency_launch();
  grid_dependency_wait();  // the tables may have been written by the stream's previous work
  const int j = blockIdx.y;
  const size_t In = n_in[j], On = n_out[j];
  if (In < 1 || On < 1 || In > max_in || On > max_out || bconv_smem_bytes<W>((int)In, (int)On) > smem_limit) {
    if (threadIdx.x == 0 && status != nullptr) atomicOr(status, kStatusBconvShape);
    return;
  }
  const int I = (int)In, O = (int)On;
  BconvDesc<W> d{};
  d.in = ins[j];
  d.out = outs[j];
  d.I = I;
  d.O = O;
  W* sfac = reinterpret_cast<W*>(smem_raw);
  const bool wide = bconv_is_wide32<W>(I);
  const int P = wide ? (I + 3) / 4 * 4 : I;  // words per staged factor row
  const size_t fac_bytes = ((size_t)O * P * sizeof(W) + 15) / 16 * 16;
  BconvOut<W>* sout = reinterpret_cast<BconvOut<W>*>(smem_raw + fac_bytes);
  const size_t out_bytes = ((size_t)O * sizeof(BconvOut<W>) + 15) / 16 * 16;
  W* scol = reinterpret_cast<W*>(smem_raw + fac_bytes + out_bytes);
  const W* fac = factors[j];
  const W* omod = out_moduli[j];
  for (int k = threadIdx.x; k < O * P; k += kBconvThreads) {
    const int jj = k / P, i = k - jj * P;
    sfac[k] = i < I ? fac[(size_t)jj * I + i] : (W)0;
  }
  for (int o = threadIdx.x; o < O; o += kBconvThreads) {
    const W q = omod[o];
    BconvOut<W> c{};
    c.q = q;
    c.q2 = q + q;
    if (sizeof(W) == 4) {
      // floor(2^64 / q) = floor((2^64 - 1) / q) for a q that is not a power of two
      const uint64_t mu = ~(uint64_t)0 / (uint64_t)q;
      c.mu_hi = (W)(mu >> 32);
      c.mu_lo = (W)(mu & 0xffffffffu);
    } else {
      // floor(2^128 / q) by two divisions: 2^64 = a q + r, then 2^128 / q = a 2^64 + floor(r 2^64 / q)
      const uint64_t a = ~(uint64_t)0 / (uint64_t)q;
      uint64_t r = ~(uint64_t)0 - a * (uint64_t)q + 1;  // 2^64 mod q (or q itself, fixed below)
      uint64_t hi = a;
      if (r >= (uint64_t)q) { r -= (uint64_t)q; hi += 1; }
      // long division of r * 2^64 by q, one bit at a time (r < q < 2^60, so 2r never overflows)
      uint64_t lo = 0;
      for (int bit = 0; bit < 64; bit++) {
        r <<= 1;
        lo <<= 1;
        if (r >= (uint64_t)q) { r -= (uint64_t)q; lo |= 1; }
      }
      c.mu_hi = (W)hi;
      c.mu_lo = (W)lo;
    }
    sout[o] = c;
  }
  __syncthreads();
  const int coeff = blockIdx.x * kBconvThreads + threadIdx.x;
  if (coeff >= kN) return;
  if (wide) {
    bconv_wide32(reinterpret_cast<const BconvDesc<uint32_t>&>(d), reinterpret_cast<const uint32_t*>(sfac),
                 reinterpret_cast<const BconvOut<uint32_t>*>(sout), coeff);
    return;
  }
  switch (I) {
    case 1: bconv_body<W, 1>(d, sfac, sout, scol, coeff); break;
    case 2: bconv_body<W, 2>(d, sfac, sout, scol, coeff); break;
    case 3: bconv_body<W, 3>(d, sfac, sout, scol, coeff); break;
    case 4: bconv_body<W, 4>(d, sfac, sout, scol, coeff); break;
    case 5: bconv_body<W, 5>(d, sfac, sout, scol, coeff); break;
    case 6: bconv_body<W, 6>(d, sfac, sout, scol, coeff); break;
    case 7: bconv_body<W, 7>(d, sfac, sout, scol, coeff); break;
    case 8: bconv_body<W, 8>(d, sfac, sout, scol, coeff); break;
    default: bconv_body<W, 0>(d, sfac, sout, scol, coeff); break;
  }
}

}  // namespace cerium
