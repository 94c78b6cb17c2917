// Client-side conversions of the encoder and decoder: integer-valued doubles (and small noise) to
// residues, and residues back to the centred integer as a correctly rounded double.
//
// Replace the host loops of the reference's encoder / decoder over SEAL's CRT composition
// (cerium/runtime/io/ckks-encoder.h:170-372): there one multi-word integer per coefficient is composed
// and decomposed on the CPU.
#pragma once
#include "modarith.cuh"

namespace cerium {

constexpr int kClientThreads = 256;
constexpr int kClientMaxLimbs = 128;

template <typename W>
struct ResidueArgs {
  const double* values;   // [N] integer-valued, any magnitude
  const int32_t* small;   // [N] added to the values, or null
  W* out;                 // [limbs][N]
  size_t out_stride;
  uint8_t prime[kClientMaxLimbs];
};

// out[l][i] = (values[i] + small[i]) mod q_l.  A double is M * 2^E with a 53-bit M: M mod q by Barrett, times
// 2^E mod q (square and multiply; only values of 2^53 and more have E > 0).  One thread per word, grid =
// (N / 256, limbs); bound by its 12 bytes read (the operands of all limbs but the first from L2) and the word
// written: one launch in place of a table look-up, two products and three passes per limb on the host.
template <typename W>
__global__ void __launch_bounds__(kClientThreads) residues_kernel(const ResidueArgs<W> g, const PrimeConst<W>* __restrict__ pcs) {
  grid_dependency_launch();
  grid_dependency_wait();
  const int b = blockIdx.y;
  const PrimeConst<W> pc = pcs[g.prime[b]];
  const int i = blockIdx.x * kClientThreads + threadIdx.x;
  const uint64_t bits = (uint64_t)__double_as_longlong(g.values[i]);
  const int field = (int)(bits >> 52) & 0x7ff;
  uint64_t m = field != 0 ? (bits & 0xfffffffffffffull) | (1ull << 52) : 0;  // a subnormal is no integer but zero
  int e = field - 1075;
  if (e < 0) {
    m = e > -64 ? m >> -e : 0;
    e = 0;
  }
  W r = sizeof(W) == 4 ? barrett2<W>((W)(m >> (sizeof(W) == 4 ? 32 : 0)), (W)m, pc) : reduce_word<W>((W)m, pc);
  if (e > 0) {
    W p = reduce_word<W>((W)1, pc), base = reduce_word<W>((W)2, pc);
    for (; e != 0; e >>= 1) {
      if (e & 1) p = mul_mod<W>(p, base, pc);
      base = mul_mod<W>(base, base, pc);
    }
    r = mul_mod<W>(r, p, pc);
  }
  if (bits >> 63) r = r != 0 ? pc.q - r : (W)0;
  if (g.small != nullptr) {
    const int32_t s = g.small[i];
    W t = reduce_word<W>((W)(s < 0 ? -(int64_t)s : (int64_t)s), pc);
    if (s < 0 && t != 0) t = pc.q - t;
    r = add_mod<W>(r, t, pc.q);
  }
  g.out[(size_t)b * g.out_stride + i] = r;
}

// Exact CRT composition of `limbs` 32-bit residues per coefficient.  With y_i = x_i [Qhat_i^-1] mod q_i the
// value is v = sum_i y_i Qhat_i - k Q, k the integer next to sum_i y_i / q_i: that is the centred representative
// (the sum of L terms below 1 is off by at most (L^2 + L) 2^-53 as a double, 2^-44 for 17 limbs and 2^-37 for 255, and where
// it is that close to a half the comparison with Q / 2 below decides), kept in two's complement over `words` 32-bit words, one column at a time.
struct ComposeArgs {
  const uint32_t* in;        // [limbs][N], coefficient form, canonical
  size_t in_stride;
  double* out;               // [N]
  const uint32_t* table;     // [limbs][words] Qhat_i, then [words] Q
  const uint32_t* inv;       // [limbs] [Qhat_i^-1]_{q_i}, then [limbs] Shoup companions, then [limbs] q_i
  const double* qinv;        // [limbs] RN(1 / q_i)
  int limbs, words;
};
constexpr int kComposeThreads = 32;    // the words and digits of a coefficient sit in shared memory: 32 columns
constexpr int kComposeMaxLimbs = 255;  // of at most 255 + 240 words are 62 KiB (8 KiB for the chain of 51 limbs)

// grid = N / 32.  Bound by limbs * words multiply-adds per coefficient (17 limbs: 272), i.e. by nothing at all
// beside the copies around it; the host composition it replaces took 7 us a coefficient and limb.
__global__ void __launch_bounds__(kComposeThreads) compose_kernel(const ComposeArgs g) {
  CERIUM_DYN_SMEM(raw);
  grid_dependency_launch();
  grid_dependency_wait();
  const int tid = threadIdx.x, L = g.limbs, n = g.words;
  const int i = blockIdx.x * kComposeThreads + tid;
  uint32_t* y = reinterpret_cast<uint32_t*>(raw) + tid;                  // y[l * threads]
  uint32_t* v = y + (size_t)L * kComposeThreads;                        // v[w * threads]
  const uint32_t* big_q = g.table + (size_t)L * n;
  double share = 0.0;
  for (int l = 0; l < L; l++) {
    const uint32_t q = g.inv[2 * L + l];
    const uint32_t t = csub<uint32_t>(mul_shoup_lazy<uint32_t>(g.in[(size_t)l * g.in_stride + i], g.inv[l], g.inv[L + l], q), q);
    y[l * kComposeThreads] = t;
    share = __fma_rn((double)t, g.qinv[l], share);
  }
  const uint32_t k = (uint32_t)__double2ll_rn(share);  // at most limbs
  // column w: sum_l y_l Qhat_l[w] - k Q[w] + carry; up to 255 products below 2^62, so the sum is kept as two halves
  int64_t carry = 0;
  for (int w = 0; w < n; w++) {
    uint64_t lo = 0, hi = 0;
    for (int l = 0; l < L; l++) {
      const uint64_t p = (uint64_t)y[l * kComposeThreads] * g.table[(size_t)l * n + w];
      lo += (uint32_t)p;
      hi += p >> 32;
    }
    const uint64_t s = (uint64_t)k * big_q[w];
    const int64_t low = (int64_t)lo - (int64_t)(uint32_t)s + carry;     // |low| < 2^40
    v[w * kComposeThreads] = (uint32_t)low;
    carry = (int64_t)hi - (int64_t)(s >> 32) + (low >> 32);
  }
  bool neg = (v[(n - 1) * kComposeThreads] >> 31) != 0;
  if (neg) {
    uint64_t c = 1;
    for (int w = 0; w < n; w++) {
      c += (uint32_t)~v[w * kComposeThreads];
      v[w * kComposeThreads] = (uint32_t)c;
      c >>= 32;
    }
  }
  // the magnitude is at most Q / 2 unless the rounding of k was a tie's neighbour: Q - magnitude, other sign
  int cmp = 0;
  for (int w = n - 1; w >= 0 && cmp == 0; w--) {
    const uint32_t h = (big_q[w] >> 1) | (w + 1 < n ? big_q[w + 1] << 31 : 0u), a = v[w * kComposeThreads];
    cmp = a > h ? 1 : a < h ? -1 : 0;
  }
  if (cmp > 0) {
    int64_t c = 0;
    for (int w = 0; w < n; w++) {
      c += (int64_t)big_q[w] - (int64_t)v[w * kComposeThreads];
      v[w * kComposeThreads] = (uint32_t)c;
      c >>= 32;
    }
    neg = !neg;
  }
  // the leading 64 bits, everything below them as a sticky bit, rounded once
  int t = n - 1;
  while (t > 0 && v[t * kComposeThreads] == 0) t--;
  const uint32_t w0 = v[t * kComposeThreads], w1 = t > 0 ? v[(t - 1) * kComposeThreads] : 0u,
                 w2 = t > 1 ? v[(t - 2) * kComposeThreads] : 0u;
  int z = 0;
  while (z < 32 && !((w0 << z) >> 31)) z++;
  double d = 0.0;
  if (z < 32) {
    uint64_t m = (((uint64_t)w0 << 32 | w1) << z) | (z != 0 ? w2 >> (32 - z) : 0u);
    bool sticky = (w2 << z) != 0;
    for (int w = t - 3; w >= 0; w--) sticky = sticky || v[w * kComposeThreads] != 0;
    m |= sticky ? 1u : 0u;
    // m = value * 2^-e: RN(m) * 2^e in two exact steps (the exponent may pass 1023 on its own)
    const int e = 32 * (t - 1) - z;
    d = ldexp(__ull2double_rn(m), e);
  }
  g.out[i] = neg ? -d : d;
}

}  // namespace cerium
