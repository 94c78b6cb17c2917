// Negacyclic NTT kernels for N = 2^16 over batches of RNS limbs.
//
// Replaces the reference's four NTT kernels and their launchers:
//   forward  ntt0/ntt1   cerium/compiler/backend/kernels/fhe_ntt.cuh:114-273,
//                        cerium/compiler/backend/kernels/function.cu:22-99
//   inverse  intt0/intt1 cerium/compiler/backend/kernels/fhe_ntt.cuh:470-601,
//                        cerium/compiler/backend/kernels/function.cu:199-280
//   SuD tail ntt1_sud    cerium/compiler/backend/kernels/fhe_ntt.cuh:278-359
// Same contract (standard order in -> bit-reversed order out for the forward transform,
// the inverse undoes it and scales by 1/N), different design:
//
//  * The 16 radix-2 layers are four radix-16 levels.  A level keeps 16 coefficients of one
//    thread in registers; two levels make a pass, with one shared-memory exchange between
//    them, so one limb crosses HBM twice per transform (once per pass) and the exchange
//    never leaves the SM.
//  * Twiddles are addressed through the "root prefix" S of a radix-16 group: layer t of the
//    group uses table entries (S << t) + (j >> (4 - t)), j the register index.  Level 0 has
//    S = 1, level 1 S = 16 + a, level 2 S = 256 + h, level 3 S = 4096 + 16 h + u.
//    The 255 twiddles of the column pass are the same for every column and sit in shared
//    memory; the row pass reads its twiddles in contiguous runs of 1, 2, 4, 8 entries.
//  * The column pass moves 128-byte row segments (16 u64 / 32 u32 columns per CTA); the row
//    pass gives each thread 16 consecutive coefficients and stores them as 16-byte vectors.
//  * Values stay lazy inside a transform ([0,4q) forward, [0,2q) inverse) and are reduced to
//    [0,q) by the last pass, so every buffer a caller sees is canonical.
#pragma once
#include <cstring>

#include "modarith.cuh"

namespace cerium {

template <typename W>
struct NttCfg;
template <>
struct NttCfg<uint64_t> {
  static constexpr int kCols = 16;  // 16 * 8 B = 128 B segments in the column pass
};
template <>
struct NttCfg<uint32_t> {
  static constexpr int kCols = 32;  // 32 * 4 B = 128 B
};

// Tiles of the two passes: `kCols` columns on 16 kCols threads, or rows of 256 coefficients on 16 threads each.  Batches
// that do not fill the GPU take smaller tiles (the work is spread over all SMs: 160 tiles of 256 threads on 148 SMs
// leave twelve with twice the work of the others), and rows then copy their twiddles into shared memory before
// they wait for the previous kernel, so that a warp's chain has one memory latency less.  On full launches both cost more than
// they give: the copies go through the same pipes as the data (71 -> 77 us for 245 limbs).
constexpr int kRowsPerCta = 16;
constexpr int kRowsSmall = 4;
// ... up to this many usual tiles per SM (64 and 74 limbs on 148 SMs).  From there on the usual tiles are as fast or faster
// (70 limbs of 64-bit words forward 36.9 against 37.7 us; 30 limbs inverse 20.4 against 17.9, 60 of 32-bit words 21.2 against 19.2)
template <typename W>
constexpr int kSmallBatchPerSm = sizeof(W) == 8 ? 7 : 8;
// Lane-interleaved level-3 twiddles: [row h (256)][e = 2^t - 1 + g (15)][thread u (16)] pairs per
// prime; entry = bit-reversed table[((4096 + 16 h + u) << t) + g].
constexpr int kRowTwPerPrime = 256 * 15 * 16;
// Limbs per launch: the largest multiple of 64 with which the parameters of every kernel stay within 4 KB (the asserts in the
// forward passes, whose loaders and epilogues are the long ones).  A call of more goes on in launches of that many.  512 loses 3 to
// 4 % on 513 to 576 limbs (576 forward 262.9 us against 255.2); shared out evenly, 577 limbs of 32-bit words 155.8 -> 159.7, 625 of
// 64-bit words inverse 291 -> 307.
constexpr int kMaxBatch = 576;
constexpr size_t kMaxParameters = 4096;

// Addressing of a batch of limbs: batch entry b lives at base + pos[b] * stride; its modulus
// is prime[b] (index into the context's prime list).  Passed by value as a kernel parameter.
// in_stride = 0 makes every entry read the same source limb (rescale broadcasts the last limb).
template <typename W>
struct StridedBatch {
  static constexpr bool kProduct = false;
  const W* in;
  W* out;
  size_t in_stride;   // in words
  size_t out_stride;  // in words
  W* out2;            // entries b >= split write to out2 instead of out (two result stacks, one launch)
  int split;          // kMaxBatch when unused
  uint32_t in_elt;    // inverse transform only, not 0: word i of an input limb is read at pi(i), the Galois
                      // automorphism of this element (modarith.cuh), so a rotation costs no pass of its own
  uint16_t pos[kMaxBatch];
  uint8_t prime[kMaxBatch];
  __device__ __forceinline__ const W* in_limb(int b) const { return in + (size_t)pos[b] * in_stride; }
  __device__ __forceinline__ W* out_limb(int b) const {
    return (b >= split ? out2 : out) + (size_t)pos[b] * out_stride;
  }
  __device__ __forceinline__ uint32_t prime_of(int b) const { return prime[b]; }
  __device__ __forceinline__ uint32_t gather_elt() const { return in_elt; }
};

// StridedBatch whose entries read from a slot of their own: entry b reads limb in_pos[b] of `in`
// and writes limb pos[b] of `out` (one coefficient-form limb transformed under many primes).
template <typename W>
struct GatherBatch : StridedBatch<W> {
  uint16_t in_pos[kMaxBatch];
  __device__ __forceinline__ const W* in_limb(int b) const {
    return this->in + (size_t)in_pos[b] * this->in_stride;
  }
};

// StridedBatch whose input is the product of two stacks of words with one stride (inverse transform).
template <typename W>
struct ProductBatch : StridedBatch<W> {
  static constexpr bool kProduct = true;
  const W* factor;
  __device__ __forceinline__ const W* factor_limb(int b) const { return factor + (size_t)this->pos[b] * this->in_stride; }
};

// Addressing through device-resident pointer tables, the layout the reference's launchers
// take (args_outputs / args_inputs / bases, cerium/compiler/backend/kernels/function.cu:22-39).
template <typename W>
struct PointerBatch {
  static constexpr bool kProduct = false;
  W* const* outs;
  const W* const* ins;
  const uint32_t* bases;
  int in_step;  // entry b reads ins[b * in_step + in_off] (the SuD launcher passes two inputs per entry)
  int in_off;
  __device__ __forceinline__ const W* in_limb(int b) const { return ins[b * in_step + in_off]; }
  __device__ __forceinline__ W* out_limb(int b) const { return outs[b]; }
  __device__ __forceinline__ uint32_t prime_of(int b) const { return bases[b]; }
  __device__ __forceinline__ uint32_t gather_elt() const { return 0u; }
};

// ---------------------------------------------------------------------------------------
// arithmetic policies
// ---------------------------------------------------------------------------------------

// Strict butterflies keep every value below 4q (forward) / 2q (inverse), twice that for 64-bit words, with one
// correction per butterfly; they serve 32-bit words and 64-bit primes of 52 bits or more.
// Lazy butterflies (64-bit words, primes below 2^52) use the headroom above the prime instead
// of corrections and the 32-bit-piece products of modarith.cuh.
// Fp butterflies (64-bit words, primes below 2^50) run on the FP64 pipe: the registers hold the
// bit patterns of doubles, signed residues whose bound a compile-time plan tracks.
enum : int { kArithStrict = 0, kArithLazy = 1, kArithFp = 2 };

template <typename W, int kMode>
struct Arith {
  static constexpr bool kLazy = kMode == kArithLazy;
  W q, q2, q4, nq;
  __device__ __forceinline__ explicit Arith(const PrimeConst<W>& pc)
      : q(pc.q), q2(pc.q + pc.q), q4(pc.q * 4), nq((W)0 - pc.q) {}
  // canonical residue -> the form the butterflies work on
  __device__ __forceinline__ W enter(W x) const { return x; }
  __device__ __forceinline__ W reduce(W x) const { return x; }
  __device__ __forceinline__ void fwd(W& a, W& b, W w, W ws) const {
    if (kLazy) butterfly_fwd_lazy<W>(a, b, w, ws, nq, q4);
    else butterfly_fwd(a, b, w, ws, q, q2, nq, q4);
  }
  // k = layer number inside the pass (0..7)
  __device__ __forceinline__ void inv(W& a, W& b, W w, W ws, int k) const {
    if (kLazy) butterfly_inv_lazy<W>(a, b, w, ws, nq, q4 << k);
    else butterfly_inv(a, b, w, ws, q, q2, nq, q4);
  }
  // value at the end of a forward transform -> [0, q), or only below 4q when the consumer
  // takes lazy residues (kCanonical = false)
  template <bool kCanonical>
  __device__ __forceinline__ W finish_fwd(W x, W one_shoup) const {
    if (kLazy) x = reduce_lazy(x, one_shoup, nq);
    else if constexpr (sizeof(W) == 8) x = csub<W>(csub_high(x, q4), q4);
    if (!kCanonical) return x;
    return csub<W>(csub<W>(x, q2), q);
  }
  // last inverse layer: (a + b) * last[0] and (a - b) * last[2], reduced to [0, q); last = {N^-1, Shoup companion,
  // w1 * N^-1, Shoup companion}, times the caller's scale where there is one
  __device__ __forceinline__ void inv_last(W& a, W& b, const W (&last)[4]) const {
    const W s = a + b;
    if (kLazy || sizeof(W) == 8) {
      const W d = a + (kLazy ? (q4 << 7) : q4 + q) - b;
      a = csub<W>(csub<W>(mul_shoup_approx(s, last[0], last[1], nq), q2), q);
      b = csub<W>(csub<W>(mul_shoup_approx(d, last[2], last[3], nq), q2), q);
    } else {
      const W d = a + q2 - b;
      a = csub<W>(mul_shoup_lazy<W>(s, last[0], last[1], q), q);
      b = csub<W>(mul_shoup_lazy<W>(d, last[2], last[3], q), q);
    }
  }
};

template <>
struct Arith<uint64_t, kArithFp> {
  using W = uint64_t;
  double q, nq, qinv;
  __device__ __forceinline__ explicit Arith(const PrimeConst<W>& pc) {
    q = fp_from_u64(pc.q);
    nq = -q;
    qinv = d(pc.fp_qinv);
  }
  static __device__ __forceinline__ double d(W x) { return __longlong_as_double((long long)x); }
  static __device__ __forceinline__ W u(double x) { return (W)__double_as_longlong(x); }
  __device__ __forceinline__ W enter(W x) const { return u(fp_from_u64(x)); }
  __device__ __forceinline__ W reduce(W x) const { return u(fp_reduce(d(x), qinv, nq)); }
  // y k - c q with the quotient from the rounded product: |y| <= q, 0 <= k < q < 2^50 put RN(RN(y k) RN(1/q)) off by
  // 3/2^53 * 2^50 = 3/8 at most before it is rounded, so the result is below 7/8 q (exact as in fp_mulmod)
  __device__ __forceinline__ double product(double y, double k) const {
    const double h = __dmul_rn(y, k);
    const double l = __fma_rn(y, k, -h);
    const double c = __dadd_rn(__fma_rn(h, qinv, kFpMagic), -kFpMagic);
    return __dadd_rn(__fma_rn(c, nq, h), l);
  }
  // quotient of a twiddle by q when the table holds the twiddle alone, and one as good as a tabulated one (within 2^-55 and 2^-100)
  __device__ __forceinline__ W quotient(W w) const { return u(__dmul_rn(d(w), qinv)); }
  __device__ __forceinline__ W close_quotient(W w) const {
    const double c = __dmul_rn(d(w), qinv);
    return u(__fma_rn(__fma_rn(c, nq, d(w)), qinv, c));
  }
  __device__ __forceinline__ void fwd(W& a, W& b, W w, W wq) const {
    const double r = fp_mulmod(d(b), d(w), d(wq), nq);
    const double x = d(a);
    a = u(__dadd_rn(x, r));
    b = u(__dadd_rn(x, -r));
  }
  __device__ __forceinline__ void inv(W& a, W& b, W w, W wq, int /*k*/) const {
    const double x = d(a), y = d(b);
    a = u(__dadd_rn(x, y));
    b = u(fp_mulmod(__dadd_rn(x, -y), d(w), d(wq), nq));
  }
  // |x| <= 0.63 q -> [0, q) as an integer word
  __device__ __forceinline__ W canonical(double x) const {
    return fp_to_u64(x < 0.0 ? __dadd_rn(x, q) : x);
  }
  template <bool kCanonical>
  __device__ __forceinline__ W finish_fwd(W x, W /*one_shoup*/) const {
    const double r = fp_reduce(d(x), qinv, nq);
    if (kCanonical) return canonical(r);
    return fp_to_u64(__dadd_rn(r, q));  // (0.49 q, 1.51 q): a lazy residue
  }
  // last: the two constants of the last layer, each with its quotient by q
  __device__ __forceinline__ void inv_last(W& a, W& b, const W (&last)[4]) const {
    const double x = d(a), y = d(b);
    a = canonical(fp_mulmod(__dadd_rn(x, y), d(last[0]), d(last[1]), nq));
    b = canonical(fp_mulmod(__dadd_rn(x, -y), d(last[2]), d(last[3]), nq));
  }
};

// ---------------------------------------------------------------------------------------
// Compile-time plan of the Fp butterflies: bounds in units of q / 1024, rounded up.
// A product's operand may reach 4q and comes back within q * (1/2 + operand / 32q); sums stay
// below 8q.  The plan walks the layers of a radix-16 group and reduces, just in time, the
// values whose bound would break the operand limit.
// ---------------------------------------------------------------------------------------
constexpr int kFpCanon = 1024;       // canonical input, [0, q)
constexpr int kFpReduced = 513;      // after fp_reduce
constexpr int kFpOperandMax = 4096;  // operand of a product
// k32 = 1: the twiddle comes with its tabulated quotient RN(w / q); k32 = 3: the quotient is
// computed as RN(w * RN(1 / q)) (last level of the row pass, whose table then holds w only), three
// times the error: |r| <= q * (1/2 + 3 * operand / 32q)
__host__ __device__ constexpr int fp_product_bound(int operand, int k32 = 1) {
  return 512 + (k32 * operand + 31) / 32;
}

// forward (Cooley-Tukey): a' = a + w*b, b' = a - w*b; all 16 values share one bound
struct FpFwdPlan {
  bool before[4];  // reduce every value before layer t
  int out;
};
__host__ __device__ constexpr FpFwdPlan fp_plan_fwd(int bin, int k32 = 1) {
  FpFwdPlan p{};
  int b = bin;
  for (int t = 0; t < 4; t++) {
    p.before[t] = b > kFpOperandMax;
    if (p.before[t]) b = kFpReduced;
    b += fp_product_bound(b, k32);
  }
  p.out = b;
  return p;
}

// inverse (Gentleman-Sande): a' = a + b, b' = w * (a - b); the operand a - b needs
// bound(a) + bound(b) <= 4q.  before[t] is the mask of registers to reduce before layer t.
struct FpInvPlan {
  unsigned before[4];
  int bound[16];
  int max_out;
};
__host__ __device__ constexpr FpInvPlan fp_plan_inv(int bin, int k32 = 1) {
  FpInvPlan p{};
  for (int j = 0; j < 16; j++) p.bound[j] = bin;
  for (int t = 3; t >= 0; t--) {
    const int half = 8 >> t;
    unsigned mask = 0;
    for (int g = 0; g < (1 << t); g++)
      for (int k = 0; k < half; k++) {
        const int j = g * 2 * half + k, i = j + half;
        if (p.bound[j] + p.bound[i] > kFpOperandMax) {
          const int big = p.bound[j] >= p.bound[i] ? j : i;
          p.bound[big] = kFpReduced;
          mask |= 1u << big;
          if (p.bound[j] + p.bound[i] > kFpOperandMax) {
            const int other = big == j ? i : j;
            p.bound[other] = kFpReduced;
            mask |= 1u << other;
          }
        }
        const int sum = p.bound[j] + p.bound[i];
        p.bound[j] = sum;
        p.bound[i] = fp_product_bound(sum, k32);
      }
    p.before[t] = mask;
  }
  p.max_out = 0;
  for (int j = 0; j < 16; j++) p.max_out = p.bound[j] > p.max_out ? p.bound[j] : p.max_out;
  return p;
}
// Registers above `threshold` are reduced before they are exchanged (the next group mixes the
// registers of 16 threads, so it starts from the largest bound).
struct FpExchange {
  unsigned mask;
  int out;
};
__host__ __device__ constexpr FpExchange fp_plan_exchange(const FpInvPlan& p, int threshold) {
  FpExchange e{};
  for (int j = 0; j < 16; j++) {
    int b = p.bound[j];
    if (b > threshold) {
      e.mask |= 1u << j;
      b = kFpReduced;
    }
    e.out = b > e.out ? b : e.out;
  }
  return e;
}
constexpr int kFpInvExchangeMax = 2048;

// bounds along the forward transform: the column pass starts from its loader's bound and stores at most kFpFwdMid, from which the
// row pass starts, raised digits at most kFpRaisedMid: canonical words, and what a base conversion leaves (bconv_mma.cuh): below
// 2.3 q, with a rounding term below 3.3 q.  (With 4 q for both the row of a raised digit is reduced twice on its way, so once.)
constexpr int kFpRaisedIn = 2356, kFpLoweredIn = 3380;
constexpr int fp_plan_cols(int bin) { return fp_plan_fwd(fp_plan_fwd(bin).out).out; }
constexpr int fp_max(int a, int b) { return a > b ? a : b; }
constexpr int kFpRaisedMid = fp_max(fp_plan_cols(kFpCanon), fp_plan_cols(kFpRaisedIn));
constexpr int kFpFwdMid = fp_max(kFpRaisedMid, fp_plan_cols(kFpLoweredIn));
constexpr int kFpLaneK32 = 3;  // level 3 (lane table) computes its quotients
// bounds along the inverse transform: row pass (levels 3, 2) stores kFpInvMid
constexpr int kFpInvL3 = fp_plan_exchange(fp_plan_inv(kFpCanon, kFpLaneK32), kFpInvExchangeMax).out;
constexpr int kFpInvMid = fp_plan_inv(kFpInvL3).max_out;
constexpr int kFpInvL1 = fp_plan_exchange(fp_plan_inv(kFpInvMid), kFpInvExchangeMax).out;
constexpr unsigned kFpInvRowsExMask = fp_plan_exchange(fp_plan_inv(kFpCanon, kFpLaneK32), kFpInvExchangeMax).mask;
constexpr unsigned kFpInvColsExMask = fp_plan_exchange(fp_plan_inv(kFpInvMid), kFpInvExchangeMax).mask;
static_assert(kFpFwdMid < 8192 && kFpInvMid < 8192, "stored intermediates must stay exact integers");

template <typename W, int kMode>
__device__ __forceinline__ void fp_reduce_masked(W (&x)[16], unsigned mask, const Arith<W, kMode>& ar) {
#pragma unroll
  for (int j = 0; j < 16; j++)
    if (mask >> j & 1u) x[j] = ar.reduce(x[j]);
}

// ---------------------------------------------------------------------------------------
// radix-16 register kernels
// ---------------------------------------------------------------------------------------

template <typename W, bool kGlobalTw>
__device__ __forceinline__ typename WordTraits<W>::Pair load_tw(const typename WordTraits<W>::Pair* t,
                                                                 uint32_t idx) {
  if (kGlobalTw) return __ldg(t + idx);
  return t[idx];
}

// Twiddle addressing of a radix-16 group.  Plain: entry (S << t) + g of the bit-reversed table.
// Lane-interleaved: the group's 15 twiddles sit at entries e * 16, e = 2^t - 1 + g,
// of a table pre-permuted so that the 16 threads of a row read 16 consecutive entries.  Group: at entries e.
enum : int { kTwPlain = 0, kTwLane = 1, kTwGroup = 2 };
template <int kTw>
__device__ __forceinline__ uint32_t tw_index(uint32_t S, int t, int g) {
  return kTw == kTwPlain ? (S << t) + (uint32_t)g : (uint32_t)(((1 << t) - 1 + g) * (kTw == kTwLane ? 16 : 1));
}

// Lane-interleaved table of a prime with double-precision butterflies: twiddles only, two per
// 16-byte entry; twiddle e = 2^t - 1 + g sits in double number e + 1 of the group's 16 (number 0
// is padding, so that every layer starts on an entry boundary), entry v of thread u at (v * 16).
template <typename W, bool kGlobalTw>
__device__ __forceinline__ W lane_tw_fp(const typename WordTraits<W>::Pair* tw, int t, int g) {
  const int slot = (1 << t) + g;
  const auto pv = load_tw<W, kGlobalTw>(tw, (slot >> 1) * 16);
  return (slot & 1) ? pv.y : pv.x;
}

// Four forward layers on x[0..15]; layer t pairs (j, j + (8 >> t)).  kBin: bound of the inputs
// (Fp arithmetic only).
template <typename W, bool kGlobalTw, int kMode, int kTw = kTwPlain, int kBin = 0>
__device__ __forceinline__ void radix16_fwd(W (&x)[16], const typename WordTraits<W>::Pair* tw,
                                            uint32_t S, const Arith<W, kMode>& ar) {
  static_assert(kTw == kTwPlain || kMode != kArithFp, "the lane tables of Fp primes have no companions");
  constexpr FpFwdPlan plan = fp_plan_fwd(kBin);
#pragma unroll
  for (int t = 0; t < 4; t++) {
    const int half = 8 >> t;
    if (kMode == kArithFp && plan.before[t]) fp_reduce_masked<W, kMode>(x, 0xffffu, ar);
#pragma unroll
    for (int g = 0; g < (1 << t); g++) {
      const auto w = load_tw<W, kGlobalTw>(tw, tw_index<kTw>(S, t, g));
#pragma unroll
      for (int k = 0; k < half; k++) {
        const int j = g * 2 * half + k;
        ar.fwd(x[j], x[j + half], w.x, w.y);
      }
    }
  }
}

// The four inverse layers of the same group, in reverse order; kLayer0 is the pass-local
// number of the first layer executed (0 for the first level of a pass, 4 for the second).
template <typename W, bool kGlobalTw, int kMode, int kLayer0, int kTw = kTwPlain, int kBin = 0>
__device__ __forceinline__ void radix16_inv(W (&x)[16], const typename WordTraits<W>::Pair* twi,
                                            uint32_t S, const Arith<W, kMode>& ar) {
  constexpr bool kPacked = kTw == kTwLane && kMode == kArithFp;
  constexpr FpInvPlan plan = fp_plan_inv(kBin, kPacked ? kFpLaneK32 : 1);
#pragma unroll
  for (int t = 3; t >= 0; t--) {
    const int half = 8 >> t;
    if (kMode == kArithFp) fp_reduce_masked<W, kMode>(x, plan.before[t], ar);
#pragma unroll
    for (int g = 0; g < (1 << t); g++) {
      W w0, w1;
      if constexpr (kPacked) {
        w0 = lane_tw_fp<W, kGlobalTw>(twi, t, g);
        w1 = ar.quotient(w0);
      } else {
        const auto w = load_tw<W, kGlobalTw>(twi, tw_index<kTw>(S, t, g));
        w0 = w.x;
        w1 = w.y;
      }
#pragma unroll
      for (int k = 0; k < half; k++) {
        const int j = g * 2 * half + k;
        ar.inv(x[j], x[j + half], w0, w1, kLayer0 + 3 - t);
      }
    }
  }
}

// Level 0 of the inverse transform (S = 1, layers 4..7 of the column pass): the last layer
// also multiplies by N^-1 and reduces to [0, q).
template <typename W, int kMode, int kBin = 0>
__device__ __forceinline__ void radix16_inv_final(W (&x)[16], const typename WordTraits<W>::Pair* twi,
                                                  const W (&last)[4], const Arith<W, kMode>& ar) {
  constexpr FpInvPlan plan = fp_plan_inv(kBin);
#pragma unroll
  for (int t = 3; t >= 1; t--) {
    const int half = 8 >> t;
    if (kMode == kArithFp) fp_reduce_masked<W, kMode>(x, plan.before[t], ar);
#pragma unroll
    for (int g = 0; g < (1 << t); g++) {
      const auto w = twi[(1u << t) + g];
#pragma unroll
      for (int k = 0; k < half; k++) {
        const int j = g * 2 * half + k;
        ar.inv(x[j], x[j + half], w.x, w.y, 4 + 3 - t);
      }
    }
  }
  if (kMode == kArithFp) fp_reduce_masked<W, kMode>(x, plan.before[0], ar);
#pragma unroll
  for (int j = 0; j < 8; j++) ar.inv_last(x[j], x[j + 8], last);
}

// Row-pass exchange buffer: one pad word after every 16 keeps both the strided and the
// consecutive access pattern free of bank conflicts.
__device__ __forceinline__ int row_pos(int i) { return i + (i >> 4); }
constexpr int kRowPitch = 256 + 16;

// Staging buffer that turns "each thread owns 16 consecutive words of its row" into
// "consecutive threads own consecutive 16-byte vectors" (and back) without bank conflicts.
// A row is 256 words = kVecPerRow vectors of 16 bytes; thread u owns vectors u * kVecPerThread
// + jj.  Vector v is stored at slot v ^ ((v >> 3) & (kVecPerThread - 1)) of its row: both the
// owner's accesses (8 threads, same jj) and the coalesced accesses (8 consecutive v) then fall
// into 8 different 16-byte bank groups.
template <typename W>
struct RowVec;
template <>
struct RowVec<uint64_t> {
  using Vec = ulonglong2;
  static constexpr int kWords = 2, kPerThread = 8, kPerRow = 128;
};
template <>
struct RowVec<uint32_t> {
  using Vec = uint4;
  static constexpr int kWords = 4, kPerThread = 4, kPerRow = 64;
};
template <typename W>
__device__ __forceinline__ int row_vec_slot(int v) {
  return v ^ ((v >> 3) & (RowVec<W>::kPerThread - 1));
}
__device__ __forceinline__ void vec_unpack(const ulonglong2& v, uint64_t* w) { w[0] = v.x; w[1] = v.y; }
__device__ __forceinline__ void vec_unpack(const uint4& v, uint32_t* w) { w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w; }
__device__ __forceinline__ ulonglong2 vec_pack(const uint64_t* w) { return make_ulonglong2(w[0], w[1]); }
__device__ __forceinline__ uint4 vec_pack(const uint32_t* w) { return make_uint4(w[0], w[1], w[2], w[3]); }

// Twiddles of a row pass's rows in shared memory.  Tables of integer butterflies of 64-bit words are twice as long and
// stay in global memory.
template <typename W, int kRows>
struct RowTwiddles {
  using Pair = typename WordTraits<W>::Pair;
  static constexpr int kLane = sizeof(W) == 8 ? 8 * 16 : 15 * 16;  // entries of a row's lane table
  static constexpr int kGroupPitch = 17;                           // rows of a warp in different banks
  Pair lane[kRows][kLane];
  Pair group[kRows][kGroupPitch];
};
template <typename W, int kRows, bool kStage>
struct alignas(16) RowsBuffer {
  W tile[kRows * kRowPitch];
  RowTwiddles<W, kStage ? kRows : 1> tw;
};

// Starts the copies of this warp's two rows (h0: first row of the CTA); row_twiddles_wait() before they are used.
template <typename W, int kRows>
__device__ __forceinline__ void row_twiddles_start(RowTwiddles<W, kRows>& to, const typename WordTraits<W>::Pair* tw,
                                                   const typename WordTraits<W>::Pair* twr, int h0) {
  using RT = RowTwiddles<W, kRows>;
  using Pair = typename RT::Pair;
  const int lane = threadIdx.x & 31, r0 = threadIdx.x >> 5 << 1;
  constexpr int kChunks = 2 * RT::kLane * (int)sizeof(Pair) / 16;  // the lane tables of neighbouring rows adjoin
  const char* src = reinterpret_cast<const char*>(twr + (size_t)(h0 + r0) * RT::kLane);
  char* dst = reinterpret_cast<char*>(to.lane[r0]);
#pragma unroll
  for (int k = 0; k < (kChunks + 31) / 32; k++) {
    const int i = lane + 32 * k;
    if (kChunks % 32 == 0 || i < kChunks) copy_async<16>(dst + i * 16, src + i * 16);
  }
  // level 2: entry e = 2^t - 1 + g of row r is table entry ((256 + h) << t) + g
  const int r = r0 + (lane >> 4), e = lane & 15;
  if (e < 15) {
    const int t = e < 1 ? 0 : e < 3 ? 1 : e < 7 ? 2 : 3;
    copy_async<sizeof(Pair)>(&to.group[r][e], tw + (((uint32_t)(256 + h0 + r) << t) + (uint32_t)(e - ((1 << t) - 1))));
  }
}
__device__ __forceinline__ void row_twiddles_wait() {
#if !defined(CERIUM_EMU)
  asm volatile("cp.async.wait_all;" ::: "memory");
#endif
  __syncwarp();
}

// Runs one of the instantiations of a kernel body: the arithmetic policy of this CTA's prime
// (BODY is a template name taking <W, mode, ...>; ARGS its call arguments in parentheses).
#define CERIUM_TARGS(...) __VA_ARGS__
#define CERIUM_DISPATCH_ARITH(W, pc, BODY, TARGS, ARGS)                   \
  do {                                                                   \
    if constexpr (sizeof(W) == 8) {                                      \
      if ((pc).fp_ok != 0) { BODY<W, kArithFp, TARGS> ARGS; break; }     \
      if ((pc).lazy_ok != 0) { BODY<W, kArithLazy, TARGS> ARGS; break; } \
    }                                                                    \
    BODY<W, kArithStrict, TARGS> ARGS;                                   \
  } while (0)

// ---------------------------------------------------------------------------------------
// forward transform
// ---------------------------------------------------------------------------------------

// What the column pass does with a word it has just read.
template <typename W>
struct PlainLoader {
  static constexpr bool kPlain = true;  // words of the caller, as they are
  static constexpr bool kHasSmall = false;
  static constexpr int kFpBound = kFpCanon;
  __device__ __forceinline__ W apply(W x, int /*b*/, const PrimeConst<W>& /*pc*/) const { return x; }
};

// Source residues belong to another modulus: any word -> [0, q) of the entry's prime.  This is
// the whole base conversion of a one-limb digit (Qhat = 1), fused into the transform's first read.
template <typename W>
struct ModLoader {
  static constexpr bool kPlain = false;
  static constexpr int kFpBound = kFpCanon;
  static constexpr bool kHasSmall = true;
  // small[b] != 0: the words of entry b are below 2^50 (their source prime is), so a prime with
  // double-precision butterflies converts and reduces them on the FP64 pipe (5 operations)
  // instead of the integer Shoup reduction
  uint8_t small[kMaxBatch];
  __device__ __forceinline__ W apply(W x, int /*b*/, const PrimeConst<W>& pc) const {
    return reduce_word<W>(x, pc);
  }
};

// Words as a base conversion leaves them for the transform, kBound / 1024 q at most for primes with double-precision butterflies and
// below 4q for all.
template <typename W, int kBound>
struct LazyLoader {
  static constexpr bool kPlain = false;
  static constexpr bool kHasSmall = false;
  static constexpr int kFpBound = kBound;
  __device__ __forceinline__ W apply(W x, int /*b*/, const PrimeConst<W>& /*pc*/) const { return x; }
};

// limbs per launch when per-limb scalars travel as parameters (4 KB of them at 128 limbs of 64-bit words).  Both
// polynomials of a key switch over up to 64 limbs share one launch pair: a 32-bit rotation of 51 limbs took 213.8 us with
// two launch pairs (limit 96), now 207.5
constexpr int kSudMaxBatch = 128;

// Source residues belong to another (possibly larger) modulus src_q: optionally add pre_add
// mod src_q (rounding), reduce into [0, q) of the target prime, optionally subtract
// post_sub[b] mod q.  Used when one coefficient-form limb is re-read under many primes
// (rescale, cerium/compiler/backend/compiler_rescale.cc:262-284).
template <typename W>
struct ReduceLoader {
  static constexpr bool kPlain = false;
  static constexpr bool kHasSmall = false;
  static constexpr int kFpBound = kFpCanon;
  W src_q;
  W pre_add;
  W post_sub[kSudMaxBatch];
  __device__ __forceinline__ W apply(W x, int b, const PrimeConst<W>& pc) const {
    W v = csub<W>(x + pre_add, src_q);
    v = reduce_word<W>(v, pc);
    return sub_mod<W>(v, post_sub[b], pc.q);
  }
};

template <typename W, int kMode, int kCols, typename Batch, typename Loader>
__device__ __forceinline__ void ntt_fwd_cols_body(const Batch& batch, const Loader& loader, int b,
                                                  const PrimeConst<W>& pc, W* tile,
                                                  const typename WordTraits<W>::Pair* stw) {
  const Arith<W, kMode> ar(pc);
  const int tid = threadIdx.x, c = tid % kCols, u = tid / kCols;
  const int col = blockIdx.x * kCols + c;
  // one base pointer per access pattern; the unrolled accesses are then constant offsets from it
  const W* in = batch.in_limb(b) + (unsigned)(u * 256 + col);
  W* out = batch.out_limb(b) + (unsigned)(u * 16 * 256 + col);
  W* t_strided = tile + (unsigned)(u * kCols + c);
  W* t_own = tile + (unsigned)(u * 16 * kCols + c);
  W x[16];
#pragma unroll
  for (int j = 0; j < 16; j++) x[j] = in[j * 16 * 256];
  bool entered = false;
  if constexpr (Loader::kHasSmall && kMode == kArithFp) {
    if (loader.small[b] != 0) {
#pragma unroll
      for (int j = 0; j < 16; j++) x[j] = ar.reduce(ar.enter(x[j]));
      entered = true;
    }
  }
  if (!entered) {
#pragma unroll
    for (int j = 0; j < 16; j++) x[j] = ar.enter(loader.apply(x[j], b, pc));
  }
  __syncthreads();
  radix16_fwd<W, false, kMode, kTwPlain, Loader::kFpBound>(x, stw, 1u, ar);
#pragma unroll
  for (int j = 0; j < 16; j++) t_strided[j * 16 * kCols] = x[j];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 16; j++) x[j] = t_own[j * kCols];
  radix16_fwd<W, false, kMode, kTwPlain, fp_plan_fwd(Loader::kFpBound).out>(x, stw, 16u + (uint32_t)u, ar);
#pragma unroll
  for (int j = 0; j < 16; j++) out[j * 256] = x[j];
}

// Column pass (levels 0 and 1).  grid = (256 / kCols, limbs), block = 16 * kCols.
// Element (h, l) of a limb is word h * 256 + l; the CTA owns kCols adjacent columns.
template <typename W, int kCols, typename Batch, typename Loader>
__global__ void __launch_bounds__(kCols * 16, (sizeof(W) == 8 ? 768 : 1024) / (kCols * 16))
    ntt_fwd_cols_kernel(const Batch batch, const Loader loader,
                        const typename WordTraits<W>::Pair* __restrict__ tw_all,
                        const PrimeConst<W>* __restrict__ pcs) {
  static_assert(sizeof(Batch) + sizeof(Loader) + 2 * sizeof(void*) <= kMaxParameters);
  using Pair = typename WordTraits<W>::Pair;
  __shared__ W tile[256 * kCols];
  __shared__ Pair stw[256];
  grid_dependency_launch();
  const int b = blockIdx.y;
  const uint32_t pi = batch.prime_of(b);
  const PrimeConst<W> pc = pcs[pi];
  for (int k = threadIdx.x; k < 256; k += kCols * 16) stw[k] = __ldg(tw_all + (size_t)pi * kN + k);
  grid_dependency_wait();
  CERIUM_DISPATCH_ARITH(W, pc, ntt_fwd_cols_body, CERIUM_TARGS(kCols, Batch, Loader), (batch, loader, b, pc, tile, stw));
}

__device__ __forceinline__ void prefetch_l2(const void* p) {
#if !defined(CERIUM_EMU)
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
#else
  (void)p;
#endif
}

// What the row pass does with its values, 16 bytes at a time, as the butterflies leave them.  kCanonical (epilogues without operands)
// says whether they are stored reduced to [0, q) or below 4q.  load() fetches what the epilogue reads
// itself: the row pass (radix8_fwd_rows_kernel) calls it for all of a thread's vectors before it finishes any of them.
template <typename W>
struct NoOperands {};
template <typename W>
struct StoreEpilogue {
  static constexpr bool kCanonical = true;
  __device__ __forceinline__ uint32_t scatter_elt() const { return 0u; }
  static constexpr bool kHasOperands = false;
  using Operands = NoOperands<W>;
  __device__ __forceinline__ Operands load(int, int) const { return {}; }
  template <int kMode, int kWords>
  __device__ __forceinline__ void apply_vec(W (&w)[kWords], const Operands&, int, int, uint32_t, const PrimeConst<W>& pc, const Arith<W, kMode>& ar) const {
#pragma unroll
    for (int e = 0; e < kWords; e++) w[e] = ar.template finish_fwd<true>(w[e], pc.one_shoup);
  }
  __device__ __forceinline__ void prefetch(int /*b*/, int /*idx*/) const {}
};

// Stores the transform below 4q.  Only for buffers whose one reader multiplies the values into a
// wide accumulator (the raised digits of a key switch, read by the inner product).
template <typename W>
struct LazyStoreEpilogue {
  static constexpr bool kCanonical = false;
  __device__ __forceinline__ uint32_t scatter_elt() const { return 0u; }
  static constexpr bool kHasOperands = false;
  using Operands = NoOperands<W>;
  __device__ __forceinline__ Operands load(int, int) const { return {}; }
  template <int kMode, int kWords>
  __device__ __forceinline__ void apply_vec(W (&w)[kWords], const Operands&, int, int, uint32_t, const PrimeConst<W>& pc, const Arith<W, kMode>& ar) const {
#pragma unroll
    for (int e = 0; e < kWords; e++) w[e] = ar.template finish_fwd<false>(w[e], pc.one_shoup);
  }
  __device__ __forceinline__ void prefetch(int /*b*/, int /*idx*/) const {}
};

// SuD tail: out = (minuend - NTT(in)) * factor[b] [+ addend]   (all mod q).
// minuend / addend are stacks of limbs: entry b at base + b * stride; entries b >= split belong
// to a second polynomial and use minuend2 / addend2 at (b - split) * stride.
// The row pass with it is bound by its reads (120 MB through DRAM for 70 limbs) and needs all 32 warps of an SM, at whose 64 registers
// it spills 140 bytes a thread (64-bit words; both polynomials, addend and scatter are in one kernel): operands copied to
// shared memory leave 20 (rotation of 35 limbs 275.5 -> 281 us).  Doubles are finished as doubles (integer Shoup product: 35 limbs
// 275.5 -> 274.0, 12 limbs 99.4 -> 98.6, plaintext product with rescale 32.0 -> 31.3).
template <typename W>
struct SudEpilogue {
  static constexpr bool kHasOperands = true;
  const W* minuend;
  const W* minuend2;
  size_t minuend_stride;
  const W* addend;   // may be null
  const W* addend2;  // may be null
  size_t addend_stride;
  int split;         // kSudMaxBatch when there is one polynomial
  uint32_t addend_elt;  // not 0: the addends are read through the Galois automorphism of this element
  uint32_t store_elt;   // not 0: word i of the result is stored at pi(i), the index map of this element, so
                        // the output is the automorphism of the INVERSE element applied to the result
  __device__ __forceinline__ uint32_t scatter_elt() const { return store_elt; }
  // the factor and its Shoup companion; Fp: the centred factor and its quotient by q, as bit patterns of doubles
  W factor[kSudMaxBatch];
  W factor_shoup[kSudMaxBatch];
  // starts the 16 bytes at word idx of the operands towards L2 (called before the transform, whose
  // arithmetic then hides their latency)
  __device__ __forceinline__ void prefetch(int b, int idx) const {
    const bool second = b >= split;
    const int e = second ? b - split : b;
    prefetch_l2((second ? minuend2 : minuend) + (size_t)e * minuend_stride + idx);
    const W* ap = second ? addend2 : addend;
    if (ap != nullptr && addend_elt == 0) prefetch_l2(ap + (size_t)e * addend_stride + idx);
  }
  struct Operands {
    typename RowVec<W>::Vec m, a;
  };
  // The operands of one 16-byte vector (idx0 a multiple of its words): minuend and addend come in as one 16-byte load
  // each.  With an automorphism the aligned group idx0 .. idx0 + kWords - 1 is the image of ONE aligned group of the
  // addend (the index map sends aligned 2^k blocks onto aligned 2^k blocks), so that is one load as well and the
  // words are picked from it.
  __device__ __forceinline__ Operands load(int b, int idx0) const {
    using Vec = typename RowVec<W>::Vec;
    const bool second = b >= split;
    const int e_ = second ? b - split : b;
    const W* mp = (second ? minuend2 : minuend) + (size_t)e_ * minuend_stride;
    const W* ap = second ? addend2 : addend;
    Operands o{};
    o.m = *reinterpret_cast<const Vec*>(mp + idx0);
    if (ap != nullptr) {
      const uint32_t at = addend_elt != 0 ? GaloisGroup<RowVec<W>::kWords>((uint32_t)idx0, addend_elt).at : (uint32_t)idx0;
      o.a = *reinterpret_cast<const Vec*>(ap + (size_t)e_ * addend_stride + at);
    }
    return o;
  }
  template <int kMode, int kWords>
  __device__ __forceinline__ void apply_vec(W (&w)[kWords], const Operands& o, int b, int idx0, uint32_t /*pi*/, const PrimeConst<W>& pc,
                                            const Arith<W, kMode>& ar) const {
    const W* ap = b >= split ? addend2 : addend;
    W m[kWords], a[kWords];
    vec_unpack(o.m, m);
    vec_unpack(o.a, a);
    if (ap != nullptr && addend_elt != 0) {
      W t[kWords];
      vec_unpack(o.a, t);
      GaloisGroup<kWords>((uint32_t)idx0, addend_elt).permute(t, a);
    }
    const W f = factor[b], fs = factor_shoup[b];
#pragma unroll
    for (int e = 0; e < kWords; e++) {
      if constexpr (kMode == kArithFp) {
        // |x| <= 0.51 q after the reduction, the difference within (-0.51 q, 1.51 q), its product below 0.55 q, and with the
        // addend within (-0.55 q, 1.55 q)
        using A = Arith<W, kMode>;
        const double d = __dadd_rn(fp_from_u64(m[e]), -A::d(ar.reduce(w[e])));
        double r = fp_mulmod(d, A::d(f), A::d(fs), ar.nq);
        if (ap != nullptr) {
          r = __dadd_rn(r, fp_from_u64(a[e]));
          if (r >= ar.q) r = __dadd_rn(r, ar.nq);
        }
        w[e] = ar.canonical(r);
      } else {
        const W x = ar.template finish_fwd<false>(w[e], pc.one_shoup);
        W d;
        if (sizeof(W) == 4) {
          // 32-bit words hold primes up to 2^30: m + 4q would pass 2^32, so the transform comes below 2q first
          d = m[e] + pc.q2 - csub<W>(x, pc.q2);
        } else {
          d = m[e] + (pc.q2 + pc.q2) - x;  // x < 4q: positive, and the Shoup product takes any word
        }
        d = csub<W>(mul_shoup_lazy<W>(d, f, fs, pc.q), pc.q);
        if (ap != nullptr) d = add_mod<W>(d, a[e], pc.q);
        w[e] = d;
      }
    }
  }
};

// SuD tail with the argument tables of the reference's launcher (_kernel_sud_1,
// cerium/compiler/backend/kernels/function.cu:123-149): entry b has two inputs, ins[2b] the minuend
// and ins[2b + 1] the coefficient-form limb whose transform is subtracted; factors holds one
// residue per prime of the context, indexed by the entry's prime.
template <typename W>
struct PtrSudEpilogue {
  static constexpr bool kHasOperands = true;
  const W* const* ins;
  const W* factors;
  __device__ __forceinline__ uint32_t scatter_elt() const { return 0u; }
  __device__ __forceinline__ void prefetch(int b, int idx) const { prefetch_l2(ins[2 * b] + idx); }
  struct Operands {
    W m[RowVec<W>::kWords];
  };
  __device__ __forceinline__ Operands load(int b, int idx0) const {
    Operands o;
#pragma unroll
    for (int e = 0; e < RowVec<W>::kWords; e++) o.m[e] = ins[2 * b][idx0 + e];  // caller's limbs may be unaligned
    return o;
  }
  template <int kMode, int kWords>
  __device__ __forceinline__ void apply_vec(W (&w)[kWords], const Operands& o, int /*b*/, int /*idx0*/, uint32_t pi, const PrimeConst<W>& pc,
                                            const Arith<W, kMode>& ar) const {
#pragma unroll
    for (int e = 0; e < kWords; e++) w[e] = apply(ar.template finish_fwd<false>(w[e], pc.one_shoup), o.m[e], pi, pc);
  }
  __device__ __forceinline__ W apply(W x, W m, uint32_t pi, const PrimeConst<W>& pc) const {
    // x < 4q and m < q: bring the difference to [0, q) before the Barrett product
    W d = m + pc.q2 - csub<W>(x, pc.q2);  // (m, m + 2q]
    d = csub<W>(csub<W>(d, pc.q2), pc.q);
    return mul_mod<W>(d, csub<W>(factors[pi], pc.q), pc);
  }
};

template <typename W>
__device__ __forceinline__ void store16(W* dst, const W (&x)[16]);
template <>
__device__ __forceinline__ void store16<uint64_t>(uint64_t* dst, const uint64_t (&x)[16]) {
  ulonglong2* d = reinterpret_cast<ulonglong2*>(dst);
#pragma unroll
  for (int j = 0; j < 8; j++) d[j] = make_ulonglong2(x[2 * j], x[2 * j + 1]);
}
template <>
__device__ __forceinline__ void store16<uint32_t>(uint32_t* dst, const uint32_t (&x)[16]) {
  uint4* d = reinterpret_cast<uint4*>(dst);
#pragma unroll
  for (int j = 0; j < 4; j++) d[j] = make_uint4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
}
template <typename W>
__device__ __forceinline__ void load16(const W* src, W (&x)[16]);
template <>
__device__ __forceinline__ void load16<uint64_t>(const uint64_t* src, uint64_t (&x)[16]) {
  const ulonglong2* s = reinterpret_cast<const ulonglong2*>(src);
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const ulonglong2 v = s[j];
    x[2 * j] = v.x;
    x[2 * j + 1] = v.y;
  }
}
template <>
__device__ __forceinline__ void load16<uint32_t>(const uint32_t* src, uint32_t (&x)[16]) {
  const uint4* s = reinterpret_cast<const uint4*>(src);
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const uint4 v = s[j];
    x[4 * j] = v.x;
    x[4 * j + 1] = v.y;
    x[4 * j + 2] = v.z;
    x[4 * j + 3] = v.w;
  }
}

template <typename W, int kRows, bool kStage, typename Batch, typename Epilogue>
__device__ __forceinline__ void ntt_fwd_rows_body(const Batch& batch, int b, const PrimeConst<W>& pc,
                                                  RowsBuffer<W, kRows, kStage>& buf,
                                                  const typename WordTraits<W>::Pair* tw,
                                                  const typename WordTraits<W>::Pair* twr) {
  using RV = RowVec<W>;
  using Vec = typename RV::Vec;
  W* tile = buf.tile;
  constexpr int kMode = kArithStrict;
  const Arith<W, kMode> ar(pc);
  const int tid = threadIdx.x, r = tid >> 4, u = tid & 15;
  const int h = blockIdx.x * kRows + r;
  const W* row = batch.in_limb(b) + (unsigned)(h * 256 + u);
  W* drow = batch.out_limb(b) + (unsigned)(h * 256);
  W* trow = tile + (unsigned)(r * kRowPitch);
  W* t_strided = trow + u;             // row_pos(j * 16 + u) = j * 17 + u
  W* t_own = trow + (unsigned)(u * 17);  // row_pos(u * 16 + j) = u * 17 + j
  W x[16];
#pragma unroll
  for (int j = 0; j < 16; j++) x[j] = row[j * 16];
  if constexpr (kStage) {
    row_twiddles_wait();
    radix16_fwd<W, false, kMode, kTwGroup>(x, buf.tw.group[r], 0u, ar);
  } else {
    radix16_fwd<W, true, kMode, kTwPlain>(x, tw, 256u + (uint32_t)h, ar);
  }
#pragma unroll
  for (int j = 0; j < 16; j++) t_strided[j * 17] = x[j];
  __syncwarp();  // a row's 16 threads share a warp; no other warp touches its staging rows
#pragma unroll
  for (int j = 0; j < 16; j++) x[j] = t_own[j];
  // level 3: this thread's 15 twiddles from the lane-interleaved table of row h
  if constexpr (kStage) radix16_fwd<W, false, kMode, kTwLane>(x, buf.tw.lane[r] + u, 0u, ar);
  else radix16_fwd<W, true, kMode, kTwLane>(x, twr + ((size_t)h * 15 * 16 + u), 0u, ar);
#pragma unroll
  for (int j = 0; j < 16; j++) x[j] = ar.template finish_fwd<Epilogue::kCanonical>(x[j], pc.one_shoup);
  // own 16 words -> swizzled vectors -> coalesced vectors
  __syncwarp();  // a row's 16 threads share a warp; no other warp touches its staging rows
  Vec* vrow = reinterpret_cast<Vec*>(tile + r * kRowPitch);  // same private region as the exchange rows
#pragma unroll
  for (int jj = 0; jj < RV::kPerThread; jj++)
    vrow[row_vec_slot<W>(u * RV::kPerThread + jj)] = vec_pack(&x[jj * RV::kWords]);
  __syncwarp();  // a row's 16 threads share a warp; no other warp touches its staging rows
#pragma unroll
  for (int k = 0; k < RV::kPerThread; k++) reinterpret_cast<Vec*>(drow)[u + 16 * k] = vrow[row_vec_slot<W>(u + 16 * k)];
}

// Row pass (levels 2 and 3) of 32-bit words whose epilogue reads nothing: reads the column pass's result from the batch's `in` stack
// and writes the finished transform to its `out` stack (the two may be the same buffer).
// grid = (256 / kRows, limbs), block = 16 * kRows; 16 threads own one row.
template <typename W, int kRows, bool kStage, typename Batch, typename Epilogue>
__global__ void __launch_bounds__(kRows * 16, 1024 / (kRows * 16))
    ntt_fwd_rows_kernel(const Batch batch, const typename WordTraits<W>::Pair* __restrict__ tw_all,
                        const typename WordTraits<W>::Pair* __restrict__ twr_all,
                        const PrimeConst<W>* __restrict__ pcs) {
  static_assert(sizeof(W) == 4, "64-bit words have radix8_fwd_rows_kernel");
  using Pair = typename WordTraits<W>::Pair;
  __shared__ RowsBuffer<W, kRows, kStage> buf;
  grid_dependency_launch();
  // From the last limb to the first, against the direction of the column pass: what that pass wrote last is still in L2
  // and is read, and overwritten, before it goes to memory.  The reader of a result larger than L2 then starts at the
  // first limb for the same reason.  (Rotation of 35 limbs 367 -> 355.6 us, transform of 384 limbs 190.6 -> 187.2 us.)
  const int b = (int)(gridDim.y - 1 - blockIdx.y);
  const uint32_t pi = batch.prime_of(b);
  const PrimeConst<W> pc = pcs[pi];
  const Pair* tw = tw_all + (size_t)pi * kN;
  const Pair* twr = twr_all + (size_t)pi * kRowTwPerPrime;
  if constexpr (kStage) row_twiddles_start(buf.tw, tw, twr, blockIdx.x * kRows);
  grid_dependency_wait();
  ntt_fwd_rows_body<W, kRows, kStage, Batch, Epilogue>(batch, b, pc, buf, tw, twr);
}

// ---------------------------------------------------------------------------------------
// inverse transform
// ---------------------------------------------------------------------------------------

template <typename W, int kMode, int kRows, bool kStage, typename Batch>
__device__ __forceinline__ void ntt_inv_rows_body(const Batch& batch, int b, const PrimeConst<W>& pc, RowsBuffer<W, kRows, kStage>& buf,
                                                  const typename WordTraits<W>::Pair* twi,
                                                  const typename WordTraits<W>::Pair* twri) {
  using RV = RowVec<W>;
  using Vec = typename RV::Vec;
  constexpr bool kStaged = kStage && (sizeof(W) == 4 || kMode == kArithFp);
  W* tile = buf.tile;
  const Arith<W, kMode> ar(pc);
  const int tid = threadIdx.x, r = tid >> 4, u = tid & 15;
  const int h = blockIdx.x * kRows + r;
  const W* limb_in = batch.in_limb(b);
  const W* src = limb_in + h * 256;
  const uint32_t elt = batch.gather_elt();
  W* dst = batch.out_limb(b) + h * 256;
  W* trow = tile + r * kRowPitch;
  // coalesced vectors -> swizzled staging -> own 16 consecutive words
  Vec* vrow = reinterpret_cast<Vec*>(tile + r * kRowPitch);  // same private region as the exchange rows
  Vec in[RV::kPerThread];
  if (elt == 0) {
#pragma unroll
    for (int k = 0; k < RV::kPerThread; k++) in[k] = reinterpret_cast<const Vec*>(src)[u + 16 * k];
  } else {
    // the automorphism maps aligned groups of words onto aligned groups: one vector, its words permuted
#pragma unroll
    for (int k = 0; k < RV::kPerThread; k++)
      in[k] = *reinterpret_cast<const Vec*>(limb_in + GaloisGroup<RV::kWords>((uint32_t)(h * 256 + (u + 16 * k) * RV::kWords), elt).at);
#pragma unroll
    for (int k = 0; k < RV::kPerThread; k++) {
      W t[RV::kWords], w[RV::kWords];
      vec_unpack(in[k], t);
      GaloisGroup<RV::kWords>((uint32_t)(h * 256 + (u + 16 * k) * RV::kWords), elt).permute(t, w);
      in[k] = vec_pack(w);
    }
  }
#pragma unroll
  for (int k = 0; k < RV::kPerThread; k++) vrow[row_vec_slot<W>(u + 16 * k)] = in[k];
  __syncwarp();
  W x[16];
#pragma unroll
  for (int jj = 0; jj < RV::kPerThread; jj++)
    vec_unpack(vrow[row_vec_slot<W>(u * RV::kPerThread + jj)], &x[jj * RV::kWords]);
#pragma unroll
  for (int j = 0; j < 16; j++) x[j] = ar.enter(x[j]);
  if (kStaged) row_twiddles_wait();
  radix16_inv<W, !kStaged, kMode, 0, kTwLane, kFpCanon>(
      x, kStaged ? buf.tw.lane[kStaged ? r : 0] + u : twri + ((size_t)h * (kMode == kArithFp ? 8 : 15) * 16 + u), 0u, ar);
  if (kMode == kArithFp) fp_reduce_masked<W, kMode>(x, kFpInvRowsExMask, ar);
  __syncwarp();
  W* t_own = trow + (unsigned)(u * 17);  // row_pos(u * 16 + j) = u * 17 + j
  W* t_strided = trow + u;             // row_pos(j * 16 + u) = j * 17 + u
#pragma unroll
  for (int j = 0; j < 16; j++) t_own[j] = x[j];
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 16; j++) x[j] = t_strided[j * 17];
  radix16_inv<W, !kStaged, kMode, 4, kStaged ? kTwGroup : kTwPlain, kFpInvL3>(x, kStaged ? buf.tw.group[kStaged ? r : 0] : twi, 256u + (uint32_t)h, ar);
  W* dcol = dst + u;
#pragma unroll
  for (int j = 0; j < 16; j++) dcol[j * 16] = x[j];
}

// Row pass (levels 3 and 2): in -> out; values leave below 2q (strict; 4q for 64-bit words) or below 2^10 q (lazy).
template <typename W, int kRows, bool kStage, typename Batch>
__global__ void __launch_bounds__(kRows * 16, 1024 / (kRows * 16))
    ntt_inv_rows_kernel(const Batch batch, const typename WordTraits<W>::Pair* __restrict__ twi_all,
                        const typename WordTraits<W>::Pair* __restrict__ twri_all,
                        const PrimeConst<W>* __restrict__ pcs) {
  using Pair = typename WordTraits<W>::Pair;
  __shared__ RowsBuffer<W, kRows, kStage> buf;
  grid_dependency_launch();
  const int b = blockIdx.y;
  const uint32_t pi = batch.prime_of(b);
  const PrimeConst<W> pc = pcs[pi];
  const Pair* twi = twi_all + (size_t)pi * kN;
  const Pair* twri = twri_all + (size_t)pi * kRowTwPerPrime;
  if constexpr (kStage)
    if (sizeof(W) == 4 || pc.fp_ok != 0) row_twiddles_start(buf.tw, twi, twri, blockIdx.x * kRows);
  grid_dependency_wait();
  CERIUM_DISPATCH_ARITH(W, pc, ntt_inv_rows_body, CERIUM_TARGS(kRows, kStage, Batch), (batch, b, pc, buf, twi, twri));
}

// Optional per-limb scalar of the finished inverse transform (exact base conversion wants x * [Qhat^-1] mod q):
// it is folded into the two constants of the last layer, which every value passes anyway.
template <typename W>
struct InvScale {
  const W* last;         // per batch entry the four words of Arith::inv_last, or null: plain N^-1
  const W* add;          // per batch entry, added to the scaled value modulo q (rounding term), may be null
};

// Small tiles of 32-bit words let the next kernel in late (see grid_dependency_launch): 30 limbs 11.60 -> 11.44 us, rotation of 16
// limbs with as many extension limbs 63.0 -> 59.8, of 32 96.7 -> 93.5; 64-bit words lose (24 limbs 15.18 -> 15.35).
template <typename W, int kCols>
constexpr bool kInvColsLate = sizeof(W) == 4 && kCols < NttCfg<W>::kCols;

template <typename W, int kMode, int kCols, typename Batch>
__device__ __forceinline__ void ntt_inv_cols_body(const Batch& batch, const InvScale<W>& sc, int b,
                                                  const PrimeConst<W>& pc, W* tile,
                                                  const typename WordTraits<W>::Pair* stw) {
  const Arith<W, kMode> ar(pc);
  const W q = pc.q;
  const int tid = threadIdx.x, c = tid % kCols, u = tid / kCols;
  const int col = blockIdx.x * kCols + c;
  W* buf_own = batch.out_limb(b) + (unsigned)(u * 16 * 256 + col);
  W* buf_strided = batch.out_limb(b) + (unsigned)(u * 256 + col);
  W* t_strided = tile + (unsigned)(u * kCols + c);
  W* t_own = tile + (unsigned)(u * 16 * kCols + c);
  W x[16];
#pragma unroll
  for (int j = 0; j < 16; j++) {
    x[j] = buf_own[j * 256];
    if (kMode == kArithLazy) x[j] = reduce_lazy(x[j], pc.one_shoup, (W)0 - pc.q);  // back below 4q for the second pass
  }
  __syncthreads();
  radix16_inv<W, false, kMode, 0, kTwPlain, kFpInvMid>(x, stw, 16u + (uint32_t)u, ar);
  if (kMode == kArithFp) fp_reduce_masked<W, kMode>(x, kFpInvColsExMask, ar);
#pragma unroll
  for (int j = 0; j < 16; j++) t_own[j * kCols] = x[j];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 16; j++) x[j] = t_strided[j * 16 * kCols];
  if (kInvColsLate<W, kCols>) grid_dependency_launch();
  W last[4];
  if (sc.last != nullptr) {
#pragma unroll
    for (int e = 0; e < 4; e++) last[e] = __ldg(sc.last + 4 * b + e);
  } else if (kMode == kArithFp) {
    last[0] = pc.fp_ninv, last[1] = pc.fp_ninv_q, last[2] = pc.fp_w1ninv, last[3] = pc.fp_w1ninv_q;
  } else {
    last[0] = pc.ninv, last[1] = pc.ninv_shoup, last[2] = pc.w1ninv, last[3] = pc.w1ninv_shoup;
  }
  radix16_inv_final<W, kMode, kFpInvL1>(x, stw, last, ar);
  if (sc.add != nullptr) {
    const W a = __ldg(sc.add + b);
#pragma unroll
    for (int j = 0; j < 16; j++) x[j] = add_mod<W>(x[j], a, q);
  }
#pragma unroll
  for (int j = 0; j < 16; j++) buf_strided[j * 16 * 256] = x[j];
}

// Column pass (levels 1 and 0), in place on the output limb of the row pass; scales by
// N^-1 and reduces to [0, q).
template <typename W, int kCols, typename Batch>
__global__ void __launch_bounds__(kCols * 16, (sizeof(W) == 8 ? 768 : 1024) / (kCols * 16))
    ntt_inv_cols_kernel(const Batch batch, const InvScale<W> sc,
                        const typename WordTraits<W>::Pair* __restrict__ twi_all,
                        const PrimeConst<W>* __restrict__ pcs) {
  using Pair = typename WordTraits<W>::Pair;
  __shared__ W tile[256 * kCols];
  __shared__ Pair stw[256];
  if (!kInvColsLate<W, kCols>) grid_dependency_launch();
  // against the direction of the row pass, as in the forward transform
  const int b = (int)(gridDim.y - 1 - blockIdx.y);
  const uint32_t pi = batch.prime_of(b);
  const PrimeConst<W> pc = pcs[pi];
  for (int k = threadIdx.x; k < 256; k += kCols * 16) stw[k] = __ldg(twi_all + (size_t)pi * kN + k);
  grid_dependency_wait();
  CERIUM_DISPATCH_ARITH(W, pc, ntt_inv_cols_body, CERIUM_TARGS(kCols, Batch), (batch, sc, b, pc, tile, stw));
}

}  // namespace cerium
