// Row pass of the raised digits and their inner product with the evaluation key in one kernel.
//
// A warp (two of them where there are many digits) owns one row (256 words) of one output limb.  It walks the digits: takes
// the row of the digit's column pass through the last eight layers and multiplies the result with the two key rows into
// sums that stay in its registers, so the raised digits are never written in transformed form (302 MB written and read again
// for 24 digits of 24 limbs).
//
// Bound by memory: 482 MB for 7 digits on 40 limbs of 64-bit words, 970 MB for 24 digits on 25 (451 MB through DRAM, and
// 950 with the additions of a multiplication; 101 and 204 us in a profiler, half of the issue slots).  The twiddles of a row serve every digit
// from shared memory (read through L1 for every digit they took the gain away: 147 us for the first shape, the two kernels 143).  A lane keeps 8 words and 16 sums, so that 16 warps fit an SM at 128 registers; with 16 words to a lane
// it would be 8.  The next digit's row is on its way (cp.async) while one is worked on, and the key rows are asked for before
// the butterflies that come first.  20 warps at 96 registers spill and are slower (rotation of 35 limbs 315 us against the 301 of then).
// Two rows to a CTA: whole rounds of CTAs are smaller than with four (12 limbs 117.3 us of then against 122.4).
// Key words are the first to leave L2 by an explicit priority (with .cs alone rotation of 35 limbs 296.0 us, now 293.4; 24 limbs with
// one-limb digits 431 -> 428).
// Measured, row pass + inner product -> this kernel: rotation of 35 limbs 344 -> 291 us, multiplication of 24 limbs with
// one-limb digits 542 -> 433, rotation of 51 32-bit limbs 200 -> 183; of 35 limbs of 60-bit primes 454 -> 446.  When it is used:
// rows_with_inner (api_keyswitch.cu).
#pragma once
#include "ewise_kernels.cuh"
#include "ntt_radix8.cuh"

namespace cerium {

// Sums of products of residues (integers: below 4q) with key words; 64 bits, so that partial sums of a row can be put
// together.
//   32-bit words: the products themselves, one reduction at the end.
//   64-bit integers: every product x = y k < 4 q^2 is reduced: t = x / 2^(b - 2), q of b bits (kKeySumBits to 60), is below 2^64, the
//   quotient hi(t * floor(2^(b + 62) / q)) is short by less than 1/2 + 1 + 1 + 2 (t, the factor, the product, mulhi_approx64), so the
//   remainder is below 4.5 q, and a sum below 5q + 2^32 stays there when 5q leaves it where its high word says so (csub_high).
//   These are the primes from 2^50 on, and with integer butterflies everywhere smaller ones too: a plan with one that is too
//   small for the shift, which passes over a whole word, keeps the two kernels (rows_with_inner).
//   Sums of two words take 64 registers and leave none for the key words that are on their way.
//   Fp: every product is below 7/8 q (Arith::product), eight of them on a reduced sum stay below 8 q: exact.
constexpr int kKeySumBits = 34;
template <typename W, int kMode>
struct KeySum {
  static constexpr int kTerms = 1 << 30;  // on a reduced sum
  using A = Arith<W, kMode>;
  const A& ar;
  uint64_t mu;  // 64-bit integers
  int shift;    // ... what is left of b - 2 when a word has been passed over
  __device__ __forceinline__ KeySum(const A& a, const PrimeConst<W>& pc) : ar(a), mu(0), shift(0) {
    if constexpr (sizeof(W) == 8) {
      const int bits = 64 - __clzll((long long)pc.q);
      mu = pc.mu_hi << (bits - 2) | pc.mu_lo >> (66 - bits);
      shift = bits - 2 - 32;
    }
  }
  __device__ __forceinline__ void add(uint64_t& s, W y, W k) const {
    if constexpr (sizeof(W) == 4) {
      s += (uint64_t)y * k;
    } else {
      const uint64_t lo = y * k, hi = WordTraits<W>::mulhi(y, k);
      const uint64_t t = (uint64_t)__funnelshift_r((uint32_t)hi, (uint32_t)(hi >> 32), shift) << 32 |
                         __funnelshift_r((uint32_t)(lo >> 32), (uint32_t)hi, shift);
      s = csub_high(s + (lo + mulhi_approx64(t, mu) * ar.nq), ar.q4 + ar.q);
    }
  }
  __device__ __forceinline__ void reduce(uint64_t&) const {}
  __device__ __forceinline__ void join(uint64_t& s, uint64_t t) const {
    if constexpr (sizeof(W) == 4) s += t;
    else s = csub_high(s + t, ar.q4 + ar.q);
  }
  __device__ __forceinline__ W finish(uint64_t s, const PrimeConst<W>& pc) const {
    if constexpr (sizeof(W) == 4) return barrett2<W>((W)(s >> 32), (W)s, pc);
    else return reduce_word<W>(s, pc);
  }
};
template <>
struct KeySum<uint64_t, kArithFp> {
  static constexpr int kTerms = 8;
  using A = Arith<uint64_t, kArithFp>;
  const A& ar;
  __device__ __forceinline__ KeySum(const A& a, const PrimeConst<uint64_t>&) : ar(a) {}
  __device__ __forceinline__ void add(uint64_t& s, uint64_t y, uint64_t k) const {
    s = A::u(__dadd_rn(A::d(s), ar.product(A::d(y), fp_from_u64(k))));
  }
  __device__ __forceinline__ void reduce(uint64_t& s) const { s = ar.reduce(s); }
  __device__ __forceinline__ void join(uint64_t& s, uint64_t t) const { s = A::u(__dadd_rn(A::d(s), A::d(t))); }
  __device__ __forceinline__ uint64_t finish(uint64_t s, const PrimeConst<uint64_t>&) const {
    return ar.canonical(fp_reduce(A::d(s), ar.qinv, ar.nq));
  }
};

// A row's shared memory: the digit that is worked on and the next one on its way, and the twiddles of the row, which serve
// every digit.  Pair (1 << t) + g is entry ((256 + h) << t) + g of the table, layers t = 0..7.  64-bit words: layers 0..5
// only; Fp has the last two without their quotients after them, word (1 << t) + g - 64 of `late`.  The integer butterflies of
// 64-bit words read those from global memory.
template <typename W>
struct alignas(16) RaisedRow {
  static constexpr int kPairs = sizeof(W) == 8 ? 64 : 256;
  W buf[2][kRaisedPitch];
  typename WordTraits<W>::Pair tw[kPairs];
  W late[sizeof(W) == 8 ? 192 : 2];
};
template <typename W, bool kFp>
__device__ __forceinline__ void raised_twiddles(RaisedRow<W>& row, const typename WordTraits<W>::Pair* tw, int h) {
  const int lane = threadIdx.x & 31;
  const uint32_t S = 256u + (uint32_t)h;
#pragma unroll
  for (int k = 0; k < (sizeof(W) == 8 && !kFp ? 2 : 8); k++) {
    const int i = k * 32 + lane;
    if (i == 0) continue;
    const int t = 31 - __clz(i);
    const auto w = __ldg(tw + ((S << t) + (uint32_t)(i - (1 << t))));
    if (i < RaisedRow<W>::kPairs) row.tw[i] = w;
    else row.late[sizeof(W) == 8 ? i - 64 : 0] = w.x;
  }
  if (sizeof(W) == 8 && !kFp && lane < 24)  // the others on their way: lines of 128 bytes, 8 of layer 6 and 16 of layer 7
    prefetch_l2(lane < 8 ? tw + (S * 64u + 8u * (uint32_t)lane) : tw + (S * 128u + 8u * (uint32_t)(lane - 8)));
}

// The eight layers of row h.  In: x[j] = word j * 32 + lane.  Out: x[r] = word (r / 4) * 128 + lane * 4 + r % 4, Fp:
// |x| <= 0.51 q, integers: below 4q.
template <typename W, int kMode>
__device__ __forceinline__ void raised_row(W (&x)[8], W* ex, const RaisedRow<W>& row, const typename WordTraits<W>::Pair* tw, int h,
                                           const Arith<W, kMode>& ar, const PrimeConst<W>& pc) {
  using RV = RowVec<W>;
  constexpr FpPassPlan plan = fp_plan_row(kFpRaisedMid, kFpLaneK32);
  const int lane = threadIdx.x & 31;
  radix8_fwd<W, kMode, 0, kFpRaisedMid>(x, row.tw, 1, ar);
#pragma unroll
  for (int j = 0; j < 8; j++) ex[raised_pos<W>(j * 32 + lane)] = x[j];
  __syncwarp();
  const int own = (lane >> 2) * 32 + (lane & 3);
#pragma unroll
  for (int j = 0; j < 8; j++) x[j] = ex[raised_pos<W>(own + 4 * j)];
  radix8_fwd<W, kMode, 3, kFpRaisedMid>(x, row.tw, 8 + (lane >> 2), ar);
#pragma unroll
  for (int j = 0; j < 8; j++) ex[raised_pos<W>(own + 4 * j)] = x[j];
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 8; k += RV::kWords)
    vec_unpack(*reinterpret_cast<const typename RV::Vec*>(ex + raised_pos<W>((k >> 2) * 128 + lane * 4 + (k & 3))), &x[k]);
  __syncwarp();  // the buffer is free for the digit after the next
  // One group of four after the other, its twiddles with it: with those of both at once (late_fwd) the sums leave them no registers
  // (multiplication of 24 limbs with one-limb digits 384.5 -> 392.7 us, rotation of 20 limbs 282.0 -> 286.9).
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int g = k * 32 + lane;
    W w6[2], w7[4];  // twiddles, each with its companion
    if constexpr (kMode == kArithFp) {
      W v[2];
      vec_unpack(*reinterpret_cast<const typename RV::Vec*>(row.late + 64 + 2 * g), v);
      w6[0] = row.late[g], w6[1] = ar.quotient(w6[0]);
      w7[0] = v[0], w7[1] = ar.quotient(v[0]), w7[2] = v[1], w7[3] = ar.quotient(v[1]);
    } else {
      constexpr bool kNear = sizeof(W) == 4;
      const auto* at6 = kNear ? row.tw + (64 + g) % RaisedRow<W>::kPairs : tw + ((256 + h) * 64 + g);
      const auto* at7 = kNear ? row.tw + (128 + 2 * g) % RaisedRow<W>::kPairs : tw + ((256 + h) * 128 + 2 * g);
      const auto a = at6[0], b = at7[0], c = at7[1];
      w6[0] = a.x, w6[1] = a.y, w7[0] = b.x, w7[1] = b.y, w7[2] = c.x, w7[3] = c.y;
    }
    if (kMode == kArithFp && plan.before[6]) {
#pragma unroll
      for (int j = 0; j < 4; j++) x[4 * k + j] = ar.reduce(x[4 * k + j]);
    }
    ar.fwd(x[4 * k], x[4 * k + 2], w6[0], w6[1]);
    ar.fwd(x[4 * k + 1], x[4 * k + 3], w6[0], w6[1]);
    if (kMode == kArithFp && plan.before[7]) {
#pragma unroll
      for (int j = 0; j < 4; j++) x[4 * k + j] = ar.reduce(x[4 * k + j]);
    }
    ar.fwd(x[4 * k], x[4 * k + 1], w7[0], w7[1]);
    ar.fwd(x[4 * k + 2], x[4 * k + 3], w7[2], w7[3]);
  }
#pragma unroll
  for (int j = 0; j < 8; j++) {
    if constexpr (kMode == kArithFp) x[j] = ar.reduce(x[j]);
    else x[j] = ar.template finish_fwd<false>(x[j], pc.one_shoup);
  }
}

// The inputs of a multiplication (a0, a1) (b0, b1), a1 being `own` of the inner product: the switched polynomial is a1 b1, its
// own limbs are multiplied as they are read, and a0 b0 and a0 b1 + a1 b0 join the sums, so that the three products of the
// tensor are never stored.  b0 null: none of that, as cerium_hmult has it where two warps share a row.  That variant is compiled with
// these products all the same: left out, it spills 72 bytes for 12 (24 limbs with as many digits 432.2 -> 434.5 us).
template <typename W>
struct TensorOf {
  const W* a0;
  const W* b0;
  const W* b1;
};

// Gives up the 128 bytes at p, a whole line of a buffer that is written before it is read again.  On the CPU they are
// overwritten, so that a kernel that reads them all the same computes wrong results there.
__device__ __forceinline__ void discard_line(const void* p) {
#if !defined(CERIUM_EMU)
  asm volatile("discard.global.L2 [%0], 128;" ::"l"(p) : "memory");
#else
  std::memset(const_cast<void*>(p), 0xa5, 128);
#endif
}

// kSplit warps share a row: warp `part` takes every kSplit-th digit, and finishes polynomial `part` from the sums of all of
// them (kSplit = 1: both).
template <typename W, int kMode, int kSplit>
__device__ __forceinline__ void raised_inner_body(const InnerProductArgs<W>& g, const TensorOf<W>& tensor, int b, int h, int part, const PrimeConst<W>& pc,
                                                  RaisedRow<W>* rows, const typename WordTraits<W>::Pair* tw) {
  const Arith<W, kMode> ar(pc);
  using Sum = KeySum<W, kMode>;
  const Sum ks(ar, pc);
  constexpr int kWords = RowVec<W>::kWords;
  const int lane = threadIdx.x & 31;
  RaisedRow<W>& row = rows[part];
  raised_twiddles<W, kMode == kArithFp>(row, tw, h);
  grid_dependency_wait();
  const size_t at = (size_t)(h * 256 + lane * 4);  // this lane's first quad; the second one is 128 words on
  const W* rp = g.raised + (size_t)b * g.raised_limb_stride + h * 256;
  const W* kp = g.evk + (size_t)b * g.evk_limb_stride + at;
  const int own_digit = g.own_digit[b];
  uint64_t sum[2][8];
#pragma unroll
  for (int j = 0; j < 8; j++) sum[0][j] = sum[1][j] = 0;  // 0.0 as well
  // the digits without the limb's own one, whose transform the caller has
  const int own = own_digit < 0 ? g.dnum : own_digit, digits = g.dnum - (own_digit < 0 ? 0 : 1);
  auto digit = [&](int e) { return e < own ? e : e + 1; };
  auto fetch = [&](int e, int into) {
    if (e < digits) {
#pragma unroll
      for (int j = 0; j < 8 / kWords; j++)
        copy_async<16>(row.buf[into] + (j * 32 + lane) * kWords, rp + (size_t)digit(e) * g.raised_digit_stride + (j * 32 + lane) * kWords);
    }
  };
  fetch(part, 0);
  auto fetch_key = [&](Quad<W> (&to)[2][2], int d) {
#pragma unroll
    for (int p = 0; p < 2; p++)
#pragma unroll
      for (int k = 0; k < 2; k++)
        to[p][k] = quad_load_once(kp + (size_t)d * g.evk_digit_stride + (size_t)p * g.evk_poly_stride + k * 128);
  };
  // What is known without a transform comes first, while the first digit is on its way: the own digit's products (first warp)
  // and what joins the sums (last warp).  In the middle of the loop the own digit cost registers (200 bytes spilled), and at the
  // end every load is waited for: rotation of 35 limbs 302 -> 297 us, of 12 limbs 118.6 -> 116.7.
  if (own_digit >= 0) {
    Quad<W> own_key[2][2];
    if (part == 0) fetch_key(own_key, own_digit);
    const size_t limb = (size_t)b * g.own_stride + at;
    if (tensor.b0 != nullptr) {
      Quad<W> a0[2], a1[2], b0[2], b1[2];
#pragma unroll
      for (int k = 0; k < 2; k++) {
        a1[k] = quad_load(g.own + limb + 128 * k);
        b1[k] = quad_load(tensor.b1 + limb + 128 * k);
        if (part == kSplit - 1) {
          a0[k] = quad_load(tensor.a0 + limb + 128 * k);
          b0[k] = quad_load(tensor.b0 + limb + 128 * k);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const W x1 = a1[j >> 2].v[j & 3], z1 = b1[j >> 2].v[j & 3];
        if (part == 0) {
          const W y = ar.enter(mul_mod<W>(x1, z1, pc));
          ks.add(sum[0][j], y, own_key[0][j >> 2].v[j & 3]);
          ks.add(sum[1][j], y, own_key[1][j >> 2].v[j & 3]);
        }
        if (part == kSplit - 1) {
          const W x0 = a0[j >> 2].v[j & 3], z0 = b0[j >> 2].v[j & 3];
          ks.add(sum[0][j], ar.enter(mul_mod<W>(x0, z0, pc)), g.add_factor[b]);
          Acc2<W> acc;
          acc.clear();
          acc.mad(x0, z1);
          acc.mad(x1, z0);
          ks.add(sum[1][j], ar.enter(barrett2<W>(acc.hi(), acc.lo(), pc)), g.add_factor[b]);
        }
      }
    } else {
      if (part == 0) {
#pragma unroll
        for (int k = 0; k < 2; k++) {
          Quad<W> t;
          if (g.own_elt != 0) {
            // the automorphism maps aligned groups of words onto aligned groups
            const GaloisGroup<4> gg((uint32_t)at + 128u * (uint32_t)k, g.own_elt);
            gg.permute(quad_load(g.own + (size_t)b * g.own_stride + gg.at).v, t.v);
          } else {
            t = quad_load_once(g.own + limb + 128 * k);
          }
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const W y = ar.enter(t.v[e]);
            ks.add(sum[0][4 * k + e], y, own_key[0][k].v[e]);
            ks.add(sum[1][4 * k + e], y, own_key[1][k].v[e]);
          }
        }
      }
      if (b < g.add_limbs && part == kSplit - 1) {
        const W* adds[2] = {g.add0, g.add1};
#pragma unroll
        for (int p = 0; p < 2; p++) {
          if (adds[p] == nullptr) continue;
#pragma unroll
          for (int k = 0; k < 2; k++) {
            const Quad<W> t = quad_load_once(adds[p] + (size_t)b * g.add_stride + at + 128 * k);
#pragma unroll
            for (int e = 0; e < 4; e++) ks.add(sum[p][4 * k + e], ar.enter(t.v[e]), g.add_factor[b]);
          }
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 8; j++) {
      ks.reduce(sum[0][j]);
      ks.reduce(sum[1][j]);
    }
  }
  int n = 0;  // terms so far
#pragma unroll 1
  for (int e = part; e < digits; e += kSplit, n++) {
    Quad<W> key[2][2];
    fetch_key(key, digit(e));
    W y[8];
    row_twiddles_wait();             // this digit is here, and the first time the twiddles
    fetch(e + kSplit, (n & 1) ^ 1);  // its buffer was the previous digit's
    // The row was read for the last time: its lines, which the column pass left dirty in L2, need not go to memory (50 MB of a
    // rotation of 35 limbs: 294.4 -> 289.0 us; 51 32-bit limbs 186.7 -> 182.0, 24 limbs with one-limb digits 428.3 / 429.5).
    if (lane < 2 * (int)sizeof(W)) discard_line(rp + (size_t)digit(e) * g.raised_digit_stride + lane * (128 / (int)sizeof(W)));
    W* ex = row.buf[n & 1];
#pragma unroll
    for (int j = 0; j < 8; j++) y[j] = ex[j * 32 + lane];
    __syncwarp();
    raised_row<W, kMode>(y, ex, row, tw, h, ar, pc);
    if (n != 0 && n % Sum::kTerms == 0) {
#pragma unroll
      for (int j = 0; j < 8; j++) {
        ks.reduce(sum[0][j]);
        ks.reduce(sum[1][j]);
      }
    }
#pragma unroll
    for (int p = 0; p < 2; p++)
#pragma unroll
      for (int j = 0; j < 8; j++) ks.add(sum[p][j], y[j], key[p][j >> 2].v[j & 3]);
  }
  auto finish = [&](uint64_t (&s)[8], W* out) {
#pragma unroll
    for (int k = 0; k < 2; k++) {
      Quad<W> o;
#pragma unroll
      for (int e = 0; e < 4; e++) o.v[e] = ks.finish(s[4 * k + e], pc);
      W* to = out + 128 * k;
      if (g.accumulate != 0) {
        const Quad<W> t = quad_load(to);
#pragma unroll
        for (int e = 0; e < 4; e++) o.v[e] = add_mod<W>(o.v[e], t.v[e], pc.q);
      }
      quad_store(to, o);
    }
  };
  if constexpr (kSplit == 1) {
    finish(sum[0], g.out0.at(b, (int)at));
    finish(sum[1], g.out1.at(b, (int)at));
  } else {
    // the sums take the place of the digits and the twiddles; words of a lane 256 bytes apart
    static_assert(sizeof(RaisedRow<W>) >= 2 * 8 * 32 * 8, "room for the sums of a warp");
    uint64_t* mine = reinterpret_cast<uint64_t*>(&row) + lane;
    __syncwarp();
#pragma unroll
    for (int p = 0; p < 2; p++)
#pragma unroll
      for (int j = 0; j < 8; j++) {
        ks.reduce(sum[p][j]);
        mine[(p * 8 + j) * 32] = sum[p][j];
      }
    __syncthreads();
    if (part < 2) {
      uint64_t total[8];
#pragma unroll
      for (int j = 0; j < 8; j++) {
        total[j] = 0;
#pragma unroll
        for (int o = 0; o < kSplit; o++) ks.join(total[j], (reinterpret_cast<const uint64_t*>(rows + o) + lane)[(part * 8 + j) * 32]);
      }
      finish(total, (part == 0 ? g.out0 : g.out1).at(b, (int)at));
    }
  }
}

// A CTA has kWarps warps.  grid = (256 kSplit / kWarps, limbs), block = 32 kWarps.
template <typename W, int kWarps, int kSplit>
__global__ void __launch_bounds__(32 * kWarps, (sizeof(W) == 8 ? 16 : 20) / kWarps)
    raised_inner_kernel(const InnerProductArgs<W> g, const TensorOf<W> tensor, const typename WordTraits<W>::Pair* __restrict__ tw_all,
                        const PrimeConst<W>* __restrict__ pcs) {
  static_assert(kSplit == 1 || kSplit == kWarps, "warps that share a row are the CTA");
  __shared__ RaisedRow<W> rows[kWarps];
  grid_dependency_launch();
  const int b = (int)(gridDim.y - 1 - blockIdx.y);  // against the direction of the column pass
  const int warp = threadIdx.x >> 5;
  const int h = kSplit == 1 ? blockIdx.x * kWarps + warp : blockIdx.x, part = kSplit == 1 ? 0 : warp;
  RaisedRow<W>* mine = kSplit == 1 ? rows + warp : rows;
  const uint32_t pi = g.prime[b];
  const PrimeConst<W> pc = pcs[pi];
  const auto* tw = tw_all + (size_t)pi * kN;
  CERIUM_DISPATCH_ARITH(W, pc, raised_inner_body, kSplit, (g, tensor, b, h, part, pc, mine, tw));
}

}  // namespace cerium
