// Passes of the transforms with eight words to a thread: for batches that leave the schedulers few warps, and rows.
//
// A pass of 256 words is eight layers: three, three and two on registers, with two exchanges between them, in place of the
// four and four on sixteen words of ntt_kernels.cuh.  Its warp runs half the instructions in series and there are twice as
// many of them.  The pass of a row (one warp) and of a column (32 threads) are the same transform over the same tree of
// twiddles: pair (1 << t) + g is group g of layer t.
//
// Bound by latency: with sixteen words the inverse passes of ten 60-bit limbs had two warps a scheduler, each 2000 instructions
// in series at 5.6 cycles; the row pass waited for twiddles from memory in four of seven cycles.  Here a row's twiddles are on their
// way before the previous kernel is waited for, integers' as well.  Sixteen words -> eight (and, columns, the lines of
// launch_fwd_cols), rotations with five 60-bit extension limbs: 4 limbs 74.4 -> 63.8 us, 8 limbs 91.8 -> 77.2, 12 limbs 108.0 ->
// 98.9, 20 limbs 147.6 -> 141.6, 35 limbs 284.7 -> 275.1; multiplication of 8 limbs with one-limb digits 140.4 -> 109.
// Four rows to a CTA at 64 registers: two, eight, or 85 registers differ by less than the runs do.
#pragma once
#include "ntt_kernels.cuh"

namespace cerium {

// Four consecutive words, one access of 32 bytes (64-bit words) or 16.
template <typename W>
struct Quad {
  W v[4];
};
__device__ __forceinline__ Quad<uint32_t> quad_load(const uint32_t* p) {
  const uint4 t = *reinterpret_cast<const uint4*>(p);
  return {{t.x, t.y, t.z, t.w}};
}
// words that nothing reads again soon
__device__ __forceinline__ Quad<uint32_t> quad_load_once(const uint32_t* p) {
  const uint4 t = __ldcs(reinterpret_cast<const uint4*>(p));
  return {{t.x, t.y, t.z, t.w}};
}
__device__ __forceinline__ void quad_store(uint32_t* p, const Quad<uint32_t>& q) {
  *reinterpret_cast<uint4*>(p) = make_uint4(q.v[0], q.v[1], q.v[2], q.v[3]);
}
#if defined(CERIUM_EMU)
inline Quad<uint64_t> quad_load(const uint64_t* p) { return {{p[0], p[1], p[2], p[3]}}; }
inline Quad<uint64_t> quad_load_once(const uint64_t* p) { return quad_load(p); }
inline void quad_store(uint64_t* p, const Quad<uint64_t>& q) {
  for (int e = 0; e < 4; e++) p[e] = q.v[e];
}
#else
__device__ __forceinline__ Quad<uint64_t> quad_load(const uint64_t* p) {
  Quad<uint64_t> q;
  asm volatile("ld.global.v4.b64 {%0,%1,%2,%3}, [%4];" : "=l"(q.v[0]), "=l"(q.v[1]), "=l"(q.v[2]), "=l"(q.v[3]) : "l"(p) : "memory");
  return q;
}
__device__ __forceinline__ Quad<uint64_t> quad_load_once(const uint64_t* p) {
  Quad<uint64_t> q;
  asm volatile("ld.global.L1::no_allocate.L2::evict_first.v4.b64 {%0,%1,%2,%3}, [%4];" : "=l"(q.v[0]), "=l"(q.v[1]), "=l"(q.v[2]), "=l"(q.v[3]) : "l"(p) : "memory");
  return q;
}
__device__ __forceinline__ void quad_store(uint64_t* p, const Quad<uint64_t>& q) {
  asm volatile("st.global.v4.b64 [%0], {%1,%2,%3,%4};" ::"l"(p), "l"(q.v[0]), "l"(q.v[1]), "l"(q.v[2]), "l"(q.v[3]) : "memory");
}
#endif
// The same where a limb of 64-bit words may be aligned to 16 bytes only.
__device__ __forceinline__ bool quad_aligned(const void* p) { return ((uintptr_t)p & 31u) == 0; }
__device__ __forceinline__ Quad<uint32_t> quad_load(const uint32_t* p, bool) { return quad_load(p); }
__device__ __forceinline__ void quad_store(uint32_t* p, const Quad<uint32_t>& q, bool) { quad_store(p, q); }
__device__ __forceinline__ Quad<uint64_t> quad_load(const uint64_t* p, bool aligned) {
  if (aligned) return quad_load(p);
  const ulonglong2 a = reinterpret_cast<const ulonglong2*>(p)[0], b = reinterpret_cast<const ulonglong2*>(p)[1];
  return {{a.x, a.y, b.x, b.y}};
}
__device__ __forceinline__ void quad_store(uint64_t* p, const Quad<uint64_t>& q, bool aligned) {
  if (aligned) return quad_store(p, q);
  reinterpret_cast<ulonglong2*>(p)[0] = make_ulonglong2(q.v[0], q.v[1]);
  reinterpret_cast<ulonglong2*>(p)[1] = make_ulonglong2(q.v[2], q.v[3]);
}

// ---------------------------------------------------------------------------------------
// Bounds of the Fp butterflies, as fp_plan_fwd and fp_plan_inv have them for four layers.
// ---------------------------------------------------------------------------------------

// Eight forward layers; k6 and k7: how good the quotients of the last two are (k32 of fp_product_bound).
struct FpPassPlan {
  bool before[8];
  int out;
};
__host__ __device__ constexpr FpPassPlan fp_plan_pass(int bin, int k6, int k7) {
  FpPassPlan p{};
  int b = bin;
  for (int t = 0; t < 8; t++) {
    p.before[t] = b > kFpOperandMax;
    if (p.before[t]) b = kFpReduced;
    b += fp_product_bound(b, t < 6 ? 1 : t == 6 ? k6 : k7);
  }
  p.out = b;
  return p;
}
// A row whose table has the twiddles of the last two layers alone.  kFpCloseK32: twice the error of a tabulated quotient, more than that of
// Arith::close_quotient, which is enough for seven layers after a reduction (from 4 x 1024 on the last one would want another).
constexpr int kFpCloseK32 = 2;
__host__ __device__ constexpr FpPassPlan fp_plan_row(int bin, int k6) { return fp_plan_pass(bin, k6, kFpLaneK32); }
static_assert(fp_plan_row(kFpFwdMid, kFpCloseK32).out < 8192 && fp_plan_row(kFpRaisedMid, kFpLaneK32).out < 8192, "the transform's last values must stay exact integers");
static_assert(fp_plan_pass(kFpLoweredIn, 1, 1).out <= kFpFwdMid && fp_plan_pass(kFpRaisedIn, 1, 1).out <= kFpRaisedMid &&
                  fp_plan_pass(kFpCanon, 1, 1).out <= kFpRaisedMid, "what the row pass starts from");

// Inverse layers of `regs` (4 or 8) registers, each the distance after the one before: fp_plan_inv of that many.
struct FpInvGroup {
  unsigned before[3];
  unsigned exchange;  // registers reduced before they are exchanged
  int out;            // largest bound after that
};
__host__ __device__ constexpr FpInvGroup fp_plan_inv_group(int bin, int regs, int k32, int exchange_max) {
  FpInvGroup p{};
  int bound[8] = {};
  for (int j = 0; j < regs; j++) bound[j] = bin;
  for (int t = regs == 8 ? 2 : 1; t >= 0; t--) {
    const int half = (regs / 2) >> t;
    for (int g = 0; g < (1 << t); g++)
      for (int k = 0; k < half; k++) {
        const int j = g * 2 * half + k, i = j + half;
        if (bound[j] + bound[i] > kFpOperandMax) {
          const int big = bound[j] >= bound[i] ? j : i, other = big == j ? i : j;
          bound[big] = kFpReduced;
          p.before[t] |= 1u << big;
          if (bound[j] + bound[i] > kFpOperandMax) {
            bound[other] = kFpReduced;
            p.before[t] |= 1u << other;
          }
        }
        const int sum = bound[j] + bound[i];
        bound[j] = sum;
        bound[i] = fp_product_bound(sum, k32);
      }
  }
  for (int j = 0; j < regs; j++) {
    if (bound[j] > exchange_max) {
      p.exchange |= 1u << j;
      bound[j] = kFpReduced;
    }
    p.out = bound[j] > p.out ? bound[j] : p.out;
  }
  return p;
}
// layers 7 and 6, 5 to 3, 2 to 0 of the row pass, then of the column pass
constexpr FpInvGroup kFpInvRow0 = fp_plan_inv_group(kFpCanon, 4, kFpLaneK32, kFpInvExchangeMax);
constexpr FpInvGroup kFpInvRow1 = fp_plan_inv_group(kFpInvRow0.out, 8, 1, kFpInvExchangeMax);
constexpr FpInvGroup kFpInvRow2 = fp_plan_inv_group(kFpInvRow1.out, 8, 1, kFpInvMid);
static_assert(kFpInvRow2.out <= kFpInvMid, "what the column pass starts from");
constexpr FpInvGroup kFpInvCol0 = fp_plan_inv_group(kFpInvMid, 4, 1, kFpInvExchangeMax);
constexpr FpInvGroup kFpInvCol1 = fp_plan_inv_group(kFpInvCol0.out, 8, 1, kFpInvExchangeMax);

template <typename W, int kMode>
__device__ __forceinline__ void fp_reduce_masked(W (&x)[8], unsigned mask, const Arith<W, kMode>& ar) {
  if (kMode != kArithFp) return;
#pragma unroll
  for (int j = 0; j < 8; j++)
    if (mask >> j & 1u) x[j] = ar.reduce(x[j]);
}

// ---------------------------------------------------------------------------------------
// layers on eight registers
// ---------------------------------------------------------------------------------------

// Three layers on x[0..7]; layer t pairs (j, j + (4 >> t)) with twiddle (S << t) + (j >> (3 - t)).  kLayer: number of the
// first one inside the pass.
template <typename W, int kMode, int kLayer, int kBin>
__device__ __forceinline__ void radix8_fwd(W (&x)[8], const typename WordTraits<W>::Pair* tw, int S, const Arith<W, kMode>& ar) {
  constexpr FpPassPlan plan = fp_plan_pass(kBin, 1, 1);  // the first six layers: whatever the last two are
#pragma unroll
  for (int t = 0; t < 3; t++) {
    const int half = 4 >> t;
    if (plan.before[kLayer + t]) fp_reduce_masked<W, kMode>(x, 0xffu, ar);
#pragma unroll
    for (int g = 0; g < (1 << t); g++) {
      const auto w = tw[(S << t) + g];
#pragma unroll
      for (int k = 0; k < half; k++) ar.fwd(x[g * 2 * half + k], x[g * 2 * half + k + half], w.x, w.y);
    }
  }
}

// Layers kLayer + 2 down to kLayer of the inverse transform (kBin: bound of the inputs).
template <typename W, int kMode, int kLayer, int kBin>
__device__ __forceinline__ void radix8_inv(W (&x)[8], const typename WordTraits<W>::Pair* tw, int S, const Arith<W, kMode>& ar) {
  constexpr FpInvGroup plan = fp_plan_inv_group(kBin, 8, 1, 1 << 20);
#pragma unroll
  for (int t = 2; t >= 0; t--) {
    const int half = 4 >> t;
    fp_reduce_masked<W, kMode>(x, plan.before[t], ar);
#pragma unroll
    for (int g = 0; g < (1 << t); g++) {
      const auto w = tw[(S << t) + g];
#pragma unroll
      for (int k = 0; k < half; k++) ar.inv(x[g * 2 * half + k], x[g * 2 * half + k + half], w.x, w.y, 7 - kLayer - t);
    }
  }
}
// Layers 2 to 0 of the column pass; the last one scales by N^-1 and reduces to [0, q).
template <typename W, int kMode, int kBin>
__device__ __forceinline__ void radix8_inv_final(W (&x)[8], const typename WordTraits<W>::Pair* tw, const W (&last)[4], const Arith<W, kMode>& ar) {
  constexpr FpInvGroup plan = fp_plan_inv_group(kBin, 8, 1, 1 << 20);
#pragma unroll
  for (int t = 2; t >= 1; t--) {
    const int half = 4 >> t;
    fp_reduce_masked<W, kMode>(x, plan.before[t], ar);
#pragma unroll
    for (int g = 0; g < (1 << t); g++) {
      const auto w = tw[(1 << t) + g];
#pragma unroll
      for (int k = 0; k < half; k++) ar.inv(x[g * 2 * half + k], x[g * 2 * half + k + half], w.x, w.y, 7 - t);
    }
  }
  fp_reduce_masked<W, kMode>(x, plan.before[0], ar);
#pragma unroll
  for (int j = 0; j < 4; j++) ar.inv_last(x[j], x[j + 4], last);
}

// Twiddles of the last two layers of a thread's two groups of four words: one of layer 6 and two of layer 7 for each, with
// their companions.
template <typename W>
struct LateTwiddles {
  W w6[2][2], w7[2][4];
};
// Layers 6 and 7 on two groups of four words.
template <typename W, int kMode, int kBin, int kK6, int kK7>
__device__ __forceinline__ void late_fwd(W (&x)[8], const LateTwiddles<W>& l, const Arith<W, kMode>& ar) {
  constexpr FpPassPlan plan = fp_plan_pass(kBin, kK6, kK7);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    if (plan.before[6]) fp_reduce_masked<W, kMode>(x, 0xfu << 4 * k, ar);
    ar.fwd(x[4 * k], x[4 * k + 2], l.w6[k][0], l.w6[k][1]);
    ar.fwd(x[4 * k + 1], x[4 * k + 3], l.w6[k][0], l.w6[k][1]);
    if (plan.before[7]) fp_reduce_masked<W, kMode>(x, 0xfu << 4 * k, ar);
    ar.fwd(x[4 * k], x[4 * k + 1], l.w7[k][0], l.w7[k][1]);
    ar.fwd(x[4 * k + 2], x[4 * k + 3], l.w7[k][2], l.w7[k][3]);
  }
}
template <typename W, int kMode, int kBin, int kK32>
__device__ __forceinline__ void late_inv(W (&x)[8], const LateTwiddles<W>& l, const Arith<W, kMode>& ar) {
  constexpr FpInvGroup plan = fp_plan_inv_group(kBin, 4, kK32, 1 << 20);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    fp_reduce_masked<W, kMode>(x, plan.before[1] << 4 * k, ar);
    ar.inv(x[4 * k], x[4 * k + 1], l.w7[k][0], l.w7[k][1], 0);
    ar.inv(x[4 * k + 2], x[4 * k + 3], l.w7[k][2], l.w7[k][3], 0);
    fp_reduce_masked<W, kMode>(x, plan.before[0] << 4 * k, ar);
    ar.inv(x[4 * k], x[4 * k + 2], l.w6[k][0], l.w6[k][1], 1);
    ar.inv(x[4 * k + 1], x[4 * k + 3], l.w6[k][0], l.w6[k][1], 1);
  }
}

// Exchange buffer of a row: word i at i + 4 (i / 32), 64-bit words with bit 1 of i flipped where bit 4 is set.  The three
// patterns (a run of 32; 8 runs of 4 at a distance of 32; 4 words of each of 32 neighbouring lanes, 16 bytes at a time) are
// then free of bank conflicts.
constexpr int kRaisedPitch = 256 + 8 * 4;
template <typename W>
__device__ __forceinline__ int raised_pos(int i) {
  return (sizeof(W) == 8 ? i ^ ((i >> 3) & 2) : i) + (i >> 5) * 4;
}
template <typename W>
__device__ __forceinline__ void row_put_quads(W* ex, const W (&x)[8]) {
  using RV = RowVec<W>;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < 8; k += RV::kWords)
    *reinterpret_cast<typename RV::Vec*>(ex + raised_pos<W>((k >> 2) * 128 + lane * 4 + (k & 3))) = vec_pack(&x[k]);
}
template <typename W>
__device__ __forceinline__ void row_get_quads(const W* ex, W (&x)[8]) {
  using RV = RowVec<W>;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < 8; k += RV::kWords)
    vec_unpack(*reinterpret_cast<const typename RV::Vec*>(ex + raised_pos<W>((k >> 2) * 128 + lane * 4 + (k & 3))), &x[k]);
}

// A row's shared memory: the exchange buffer, and the twiddles of layers 0 to 5, which several lanes use.  Those of the last
// two layers have one lane each and go from global memory to its registers.
template <typename W>
struct alignas(16) Radix8Row {
  W ex[kRaisedPitch];
  typename WordTraits<W>::Pair tw[64];
};
// Copies pairs 1 to 63 of row h; row_twiddles_wait() before they are used.
template <typename W>
__device__ __forceinline__ void radix8_row_twiddles(Radix8Row<W>& row, const typename WordTraits<W>::Pair* tw, int h) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int i = k * 32 + lane;
    if (i == 0) continue;
    const int t = 31 - __clz(i);
    copy_async<sizeof(typename WordTraits<W>::Pair)>(&row.tw[i], tw + (((256u + (uint32_t)h) << t) + (uint32_t)(i - (1 << t))));
  }
}
// Those of this lane's groups k * 32 + lane of layer 6; Fp: from the lane table (lane_tw_fp), which has no companions.
template <typename W, int kMode>
__device__ __forceinline__ void late_row_load(LateTwiddles<W>& l, const typename WordTraits<W>::Pair* tw,
                                              const typename WordTraits<W>::Pair* twr, int h) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    if constexpr (kMode == kArithFp) {
      const auto* of = twr + (size_t)(h * 8 * 16 + k * 8 + (lane >> 2));
      l.w6[k][0] = __ldg(reinterpret_cast<const W*>(of + (2 + (lane >> 1 & 1)) * 16) + (lane & 1));
      const auto w = __ldg(of + (4 + (lane & 3)) * 16);
      l.w7[k][0] = w.x, l.w7[k][2] = w.y;
    } else {
      const uint32_t g = (uint32_t)(k * 32 + lane), S = 256u + (uint32_t)h;
      const auto a = __ldg(tw + S * 64u + g);
      const Quad<W> b = quad_load(reinterpret_cast<const W*>(tw + S * 128u + 2u * g));
      l.w6[k][0] = a.x, l.w6[k][1] = a.y;
#pragma unroll
      for (int e = 0; e < 4; e++) l.w7[k][e] = b.v[e];
    }
  }
}
template <typename W, int kMode>
__device__ __forceinline__ void late_row_quotients(LateTwiddles<W>& l, const Arith<W, kMode>& ar) {
  if constexpr (kMode == kArithFp) {
#pragma unroll
    for (int k = 0; k < 2; k++) {
      l.w6[k][1] = ar.close_quotient(l.w6[k][0]);
      l.w7[k][1] = ar.quotient(l.w7[k][0]), l.w7[k][3] = ar.quotient(l.w7[k][2]);
    }
  }
}

// ---------------------------------------------------------------------------------------
// row passes: a warp has one row
// ---------------------------------------------------------------------------------------
constexpr int kRadix8Rows = 4;                      // of a CTA
constexpr int kRadix8RowsPerSm = 32 / kRadix8Rows;  // CTAs that an SM holds: 32 warps of 64 registers a thread
// Forward rows of 32-bit words, which read operands, let the next kernel in late in grids of two rounds as well (division of 22 limbs
// 10.96 -> 10.05 us, of 34 limbs 14.8 -> 13.9, of 20 limbs through pointer tables 11.8 -> 10.0); 64-bit words lose (34 limbs 23.5 -> 24.1).
template <typename W>
constexpr int kRadix8FwdRowsLate = sizeof(W) == 4 ? 2 * kRadix8RowsPerSm : kRadix8RowsPerSm;

template <typename W, int kMode, typename Batch, typename Epilogue>
__device__ __forceinline__ void radix8_fwd_rows_body(const Batch& batch, const Epilogue& epi, int b, uint32_t pi, const PrimeConst<W>& pc,
                                                     Radix8Row<W>& row, const typename WordTraits<W>::Pair* tw,
                                                     const typename WordTraits<W>::Pair* twr, int h) {
  using RV = RowVec<W>;
  constexpr int kVecs = 4 / RV::kWords;  // 16-byte vectors of a group of four words
  const Arith<W, kMode> ar(pc);
  const int lane = threadIdx.x & 31, own = (lane >> 2) * 32 + (lane & 3);
  radix8_row_twiddles<W>(row, tw, h);
  LateTwiddles<W> late;
  late_row_load<W, kMode>(late, tw, twr, h);
  grid_dependency_wait();
  const W* in = batch.in_limb(b) + (unsigned)(h * 256 + lane);
  W* limb_out = batch.out_limb(b);
  W x[8];
#pragma unroll
  for (int j = 0; j < 8; j++) x[j] = in[j * 32];
#pragma unroll
  for (int k = 0; k < 2; k++)
#pragma unroll
    for (int v = 0; v < kVecs; v++) epi.prefetch(b, h * 256 + k * 128 + lane * 4 + v * RV::kWords);
  row_twiddles_wait();
  radix8_fwd<W, kMode, 0, kFpFwdMid>(x, row.tw, 1, ar);
#pragma unroll
  for (int j = 0; j < 8; j++) row.ex[raised_pos<W>(j * 32 + lane)] = x[j];
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 8; j++) x[j] = row.ex[raised_pos<W>(own + 4 * j)];
  radix8_fwd<W, kMode, 3, kFpFwdMid>(x, row.tw, 8 + (lane >> 2), ar);
#pragma unroll
  for (int j = 0; j < 8; j++) row.ex[raised_pos<W>(own + 4 * j)] = x[j];
  __syncwarp();
  typename Epilogue::Operands ops[2][kVecs];
#pragma unroll
  for (int k = 0; k < 2; k++)
#pragma unroll
    for (int v = 0; v < kVecs; v++) ops[k][v] = epi.load(b, h * 256 + k * 128 + lane * 4 + v * RV::kWords);
  if (grid_resident(kRadix8FwdRowsLate<W>)) grid_dependency_launch();
  row_get_quads<W>(row.ex, x);
  late_row_quotients<W, kMode>(late, ar);
  late_fwd<W, kMode, kFpFwdMid, kFpCloseK32, kFpLaneK32>(x, late, ar);
  const uint32_t selt = epi.scatter_elt();
  const bool wide = quad_aligned(limb_out);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int at = h * 256 + k * 128 + lane * 4;
    Quad<W> o;
#pragma unroll
    for (int v = 0; v < kVecs; v++) {
      W w[RV::kWords];
#pragma unroll
      for (int e = 0; e < RV::kWords; e++) w[e] = x[4 * k + v * RV::kWords + e];
      epi.apply_vec(w, ops[k][v], b, at + v * RV::kWords, pi, pc, ar);
#pragma unroll
      for (int e = 0; e < RV::kWords; e++) o.v[v * RV::kWords + e] = w[e];
    }
    if (selt != 0) {
      // an aligned group of words lands on an aligned group of the output limb
      const GaloisGroup<4> gg((uint32_t)at, selt);
      Quad<W> t;
      gg.template permute<true>(o.v, t.v);
      quad_store(limb_out + gg.at, t, wide);
    } else {
      quad_store(limb_out + at, o, wide);
    }
  }
}

// grid = (256 / kRadix8Rows, limbs), block = 32 kRadix8Rows.
template <typename W, typename Batch, typename Epilogue>
__global__ void __launch_bounds__(32 * kRadix8Rows, kRadix8RowsPerSm)
    radix8_fwd_rows_kernel(const Batch batch, const Epilogue epi, const typename WordTraits<W>::Pair* __restrict__ tw_all,
                           const typename WordTraits<W>::Pair* __restrict__ twr_all, const PrimeConst<W>* __restrict__ pcs) {
  static_assert(sizeof(Batch) + sizeof(Epilogue) + 3 * sizeof(void*) <= kMaxParameters);
  __shared__ Radix8Row<W> rows[kRadix8Rows];
  if (!grid_resident(kRadix8FwdRowsLate<W>)) grid_dependency_launch();
  const int b = (int)(gridDim.y - 1 - blockIdx.y);  // against the direction of the column pass
  const int warp = threadIdx.x >> 5, h = blockIdx.x * kRadix8Rows + warp;
  const uint32_t pi = batch.prime_of(b);
  const PrimeConst<W> pc = pcs[pi];
  CERIUM_DISPATCH_ARITH(W, pc, radix8_fwd_rows_body, CERIUM_TARGS(Batch, Epilogue),
                        (batch, epi, b, pi, pc, rows[warp], tw_all + (size_t)pi * kN, twr_all + (size_t)pi * kRowTwPerPrime, h));
}

template <typename W, int kMode, typename Batch>
__device__ __forceinline__ void radix8_inv_rows_body(const Batch& batch, int b, const PrimeConst<W>& pc, Radix8Row<W>& row,
                                                     const typename WordTraits<W>::Pair* twi, const typename WordTraits<W>::Pair* twri, int h) {
  const Arith<W, kMode> ar(pc);
  const int lane = threadIdx.x & 31, own = (lane >> 2) * 32 + (lane & 3);
  radix8_row_twiddles<W>(row, twi, h);
  LateTwiddles<W> late;
  late_row_load<W, kMode>(late, twi, twri, h);
  grid_dependency_wait();
  const W* in = batch.in_limb(b);
  const uint32_t elt = batch.gather_elt();
  const bool wide = quad_aligned(in);
  W x[8];
  Quad<W> t[2];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const uint32_t at = (uint32_t)(h * 256 + k * 128 + lane * 4);
    // the automorphism maps aligned groups of words onto aligned groups
    t[k] = quad_load(in + (elt != 0 ? GaloisGroup<4>(at, elt).at : at), wide);
  }
  if constexpr (Batch::kProduct) {
    const W* factor = batch.factor_limb(b);
    const bool fwide = quad_aligned(factor);
    Quad<W> f[2];
#pragma unroll
    for (int k = 0; k < 2; k++) f[k] = quad_load(factor + (h * 256 + k * 128 + lane * 4), fwide);
#pragma unroll
    for (int k = 0; k < 2; k++)
#pragma unroll
      for (int e = 0; e < 4; e++) t[k].v[e] = mul_mod<W>(t[k].v[e], f[k].v[e], pc);
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    if (elt != 0) {
      Quad<W> p;
      GaloisGroup<4>((uint32_t)(h * 256 + k * 128 + lane * 4), elt).permute(t[k].v, p.v);
      t[k] = p;
    }
#pragma unroll
    for (int e = 0; e < 4; e++) x[4 * k + e] = ar.enter(t[k].v[e]);
  }
  late_row_quotients<W, kMode>(late, ar);
  late_inv<W, kMode, kFpCanon, kFpLaneK32>(x, late, ar);
  fp_reduce_masked<W, kMode>(x, kFpInvRow0.exchange * 0x11u, ar);
  row_put_quads<W>(row.ex, x);
  row_twiddles_wait();  // and every lane's words are there
#pragma unroll
  for (int j = 0; j < 8; j++) x[j] = row.ex[raised_pos<W>(own + 4 * j)];
  radix8_inv<W, kMode, 3, kFpInvRow0.out>(x, row.tw, 8 + (lane >> 2), ar);
  fp_reduce_masked<W, kMode>(x, kFpInvRow1.exchange, ar);
#pragma unroll
  for (int j = 0; j < 8; j++) row.ex[raised_pos<W>(own + 4 * j)] = x[j];
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 8; j++) x[j] = row.ex[raised_pos<W>(j * 32 + lane)];
  if (grid_resident(kRadix8RowsPerSm)) grid_dependency_launch();
  radix8_inv<W, kMode, 0, kFpInvRow1.out>(x, row.tw, 1, ar);
  fp_reduce_masked<W, kMode>(x, kFpInvRow2.exchange, ar);
  W* out = batch.out_limb(b) + (unsigned)(h * 256 + lane);
#pragma unroll
  for (int j = 0; j < 8; j++) out[j * 32] = x[j];
}

template <typename W, typename Batch>
__global__ void __launch_bounds__(32 * kRadix8Rows, kRadix8RowsPerSm)
    radix8_inv_rows_kernel(const Batch batch, const typename WordTraits<W>::Pair* __restrict__ twi_all,
                           const typename WordTraits<W>::Pair* __restrict__ twri_all, const PrimeConst<W>* __restrict__ pcs) {
  __shared__ Radix8Row<W> rows[kRadix8Rows];
  if (!grid_resident(kRadix8RowsPerSm)) grid_dependency_launch();
  const int b = blockIdx.y;
  const int warp = threadIdx.x >> 5, h = blockIdx.x * kRadix8Rows + warp;
  const uint32_t pi = batch.prime_of(b);
  const PrimeConst<W> pc = pcs[pi];
  CERIUM_DISPATCH_ARITH(W, pc, radix8_inv_rows_body, CERIUM_TARGS(Batch),
                        (batch, b, pc, rows[warp], twi_all + (size_t)pi * kN, twri_all + (size_t)pi * kRowTwPerPrime, h));
}

// ---------------------------------------------------------------------------------------
// column passes: 32 threads have a column, a CTA kCols adjacent ones
// ---------------------------------------------------------------------------------------

// CTAs that an SM holds: 256 threads of 64 registers, 512 of 40 (32-bit words forward) or 64
template <typename W>
constexpr int kRadix8FwdColsPerSm = sizeof(W) == 8 ? 4 : 3;
template <typename W>
constexpr int kRadix8InvColsPerSm = sizeof(W) == 8 ? 4 : 2;
// Inverse columns let the next kernel in late in grids of up to two rounds, which the lines of launch_inv_cols keep them to.  Without
// the branch the compiler orders the last layers otherwise: 10 limbs of 64-bit words 8.57 -> 8.82 us.
template <typename W>
constexpr int kRadix8InvColsLate = 2 * kRadix8InvColsPerSm<W>;

// Rows of the tile whose words share a bank lie eight apart in one of the three patterns (rows v * 8 + j of neighbouring
// threads v).  Two rows make a line of 128 bytes, of 8 words of 64 bits or 16 of 32: bit 3 of the row's number goes into the lowest one.
template <typename W, int kCols>
__device__ __forceinline__ int radix8_tile(int r, int c) {
  static_assert(2 * kCols * sizeof(W) == 128, "two rows to a line");
  return (r ^ (r >> 3 & 1)) * kCols + c;
}
// Barrier of the four threads that exchange a column's rows of one block of 32.
template <int kCols>
__device__ __forceinline__ void radix8_quad_sync() {
  if (4 * kCols <= 32) __syncwarp();
  else __syncthreads();
}
template <typename W>
__device__ __forceinline__ void late_column_load(LateTwiddles<W>& l, const typename WordTraits<W>::Pair* stw, int v) {
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const auto a = stw[64 + 2 * v + k], b = stw[128 + 4 * v + 2 * k], c = stw[128 + 4 * v + 2 * k + 1];
    l.w6[k][0] = a.x, l.w6[k][1] = a.y;
    l.w7[k][0] = b.x, l.w7[k][1] = b.y, l.w7[k][2] = c.x, l.w7[k][3] = c.y;
  }
}

template <typename W, int kMode, int kCols, typename Batch, typename Loader>
__device__ __forceinline__ void radix8_fwd_cols_body(const Batch& batch, const Loader& loader, int b, const PrimeConst<W>& pc, W* tile,
                                                     const typename WordTraits<W>::Pair* stw) {
  const Arith<W, kMode> ar(pc);
  const int c = threadIdx.x % kCols, v = threadIdx.x / kCols;
  const int col = blockIdx.x * kCols + c, own = (v >> 2) * 32 + (v & 3);
  const W* in = batch.in_limb(b) + (unsigned)(v * 256 + col);
  W* out = batch.out_limb(b) + (unsigned)(v * 8 * 256 + col);
  W x[8];
#pragma unroll
  for (int j = 0; j < 8; j++) x[j] = in[j * 32 * 256];
  bool entered = false;
  if constexpr (Loader::kHasSmall && kMode == kArithFp) {
    if (loader.small[b] != 0) {
#pragma unroll
      for (int j = 0; j < 8; j++) x[j] = ar.reduce(ar.enter(x[j]));
      entered = true;
    }
  }
  if (!entered) {
#pragma unroll
    for (int j = 0; j < 8; j++) x[j] = ar.enter(loader.apply(x[j], b, pc));
  }
  __syncthreads();  // the twiddles are there
  radix8_fwd<W, kMode, 0, Loader::kFpBound>(x, stw, 1, ar);
#pragma unroll
  for (int j = 0; j < 8; j++) tile[radix8_tile<W, kCols>(j * 32 + v, c)] = x[j];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 8; j++) x[j] = tile[radix8_tile<W, kCols>(own + 4 * j, c)];
  radix8_fwd<W, kMode, 3, Loader::kFpBound>(x, stw, 8 + (v >> 2), ar);
#pragma unroll
  for (int j = 0; j < 8; j++) tile[radix8_tile<W, kCols>(own + 4 * j, c)] = x[j];
  radix8_quad_sync<kCols>();
#pragma unroll
  for (int j = 0; j < 8; j++) x[j] = tile[radix8_tile<W, kCols>(v * 8 + j, c)];
  if (grid_resident(kRadix8FwdColsPerSm<W>)) grid_dependency_launch();
  LateTwiddles<W> late;
  late_column_load<W>(late, stw, v);
  late_fwd<W, kMode, Loader::kFpBound, 1, 1>(x, late, ar);
#pragma unroll
  for (int j = 0; j < 8; j++) out[j * 256] = x[j];
}

// grid = (256 / kCols, limbs), block = 32 kCols.
template <typename W, int kCols, typename Batch, typename Loader>
__global__ void __launch_bounds__(kCols * 32, kRadix8FwdColsPerSm<W>)
    radix8_fwd_cols_kernel(const Batch batch, const Loader loader, const typename WordTraits<W>::Pair* __restrict__ tw_all,
                           const PrimeConst<W>* __restrict__ pcs) {
  static_assert(sizeof(Batch) + sizeof(Loader) + 2 * sizeof(void*) <= kMaxParameters);
  __shared__ W tile[256 * kCols];
  __shared__ typename WordTraits<W>::Pair stw[256];
  if (!grid_resident(kRadix8FwdColsPerSm<W>)) grid_dependency_launch();
  const int b = blockIdx.y;
  const uint32_t pi = batch.prime_of(b);
  const PrimeConst<W> pc = pcs[pi];
  for (int k = threadIdx.x; k < 256; k += kCols * 32) stw[k] = __ldg(tw_all + (size_t)pi * kN + k);
  grid_dependency_wait();
  CERIUM_DISPATCH_ARITH(W, pc, radix8_fwd_cols_body, CERIUM_TARGS(kCols, Batch, Loader), (batch, loader, b, pc, tile, stw));
}

template <typename W, int kMode, int kCols, typename Batch>
__device__ __forceinline__ void radix8_inv_cols_body(const Batch& batch, const InvScale<W>& sc, int b, const PrimeConst<W>& pc, W* tile,
                                                     const typename WordTraits<W>::Pair* stw) {
  const Arith<W, kMode> ar(pc);
  const int c = threadIdx.x % kCols, v = threadIdx.x / kCols;
  const int col = blockIdx.x * kCols + c, own = (v >> 2) * 32 + (v & 3);
  const W* in = batch.out_limb(b) + (unsigned)(v * 8 * 256 + col);
  W* out = batch.out_limb(b) + (unsigned)(v * 256 + col);
  W x[8];
#pragma unroll
  for (int j = 0; j < 8; j++) {
    x[j] = in[j * 256];
    if (kMode == kArithLazy) x[j] = reduce_lazy(x[j], pc.one_shoup, (W)0 - pc.q);  // back below 4q for the second pass
  }
  W last[4];
  if (sc.last != nullptr) {
#pragma unroll
    for (int e = 0; e < 4; e++) last[e] = __ldg(sc.last + 4 * b + e);
  } else if (kMode == kArithFp) {
    last[0] = pc.fp_ninv, last[1] = pc.fp_ninv_q, last[2] = pc.fp_w1ninv, last[3] = pc.fp_w1ninv_q;
  } else {
    last[0] = pc.ninv, last[1] = pc.ninv_shoup, last[2] = pc.w1ninv, last[3] = pc.w1ninv_shoup;
  }
  __syncthreads();  // the twiddles are there
  LateTwiddles<W> late;
  late_column_load<W>(late, stw, v);
  late_inv<W, kMode, kFpInvMid, 1>(x, late, ar);
  fp_reduce_masked<W, kMode>(x, kFpInvCol0.exchange * 0x11u, ar);
#pragma unroll
  for (int j = 0; j < 8; j++) tile[radix8_tile<W, kCols>(v * 8 + j, c)] = x[j];
  radix8_quad_sync<kCols>();
#pragma unroll
  for (int j = 0; j < 8; j++) x[j] = tile[radix8_tile<W, kCols>(own + 4 * j, c)];
  radix8_inv<W, kMode, 3, kFpInvCol0.out>(x, stw, 8 + (v >> 2), ar);
  fp_reduce_masked<W, kMode>(x, kFpInvCol1.exchange, ar);
#pragma unroll
  for (int j = 0; j < 8; j++) tile[radix8_tile<W, kCols>(own + 4 * j, c)] = x[j];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 8; j++) x[j] = tile[radix8_tile<W, kCols>(j * 32 + v, c)];
  if (grid_resident(kRadix8InvColsLate<W>)) grid_dependency_launch();
  radix8_inv_final<W, kMode, kFpInvCol1.out>(x, stw, last, ar);
  if (sc.add != nullptr) {
    const W a = __ldg(sc.add + b);
#pragma unroll
    for (int j = 0; j < 8; j++) x[j] = add_mod<W>(x[j], a, pc.q);
  }
#pragma unroll
  for (int j = 0; j < 8; j++) out[j * 32 * 256] = x[j];
}

template <typename W, int kCols, typename Batch>
__global__ void __launch_bounds__(kCols * 32, kRadix8InvColsPerSm<W>)
    radix8_inv_cols_kernel(const Batch batch, const InvScale<W> sc, const typename WordTraits<W>::Pair* __restrict__ twi_all,
                           const PrimeConst<W>* __restrict__ pcs) {
  __shared__ W tile[256 * kCols];
  __shared__ typename WordTraits<W>::Pair stw[256];
  if (!grid_resident(kRadix8InvColsLate<W>)) grid_dependency_launch();
  const int b = (int)(gridDim.y - 1 - blockIdx.y);  // against the direction of the row pass
  const uint32_t pi = batch.prime_of(b);
  const PrimeConst<W> pc = pcs[pi];
  for (int k = threadIdx.x; k < 256; k += kCols * 32) stw[k] = __ldg(twi_all + (size_t)pi * kN + k);
  grid_dependency_wait();
  CERIUM_DISPATCH_ARITH(W, pc, radix8_inv_cols_body, CERIUM_TARGS(kCols, Batch), (batch, sc, b, pc, tile, stw));
}

}  // namespace cerium
