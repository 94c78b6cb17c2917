// Context, NTT, SuD, element-wise, automorphism and base-conversion entry points of the C ABI.
// Host code here only validates arguments, fills by-value parameter blocks and launches; the
// arithmetic lives in the *_kernels.cuh headers.  Mirrors the role of
// cerium/runtime/execution/evaluator.cpp (Evaluator::fn_*) and device_utils.cu (execute_*).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "internal.h"

namespace cerium {

static thread_local std::string g_last_error;

void set_error(const std::string& msg) { g_last_error = msg; }
int fail(int code, const std::string& msg) {
  g_last_error = msg;
  return code;
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

template <typename W>
static int fill_batch(cerium_context* ctx, StridedBatch<W>& sb, const uint32_t* pos, const uint32_t* prime,
                      int first, int count) {
  for (int b = 0; b < count; b++) {
    const uint32_t p = prime[first + b];
    if (p >= (uint32_t)ctx->n_primes) return fail(CERIUM_ERR_INVALID, "prime index out of range");
    const uint32_t s = pos ? pos[first + b] : (uint32_t)(first + b);
    if (s > 0xffffu) return fail(CERIUM_ERR_INVALID, "limb slot exceeds 65535");
    sb.prime[b] = (uint8_t)p;
    sb.pos[b] = (uint16_t)s;
  }
  return CERIUM_OK;
}

static int check_stack(const void* p, size_t stride_words, size_t word_bytes, const char* what,
                       bool allow_zero_stride = false) {
  if (p == nullptr) return fail(CERIUM_ERR_INVALID, std::string(what) + " is null");
  if (!aligned16(p)) return fail(CERIUM_ERR_INVALID, std::string(what) + " is not 16-byte aligned");
  if ((stride_words * word_bytes) % 16) return fail(CERIUM_ERR_INVALID, std::string(what) + " stride is not a multiple of 16 bytes");
  if (!allow_zero_stride && stride_words < (size_t)kN) return fail(CERIUM_ERR_INVALID, std::string(what) + " stride is smaller than N");
  return CERIUM_OK;
}

// ---------------------------------------------------------------------------------------
// NTT launchers
// ---------------------------------------------------------------------------------------

// The passes of `limbs` limbs, in small tiles where those of the usual size would leave SMs without a full set of CTAs.
template <typename W>
static bool small_batch(const cerium_context* ctx, int limbs) { return limbs * (256 / kRowsPerCta) <= kSmallBatchPerSm<W> * ctx->sm_count; }
// Limbs up to which a pass takes eight words to a thread (ntt_radix8.cuh) and not sixteen, on 148 SMs; us with eight / sixteen.
//   Columns: beyond the lines the second barrier and the narrow tiles cost more than the shorter chain gives.
//     64-bit words inverse: 23 limbs alone 14.5 / 15.0, 24 limbs 15.9 / 15.5, 40 limbs 22.8 / 22.1, rotation of 24 limbs 167.9 / 167.4,
//     of 35 limbs 271.6 / 270.7.  Integer butterflies alike: 23 limbs 21.9 / 23.0, 24 limbs 23.9 / 23.3.
//     32-bit words inverse: 27 limbs 10.8 / 10.9, 28 limbs 11.9 / 11.3, rotation of 28 limbs with 14 extension limbs 88.2 / 86.0.
//     Forward: 32 limbs 18.2 / 18.8; 32-bit words only where they come from a conversion or a division (rotation of 6
//     limbs 42.4 / 44.4; alone, 3 limbs 6.9 / 4.7, 20 limbs 9.9 / 9.3).
//   Forward rows: 64-bit words eight for every batch (257 limbs alone 115.5 / 117.8, in pointer tables 119.5 / 124.9, of integers
//     176.3 / 183.9; 384 limbs under the power limit 185.3 / 185.7).  32-bit words only where the epilogue reads operands
//     (rotation of 51 limbs 173.9 / 176.9; plain, 245 limbs 69.2 / 66.4).
//   Inverse rows: eight, and sixteen without twiddles in shared memory from 129 limbs on where the GPU is at its power limit
//     (128 limbs 59.2 / 62.6; 140 limbs 73.8 / 72.9, 384 limbs 197.8 / 193.3) and from 91 of 32-bit words (85 limbs 26.6 / 26.6, 100 limbs
//     31.0 / 30.6, 256 limbs 72.6 / 70.8).  Stacks of limbs with their twiddles in shared memory, in small tiles, do better between:
//     32-bit words from 56 limbs on (46 limbs 15.3 / 15.4, 60 limbs 19.6 / 19.2, 74 limbs 23.1 / 22.0, rotation of 60 limbs 207.3 / 208.4),
//     64-bit words on doubles from 36 (32 limbs 18.2 / 18.3, 40 limbs 22.2 / 21.8, 64 limbs 32.9 / 31.8, rotation of 35 limbs 275.4 /
//     276.4, of 45 limbs 406.7 / 407.4).  Not of pointer tables (74 limbs of 32-bit words 22.4 / 23.1) and not of products
//     (multiplication of 25 limbs 226.9 / 231.8).  Stacks of integers take eight whatever their number (28 limbs 27.1 / 31.2, 64 limbs
//     51.0 / 59.5, 140 limbs under the power limit 109.7 / 117.1).
template <typename W>
constexpr int kRadix8InvCols = sizeof(W) == 8 ? 23 : 27;
constexpr int kRadix8FwdCols = 32;
template <typename W>
constexpr int kRadix8InvRows = sizeof(W) == 8 ? 128 : 90;
template <typename W>
constexpr int kRadix8InvRowsOfStacks = sizeof(W) == 8 ? 35 : 55;

template <typename W, typename Batch, typename Loader>
static void launch_fwd_cols(cerium_context* ctx, const Batch& batch, const Loader& loader, int limbs, cudaStream_t stream) {
  constexpr int kCols = NttCfg<W>::kCols;
  const auto* tw = static_cast<const typename WordTraits<W>::Pair*>(ctx->d_tw_fwd);
  const auto* pcs = static_cast<const PrimeConst<W>*>(ctx->d_pcs);
  if constexpr (sizeof(W) == 8 || !Loader::kPlain) {
    if (limbs <= kRadix8FwdCols) {
      auto kfn = radix8_fwd_cols_kernel<W, kCols / 2, Batch, Loader>;
      CERIUM_LAUNCH(kfn, dim3(512 / kCols, limbs), kCols * 16, 0, stream, batch, loader, tw, pcs);
      return;
    }
  }
  if (small_batch<W>(ctx, limbs)) {
    auto kfn = ntt_fwd_cols_kernel<W, kCols / 2, Batch, Loader>;
    CERIUM_LAUNCH(kfn, dim3(512 / kCols, limbs), kCols * 8, 0, stream, batch, loader, tw, pcs);
  } else {
    auto kfn = ntt_fwd_cols_kernel<W, kCols, Batch, Loader>;
    CERIUM_LAUNCH(kfn, dim3(256 / kCols, limbs), kCols * 16, 0, stream, batch, loader, tw, pcs);
  }
}
template <typename W, typename Batch>
static void launch_inv_cols(cerium_context* ctx, const Batch& batch, const InvScale<W>& scale, int limbs, cudaStream_t stream) {
  constexpr int kCols = NttCfg<W>::kCols;
  const auto* tw = static_cast<const typename WordTraits<W>::Pair*>(ctx->d_tw_inv);
  const auto* pcs = static_cast<const PrimeConst<W>*>(ctx->d_pcs);
  if (limbs <= kRadix8InvCols<W>) {
    auto kfn = radix8_inv_cols_kernel<W, kCols / 2, Batch>;
    CERIUM_LAUNCH(kfn, dim3(512 / kCols, limbs), kCols * 16, 0, stream, batch, scale, tw, pcs);
  } else if (small_batch<W>(ctx, limbs)) {
    auto kfn = ntt_inv_cols_kernel<W, kCols / 2, Batch>;
    CERIUM_LAUNCH(kfn, dim3(512 / kCols, limbs), kCols * 8, 0, stream, batch, scale, tw, pcs);
  } else {
    auto kfn = ntt_inv_cols_kernel<W, kCols, Batch>;
    CERIUM_LAUNCH(kfn, dim3(256 / kCols, limbs), kCols * 16, 0, stream, batch, scale, tw, pcs);
  }
}
template <typename W, typename Batch, typename Epilogue>
static void launch_fwd_rows(cerium_context* ctx, const Batch& batch, const Epilogue& epi, int limbs, cudaStream_t stream) {
  using Pair = typename WordTraits<W>::Pair;
  const auto* tw = static_cast<const Pair*>(ctx->d_tw_fwd);
  const auto* twr = static_cast<const Pair*>(ctx->d_twr_fwd);
  const auto* pcs = static_cast<const PrimeConst<W>*>(ctx->d_pcs);
  if constexpr (sizeof(W) == 8 || Epilogue::kHasOperands) {
    auto kfn = radix8_fwd_rows_kernel<W, Batch, Epilogue>;
    CERIUM_LAUNCH(kfn, dim3(256 / kRadix8Rows, limbs), kRadix8Rows * 32, 0, stream, batch, epi, tw, twr, pcs);
  } else if (small_batch<W>(ctx, limbs)) {
    auto kfn = ntt_fwd_rows_kernel<W, kRowsSmall, true, Batch, Epilogue>;
    CERIUM_LAUNCH(kfn, dim3(256 / kRowsSmall, limbs), kRowsSmall * 16, 0, stream, batch, tw, twr, pcs);
  } else {
    auto kfn = ntt_fwd_rows_kernel<W, kRowsPerCta, false, Batch, Epilogue>;
    CERIUM_LAUNCH(kfn, dim3(256 / kRowsPerCta, limbs), kRowsPerCta * 16, 0, stream, batch, tw, twr, pcs);
  }
}
// doubles: most of the primes have butterflies on doubles (stacks of 64-bit words)
template <typename W, typename Batch>
static void launch_inv_rows(cerium_context* ctx, const Batch& batch, int limbs, cudaStream_t stream, bool doubles = false) {
  using Pair = typename WordTraits<W>::Pair;
  const auto* tw = static_cast<const Pair*>(ctx->d_tw_inv);
  const auto* twr = static_cast<const Pair*>(ctx->d_twr_inv);
  const auto* pcs = static_cast<const PrimeConst<W>*>(ctx->d_pcs);
  constexpr bool kStack = std::is_same_v<Batch, StridedBatch<W>>;
  if constexpr (kStack) {
    if (limbs > kRadix8InvRowsOfStacks<W> && small_batch<W>(ctx, limbs) && (sizeof(W) == 4 || doubles)) {
      auto kfn = ntt_inv_rows_kernel<W, kRowsSmall, true, Batch>;
      CERIUM_LAUNCH(kfn, dim3(256 / kRowsSmall, limbs), kRowsSmall * 16, 0, stream, batch, tw, twr, pcs);
      return;
    }
  }
  if constexpr (!Batch::kProduct) {  // products have the limbs of a plan, 64 at most
    if (limbs > kRadix8InvRows<W> && (!kStack || sizeof(W) == 4 || doubles)) {
      auto kfn = ntt_inv_rows_kernel<W, kRowsPerCta, false, Batch>;
      CERIUM_LAUNCH(kfn, dim3(256 / kRowsPerCta, limbs), kRowsPerCta * 16, 0, stream, batch, tw, twr, pcs);
      return;
    }
  }
  auto kfn = radix8_inv_rows_kernel<W, Batch>;
  CERIUM_LAUNCH(kfn, dim3(256 / kRadix8Rows, limbs), kRadix8Rows * 32, 0, stream, batch, tw, twr, pcs);
}

int launch_ntt_forward(cerium_context* ctx, const NttCall& c, cudaStream_t stream, bool lazy_out) {
  if (c.count == 0) return CERIUM_OK;
  return dispatch_word(ctx->word_bits, [&](auto tag) -> int {
    using W = decltype(tag);
    for (int first = 0; first < c.count; first += kMaxBatch) {
      const int cnt = std::min(kMaxBatch, c.count - first);
      StridedBatch<W> cols{};
      cols.in = static_cast<const W*>(c.in);
      cols.out = static_cast<W*>(c.out);
      cols.in_stride = c.in_stride;
      cols.out_stride = c.out_stride;
      cols.split = kMaxBatch;
      if (int rc = fill_batch<W>(ctx, cols, c.pos, c.prime, first, cnt)) return rc;
      StridedBatch<W> rows = cols;
      rows.in = static_cast<const W*>(c.out);
      rows.in_stride = c.out_stride;
      if (c.src_pos != nullptr) {
        GatherBatch<W> gb{};
        static_cast<StridedBatch<W>&>(gb) = cols;
        for (int b = 0; b < cnt; b++) {
          if (c.src_pos[first + b] > 0xffffu) return fail(CERIUM_ERR_INVALID, "limb slot exceeds 65535");
          gb.in_pos[b] = (uint16_t)c.src_pos[first + b];
        }
        ModLoader<W> ml{};
        for (int b = 0; b < cnt; b++)
          ml.small[b] = (c.src_prime != nullptr && ctx->moduli[c.src_prime[first + b]] < ((uint64_t)1 << 50)) ? 1 : 0;
        launch_fwd_cols<W>(ctx, gb, ml, cnt, stream);
      } else if (c.raised_in) {
        launch_fwd_cols<W>(ctx, cols, LazyLoader<W, kFpRaisedIn>{}, cnt, stream);
      } else if (c.lowered_in) {
        launch_fwd_cols<W>(ctx, cols, LazyLoader<W, kFpLoweredIn>{}, cnt, stream);
      } else {
        launch_fwd_cols<W>(ctx, cols, PlainLoader<W>{}, cnt, stream);
      }
      if (c.cols_only) continue;
      if (lazy_out) {
        launch_fwd_rows<W>(ctx, rows, LazyStoreEpilogue<W>{}, cnt, stream);
      } else {
        launch_fwd_rows<W>(ctx, rows, StoreEpilogue<W>{}, cnt, stream);
      }
    }
    CERIUM_LAUNCH_CHECK("ntt_forward");
    return CERIUM_OK;
  });
}

void inverse_last_words(const cerium_context* ctx, int k, uint64_t scale, uint64_t (&out)[4]) {
  const uint64_t q = ctx->moduli[k];
  for (int h = 0; h < 2; h++) {
    const uint64_t w = host::mulmod(h == 0 ? ctx->ninv[k] : ctx->w1ninv[k], scale % q, q);
    if (ctx->fp_ok[k]) {
      const double wd = host::centred(w, q), wq = wd / (double)q;
      std::memcpy(&out[2 * h], &wd, 8);
      std::memcpy(&out[2 * h + 1], &wq, 8);
    } else {
      out[2 * h] = w;
      out[2 * h + 1] = host::shoup(w, q, ctx->word_bits);
    }
  }
}

int launch_ntt_inverse(cerium_context* ctx, const NttCall& c, cudaStream_t stream, const void* last, const void* add) {
  if (c.count == 0) return CERIUM_OK;
  return dispatch_word(ctx->word_bits, [&](auto tag) -> int {
    using W = decltype(tag);
    for (int first = 0; first < c.count; first += kMaxBatch) {
      const int cnt = std::min(kMaxBatch, c.count - first);
      StridedBatch<W> sb{};
      sb.in = static_cast<const W*>(c.in);
      sb.out = static_cast<W*>(c.out);
      sb.in_stride = c.in_stride;
      sb.out_stride = c.out_stride;
      sb.split = kMaxBatch;
      sb.in_elt = c.in_galois;
      if (int rc = fill_batch<W>(ctx, sb, c.pos, c.prime, first, cnt)) return rc;
      InvScale<W> sc{};
      if (last != nullptr) sc.last = static_cast<const W*>(last) + 4 * (size_t)first;
      if (add != nullptr) sc.add = static_cast<const W*>(add) + first;
      if (c.src_pos != nullptr) {
        // entry b reads limb src_pos[b] of `in` and writes limb pos[b] of `out`
        GatherBatch<W> gb{};
        static_cast<StridedBatch<W>&>(gb) = sb;
        for (int b = 0; b < cnt; b++) {
          if (c.src_pos[first + b] > 0xffffu) return fail(CERIUM_ERR_INVALID, "limb slot exceeds 65535");
          gb.in_pos[b] = (uint16_t)c.src_pos[first + b];
        }
        launch_inv_rows<W>(ctx, gb, cnt, stream);
      } else if (c.factor != nullptr) {
        ProductBatch<W> pb{};
        static_cast<StridedBatch<W>&>(pb) = sb;
        pb.factor = static_cast<const W*>(c.factor);
        launch_inv_rows<W>(ctx, pb, cnt, stream);
      } else {
        int doubles = 0;
        for (int b = 0; b < cnt; b++) doubles += ctx->fp_ok[c.prime[first + b]] ? 1 : 0;
        launch_inv_rows<W>(ctx, sb, cnt, stream, 2 * doubles > cnt);
      }
      launch_inv_cols<W>(ctx, sb, sc, cnt, stream);
    }
    CERIUM_LAUNCH_CHECK("ntt_inverse");
    return CERIUM_OK;
  });
}

int launch_sud(cerium_context* ctx, const SudCall& c, cudaStream_t stream) {
  if (c.count == 0) return CERIUM_OK;
  return dispatch_word(ctx->word_bits, [&](auto tag) -> int {
    using W = decltype(tag);
    const int bits = ctx->word_bits;
    if (c.split > 0 && c.count > kSudMaxBatch) return fail(CERIUM_ERR_INVALID, "sud: a two-polynomial launch holds at most 128 limbs");
    {
      // the tail reads minuend and addend as 16-byte vectors
      const size_t wb = sizeof(W);
      const uintptr_t ptrs = (uintptr_t)c.minuend | (uintptr_t)c.minuend2 | (uintptr_t)c.addend | (uintptr_t)c.addend2;
      if (ptrs % 16 != 0 || (c.minuend_stride * wb) % 16 != 0 || (c.addend != nullptr && (c.addend_stride * wb) % 16 != 0))
        return fail(CERIUM_ERR_INVALID, "sud: minuend and addend limbs must be 16-byte aligned");
    }
    for (int first = 0; first < c.count; first += kSudMaxBatch) {
      const int cnt = std::min(kSudMaxBatch, c.count - first);
      StridedBatch<W> cols{};
      cols.in = static_cast<const W*>(c.src) + (c.src_stride ? (size_t)first * c.src_stride : 0);
      cols.out = static_cast<W*>(c.work) + (size_t)first * c.work_stride;
      cols.in_stride = c.src_stride;
      cols.out_stride = c.work_stride;
      cols.split = kMaxBatch;
      if (int rc = fill_batch<W>(ctx, cols, nullptr, c.prime + first, 0, cnt)) return rc;
      StridedBatch<W> rows = cols;
      rows.in = cols.out;
      rows.in_stride = c.work_stride;
      rows.out = static_cast<W*>(c.dst) + (size_t)first * c.dst_stride;
      rows.out_stride = c.dst_stride;
      SudEpilogue<W> epi{};
      epi.minuend = static_cast<const W*>(c.minuend) + (size_t)first * c.minuend_stride;
      epi.minuend_stride = c.minuend_stride;
      epi.addend = c.addend ? static_cast<const W*>(c.addend) + (size_t)first * c.addend_stride : nullptr;
      epi.addend_stride = c.addend_stride;
      epi.addend_elt = c.addend_galois;
      epi.store_elt = c.store_galois;
      epi.split = kSudMaxBatch;
      if (c.split > 0) {
        // second polynomial: entry b lands at slot b - split of dst2 (the slot number itself stays b,
        // it also addresses the work stack), so the base is moved back by split limbs
        rows.split = c.split;
        rows.out2 = static_cast<W*>(c.dst2) - (ptrdiff_t)c.split * (ptrdiff_t)c.dst_stride;
        epi.split = c.split;
        epi.minuend2 = static_cast<const W*>(c.minuend2);
        epi.addend2 = static_cast<const W*>(c.addend2);
      }
      for (int b = 0; b < cnt; b++) {
        const uint64_t q = ctx->moduli[c.prime[first + b]];
        const uint64_t f = c.factor[first + b] % q;
        if (ctx->fp_ok[c.prime[first + b]]) {
          const double fd = host::centred(f, q), fq = fd / (double)q;
          std::memcpy(&epi.factor[b], &fd, sizeof(W));
          std::memcpy(&epi.factor_shoup[b], &fq, sizeof(W));
        } else {
          epi.factor[b] = (W)f;
          epi.factor_shoup[b] = (W)host::shoup(f, q, bits);
        }
      }
      if (c.cols_done) {
        // the rows only
      } else if (c.reduce_src) {
        ReduceLoader<W> ld{};
        ld.src_q = (W)c.src_q;
        ld.pre_add = (W)c.pre_add;
        for (int b = 0; b < cnt; b++) ld.post_sub[b] = c.post_sub ? (W)c.post_sub[first + b] : (W)0;
        if (c.src_pos != nullptr) {
          GatherBatch<W> gb{};
          static_cast<StridedBatch<W>&>(gb) = cols;
          gb.in = static_cast<const W*>(c.src);
          for (int b = 0; b < cnt; b++) gb.in_pos[b] = (uint16_t)c.src_pos[first + b];
          launch_fwd_cols<W>(ctx, gb, ld, cnt, stream);
        } else {
          launch_fwd_cols<W>(ctx, cols, ld, cnt, stream);
        }
      } else if (c.lazy_src) {
        launch_fwd_cols<W>(ctx, cols, LazyLoader<W, kFpLoweredIn>{}, cnt, stream);
      } else {
        launch_fwd_cols<W>(ctx, cols, PlainLoader<W>{}, cnt, stream);
      }
      launch_fwd_rows<W>(ctx, rows, epi, cnt, stream);
    }
    CERIUM_LAUNCH_CHECK("sud");
    return CERIUM_OK;
  });
}

// ---------------------------------------------------------------------------------------
// base conversion
// ---------------------------------------------------------------------------------------

// Packs several small tables into one device allocation: append() returns the byte offset
// of a 16-byte aligned copy of the data.
struct Blob {
  std::vector<char> bytes;
  size_t append(const void* p, size_t n) {
    const size_t off = bytes.size();
    bytes.resize(off + (n + 15) / 16 * 16, 0);
    if (n) std::memcpy(bytes.data() + off, p, n);
    return off;
  }
  template <typename W>
  size_t append_words(const std::vector<uint64_t>& v) {
    std::vector<W> t(v.size());
    for (size_t i = 0; i < v.size(); i++) t[i] = (W)v[i];
    return append(t.data(), t.size() * sizeof(W));
  }
};

int create_bconv(cerium_context* ctx, cerium_bconv** out, int mode, const uint32_t* in_primes, int n_in,
                 const uint32_t* out_primes, int n_out, const BconvOptions& opt) {
  if (!ctx || !out || !in_primes || !out_primes) return fail(CERIUM_ERR_INVALID, "bconv_create: null argument");
  if (mode != CERIUM_BCONV_LAZY && mode != CERIUM_BCONV_EXACT) return fail(CERIUM_ERR_INVALID, "bconv_create: unknown mode");
  if (n_in < 1 || n_in > kMmaMaxInputs || n_out < 1 || n_out > 255) return fail(CERIUM_ERR_INVALID, "bconv_create: need 1..64 inputs and 1..255 outputs");
  if (!opt.out_pos.empty() && (int)opt.out_pos.size() != n_out) return fail(CERIUM_ERR_INVALID, "bconv_create: out_pos size");
  if (!opt.in_pos.empty() && (int)opt.in_pos.size() != n_in) return fail(CERIUM_ERR_INVALID, "bconv_create: in_pos size");
  for (int i = 0; i < n_in; i++)
    if (in_primes[i] >= (uint32_t)ctx->n_primes) return fail(CERIUM_ERR_INVALID, "bconv_create: input prime index out of range");
  for (int j = 0; j < n_out; j++)
    if (out_primes[j] >= (uint32_t)ctx->n_primes) return fail(CERIUM_ERR_INVALID, "bconv_create: output prime index out of range");
  // the unreduced sum of products must fit the two-word accumulator
  for (int j = 0; j < n_out; j++) {
    long double sum = 0;
    for (int i = 0; i < n_in; i++) sum += (long double)ctx->moduli[in_primes[i]] * (long double)ctx->moduli[out_primes[j]];
    if (sum >= (ctx->word_bits == 32 ? 1.8e19L : 3.4e38L))
      return fail(CERIUM_ERR_UNSUPPORTED, "bconv_create: too many inputs for primes this wide (sum of products overflows)");
  }
  DeviceGuard guard(ctx->device);
  if (!guard.ok) return fail(CERIUM_ERR_CUDA, "bconv_create: cannot select device");
  auto* bc = new cerium_bconv();
  bc->ctx = ctx;
  bc->mode = mode;
  bc->lazy_out = opt.lazy_out;
  bc->I = n_in;
  bc->O = n_out;
  bc->in_primes.assign(in_primes, in_primes + n_in);
  const auto& m = ctx->moduli;
  const int bits = ctx->word_bits;
  // [Qhat_i^-1]_{q_i}
  std::vector<uint64_t> inv(n_in), inv_shoup(n_in);
  for (int i = 0; i < n_in; i++) {
    const uint64_t qi = m[in_primes[i]];
    uint64_t p = 1 % qi;
    for (int k = 0; k < n_in; k++)
      if (k != i) p = host::mulmod(p, m[in_primes[k]] % qi, qi);
    inv[i] = host::invmod(p, qi);
    if (qi > 1 && inv[i] == 0 && n_in > 1) {
      delete bc;
      return fail(CERIUM_ERR_INVALID, "bconv_create: input primes are not pairwise distinct");
    }
    if (n_in == 1) inv[i] = 1;
    inv_shoup[i] = host::shoup(inv[i], qi, bits);
  }
  bc->inv_host = inv;
  std::vector<uint64_t> factors((size_t)n_out * n_in);
  for (int j = 0; j < n_out; j++) {
    const uint64_t pj = m[out_primes[j]];
    for (int i = 0; i < n_in; i++) {
      uint64_t qhat = 1 % pj;
      for (int k = 0; k < n_in; k++)
        if (k != i) qhat = host::mulmod(qhat, m[in_primes[k]] % pj, pj);
      factors[(size_t)j * n_in + i] =
          mode == CERIUM_BCONV_LAZY ? host::mulmod(inv[i] % pj, qhat, pj) : qhat;
    }
  }
  std::vector<uint64_t> in_add, out_sub;
  if (opt.round_half) {
    // floor(P/2) = (P-1)/2 for odd P = prod of input primes
    in_add.resize(n_in);
    out_sub.resize(n_out);
    std::vector<uint32_t> idx(in_primes, in_primes + n_in);
    auto half_mod = [&](uint64_t q) {
      const uint64_t p = host::product_mod(m, idx, q);
      const uint64_t pm1 = (p + q - 1 % q) % q;
      return host::mulmod(pm1, host::invmod(2, q), q);
    };
    for (int i = 0; i < n_in; i++) {
      in_add[i] = half_mod(m[in_primes[i]]);
      // inputs that arrive pre-scaled by [Qhat_i^-1] need the rounding term scaled alike:
      // (x + h) * inv = x * inv + h * inv  (mod q_i)
      if (mode == CERIUM_BCONV_EXACT && opt.prescaled) in_add[i] = host::mulmod(in_add[i], inv[i], m[in_primes[i]]);
    }
    for (int j = 0; j < n_out; j++) out_sub[j] = half_mod(m[out_primes[j]]);
  }
  bc->in_add_host = in_add;
  const bool use_inv = mode == CERIUM_BCONV_EXACT && !opt.prescaled && n_in > 1;
  Blob blob;
  size_t o_inv = 0, o_invs = 0;
  dispatch_word(bits, [&](auto tag) -> int {
    using W = decltype(tag);
    o_inv = blob.append_words<W>(inv);
    o_invs = blob.append_words<W>(inv_shoup);
    return 0;
  });
  size_t o_outc = 0, o_table = 0;
  dispatch_word(bits, [&](auto tag) -> int {
    using W = decltype(tag);
    // table entry of (output j, byte plane m, input i, byte k): byte m of factor[j][i] * 2^(8k) mod p_j, laid out as
    // the fragments of an m16n8k32 product (bconv_mma.cuh)
    const auto steps_of = [](int inputs) {
      const int steps = (inputs * (int)sizeof(W) + 31) / 32;
      return sizeof(W) == 4 && steps == 3 ? 4 : steps;  // kernels with fragments in registers come for 1, 2 and 4 steps
    };
    // A step more shares the launch of a longer conversion as long as the fragments stay in registers: digits of 5 and 4 64-bit
    // limbs (9 limbs in a rotation) 79.8 us apart, 78.5 together; 9 and 8 (33 limbs) 254 apart, 291 together; 32-bit words, 9 and
    // 8 limbs (25) 87.3 / 85.6, 17 and 16 (33) 110.5 / 107.5.
    const int together = steps_of(std::max(n_in, opt.inputs_together));
    bc->steps = together <= kMmaRegSteps<W> ? together : steps_of(n_in);
    std::vector<uint4> table(bconv_mma_table_entries<W>(n_out, bc->steps), make_uint4(0, 0, 0, 0));
    unsigned char* bytes = reinterpret_cast<unsigned char*>(table.data());
    std::vector<BconvMmaOut<W>> outc(n_out);
    for (int j = 0; j < n_out; j++) {
      const uint64_t q = m[out_primes[j]];
      for (int i = 0; i < n_in; i++)
        for (int k = 0; k < (int)sizeof(W); k++) {
          const uint64_t g = host::mulmod(factors[(size_t)j * n_in + i], ((uint64_t)1 << (8 * k)) % q, q);
          const int group = j / kMmaRows<W>, in_group = j % kMmaRows<W>, col = i * (int)sizeof(W) + k;
          const bool pair = sizeof(W) == 8 || n_out - group * kMmaRows<W> <= 8;
          for (int b = 0; b < (int)sizeof(W); b++) {
            const int frag = pair ? b / 2 : b, row = pair ? in_group + 8 * (b & 1) : in_group;
            const int step = col / 32, lane = (row % 8) * 4 + col % 16 / 4, reg = row / 8 + 2 * (col % 32 / 16);
            const size_t entry = bconv_mma_entry<W>(group, bc->steps) + ((size_t)frag * bc->steps + step) * 32 + lane;
            bytes[entry * 16 + reg * 4 + col % 4] = (unsigned char)(g >> (8 * b));
          }
        }
      outc[j] = bconv_mma_constants<W>(q, out_sub.empty() ? 0 : out_sub[j]);
      outc[j].pos = opt.out_pos.empty() ? (uint32_t)j : opt.out_pos[j];
      bc->all_wide = bc->all_wide && outc[j].cls == kMmaWide;
    }
    o_outc = blob.append(outc.data(), outc.size() * sizeof(BconvMmaOut<W>));
    o_table = blob.append(table.data(), table.size() * sizeof(uint4));
    return 0;
  });
  const size_t o_ip = blob.append(bc->in_primes.data(), bc->in_primes.size() * 4);
  const size_t o_ipos = blob.append(opt.in_pos.data(), opt.in_pos.size() * 4);
  if (cudaMalloc(&bc->d_block, blob.bytes.size() + 16) != cudaSuccess) {
    delete bc;
    return fail(CERIUM_ERR_CUDA, "bconv_create: cudaMalloc failed");
  }
  if (cudaMemcpy(bc->d_block, blob.bytes.data(), blob.bytes.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
      uploads_done() != cudaSuccess) {
    cudaFree(bc->d_block);
    delete bc;
    return fail(CERIUM_ERR_CUDA, "bconv_create: upload failed");
  }
  char* base = static_cast<char*>(bc->d_block);
  bc->d_outc = base + o_outc;
  bc->d_table = base + o_table;
  bc->d_inv = use_inv ? base + o_inv : nullptr;
  bc->d_inv_shoup = use_inv ? base + o_invs : nullptr;
  bc->d_in_prime = reinterpret_cast<uint32_t*>(base + o_ip);
  bc->d_in_pos = opt.in_pos.empty() ? nullptr : reinterpret_cast<uint32_t*>(base + o_ipos);
  *out = bc;
  return CERIUM_OK;
}

// Kernel of a batch: fragments in registers up to the number of steps they fit for, then the way outputs are finished.  half: the
// inputs end in the first half of the last step.  more: 24 warps to an SM and not 16, for words of 64 bits that the kernel
// prepares itself and reads its fragments for: where 16 do not hold the grid at once (9 inputs to 35 outputs 34.0 -> 21.7 us, 24
// to 35 56.9 -> 40.2); with fewer CTAs 128 registers are better (24 inputs to 13 outputs 27.3 / 29.7, 32 to 24 34.4 / 40.4).
template <typename W, bool kPrepare>
static auto bconv_mma_pick(int steps, int finish, bool half, bool more) -> decltype(&bconv_mma_kernel<W, 0, kMmaGeneral, kPrepare>) {
  if constexpr (sizeof(W) == 8) {
    if (kPrepare && more && steps > kMmaRegSteps<W>)
      return finish == kMmaBig ? bconv_mma_kernel<W, 0, kMmaBig, kPrepare, false, 24> : bconv_mma_kernel<W, 0, kMmaGeneral, kPrepare, false, 24>;
    if (finish == kMmaBig) return bconv_mma_kernel<W, 0, kMmaBig, kPrepare>;
  }
  if (finish <= kMmaLazyAdd && !kPrepare) {
    const bool add = finish == kMmaLazyAdd;
    if (steps == 1 && half) return add ? bconv_mma_kernel<W, 1, kMmaLazyAdd, false, true> : bconv_mma_kernel<W, 1, kMmaLazy, false, true>;
    if (steps == 1) return add ? bconv_mma_kernel<W, 1, kMmaLazyAdd, false> : bconv_mma_kernel<W, 1, kMmaLazy, false>;
    if (steps == 2 && half) return add ? bconv_mma_kernel<W, 2, kMmaLazyAdd, false, true> : bconv_mma_kernel<W, 2, kMmaLazy, false, true>;
    if (steps == 2) return add ? bconv_mma_kernel<W, 2, kMmaLazyAdd, false> : bconv_mma_kernel<W, 2, kMmaLazy, false>;
    if constexpr (sizeof(W) == 4)
      if (steps == 4) return add ? bconv_mma_kernel<W, 4, kMmaLazyAdd, false> : bconv_mma_kernel<W, 4, kMmaLazy, false>;
  }
  if (steps == 1) return bconv_mma_kernel<W, 1, kMmaGeneral, kPrepare>;
  if (steps == 2) return bconv_mma_kernel<W, 2, kMmaGeneral, kPrepare>;
  if constexpr (sizeof(W) == 4)
    if (steps == 4) return bconv_mma_kernel<W, 4, kMmaGeneral, kPrepare>;
  return bconv_mma_kernel<W, 0, kMmaGeneral, kPrepare>;
}

template <typename W>
static int launch_bconv_words(cerium_context* ctx, const BconvCall* calls, int count, cudaStream_t stream) {
  for (int first = 0; first < count;) {
    // conversions of one launch share the number of steps (BconvOptions::inputs_together)
    BconvMmaBatch<W> batch{};
    const int steps = calls[first].bc->steps;
    bool lazy = true, prepare = false, add = false;
    int cnt = 0, max_groups = 1, max_i = 1;
    for (; cnt < kMmaMaxBatch && first + cnt < count && calls[first + cnt].bc->steps == steps; cnt++) {
      const BconvCall& c = calls[first + cnt];
      const cerium_bconv* bc = c.bc;
      BconvMmaDesc<W>& d = batch.d[cnt];
      d.in = static_cast<const W*>(c.in);
      d.out = static_cast<W*>(c.out);
      d.in_stride = c.in_stride;
      d.out_stride = c.out_stride;
      d.inv = static_cast<const W*>(bc->d_inv);
      d.inv_shoup = static_cast<const W*>(bc->d_inv_shoup);
      d.in_prime = bc->d_in_prime;
      d.in_pos = bc->d_in_pos;
      d.table = static_cast<const uint4*>(bc->d_table);
      d.outc = static_cast<const BconvMmaOut<W>*>(bc->d_outc);
      d.I = bc->I;
      d.O = bc->O;
      d.steps = steps;
      lazy = lazy && bc->lazy_out && bc->all_wide;
      prepare = prepare || bc->d_inv != nullptr;
      add = add || !bc->in_add_host.empty();
      max_i = std::max(max_i, bc->I);
      max_groups = std::max(max_groups, bconv_mma_groups<W>(bc->O));
    }
    const int finish = sizeof(W) == 8 && max_i > kMmaPairInputs ? kMmaBig : !lazy ? kMmaGeneral : add ? kMmaLazyAdd : kMmaLazy;
    const bool half = max_i * (int)sizeof(W) <= 32 * steps - 16;
    // a warp per group of outputs, at most 8 to a CTA
    const int slices = (max_groups + kMmaMaxWarps - 1) / kMmaMaxWarps, warps = (max_groups + slices - 1) / slices;
    const size_t smem = bconv_mma_smem_bytes<W>(max_i);
    const int ctas = kN / kMmaStage * cnt * slices;
    const auto resident = [&](int warps_per_sm) {
      return ctas <= std::min(warps_per_sm / warps, (int)(kSplitSmem / (smem + 1024))) * ctx->sm_count;
    };
    bool late = resident(prepare || (sizeof(W) == 4 && steps == kMmaRegSteps<W>) ? kMmaWarpsPerSm<W, 0, true> : kMmaWarpsPerSm<W, 0, false>);
    auto kfn = prepare ? bconv_mma_pick<W, true>(steps, finish, half, !late) : bconv_mma_pick<W, false>(steps, finish, half, false);
    if (prepare && sizeof(W) == 8 && steps > kMmaRegSteps<W>) late = resident(kMmaWarpsPerSm<W, 0, false>);
    if (smem > 48 * 1024) CERIUM_CUDA(allow_smem(kfn, bconv_mma_smem_bytes<W>(kMmaMaxInputs)));
    // Small CTAs that a kernel lets in at its start crowd on the SMs that have room first.  A grid that is resident at once asks for
    // the shared memory that keeps an SM to its share of the CTAs, and leaves the rest to the next kernel.  After an addition, 32-bit
    // words: 1 input to 17 outputs 9.9 -> 5.0 us, 16 to 24 10.7 -> 6.1; called alone, 20 to 35 8.0 -> 6.4, 64-bit words 12 to 24 20.2 -> 16.7;
    // rotations of 9 limbs of 32-bit words 46.8 -> 45.6, of 24 limbs in digits of 12 with 15 extension limbs 210 -> 199.  Not one
    // warp of 64-bit words, which gains nothing and takes room from the next kernel (inverse transform, 5 to 5, forward 25.2 -> 26.8).
    size_t room = smem;
    if (late && (sizeof(W) == 4 || warps > 1)) {
      const size_t share = (size_t)((ctas + ctx->sm_count - 1) / ctx->sm_count);
      room = std::max(smem, std::min(kSplitSmem / (share + 1), (size_t)48 * 1024));
    }
    CERIUM_LAUNCH(kfn, dim3(kN / kMmaStage, cnt, slices), 32 * warps, room, stream, late, batch,
                  static_cast<const PrimeConst<W>*>(ctx->d_pcs));
    first += cnt;
  }
  CERIUM_LAUNCH_CHECK("bconv");
  return CERIUM_OK;
}

int launch_bconv(cerium_context* ctx, const BconvCall* calls, int count, cudaStream_t stream) {
  if (count == 0) return CERIUM_OK;
  return dispatch_word(ctx->word_bits, [&](auto tag) -> int { return launch_bconv_words<decltype(tag)>(ctx, calls, count, stream); });
}

}  // namespace cerium

using namespace cerium;

// ---------------------------------------------------------------------------------------
// extern "C"
// ---------------------------------------------------------------------------------------

extern "C" {

int cerium_version(void) { return 100; }

const char* cerium_last_error(void) { return g_last_error.c_str(); }

int cerium_context_create(cerium_context** out, int device, int log_n, int word_bits, const uint64_t* moduli,
                          int n_moduli) {
  if (!out || !moduli) return fail(CERIUM_ERR_INVALID, "context_create: null argument");
  if (log_n != kLogN) return fail(CERIUM_ERR_UNSUPPORTED, "context_create: only log_n = 16 is built");
  if (word_bits != 32 && word_bits != 64) return fail(CERIUM_ERR_INVALID, "context_create: word_bits must be 32 or 64");
  if (n_moduli < 1 || n_moduli > 255) return fail(CERIUM_ERR_INVALID, "context_create: need 1..255 moduli");
  const uint64_t limit = word_bits == 32 ? ((uint64_t)1 << 30) : ((uint64_t)1 << 60);
  for (int k = 0; k < n_moduli; k++) {
    if (moduli[k] >= limit) return fail(CERIUM_ERR_INVALID, "context_create: modulus too large for the word size");
    if (!host::is_prime(moduli[k]) || (moduli[k] - 1) % ((uint64_t)2 << log_n))
      return fail(CERIUM_ERR_INVALID, "context_create: modulus is not a prime congruent to 1 mod 2N");
    for (int j = 0; j < k; j++)
      if (moduli[j] == moduli[k]) return fail(CERIUM_ERR_INVALID, "context_create: duplicate modulus");
  }
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
    return fail(CERIUM_ERR_CUDA, "context_create: no CUDA device (this library has no CPU path)");
  if (device < 0 || device >= ndev) return fail(CERIUM_ERR_INVALID, "context_create: device out of range");
  DeviceGuard guard(device);
  if (!guard.ok) return fail(CERIUM_ERR_CUDA, "context_create: cannot select device");
  auto* ctx = new cerium_context();
  ctx->device = device;
  ctx->logn = log_n;
  ctx->word_bits = word_bits;
  ctx->n_primes = n_moduli;
  ctx->moduli.assign(moduli, moduli + n_moduli);
  ctx->psi.resize(n_moduli);
  ctx->inverses.reset(new std::atomic<uint64_t>[(size_t)n_moduli * n_moduli]());
  if (cudaDeviceGetAttribute(&ctx->sm_count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || ctx->sm_count < 1) {
    delete ctx;
    return fail(CERIUM_ERR_CUDA, "context_create: cannot read the number of SMs");
  }
  if (const char* arith = std::getenv("CERIUM_B200_NTT_ARITH")) ctx->allow_fp = std::strcmp(arith, "int") != 0;
  const size_t n = kN;
  int rc = dispatch_word(word_bits, [&](auto tag) -> int {
    using W = decltype(tag);
    using Pair = typename WordTraits<W>::Pair;
    std::vector<Pair> fwd(n * n_moduli), inv(n * n_moduli);
    std::vector<Pair> rfwd((size_t)kRowTwPerPrime * n_moduli), rinv((size_t)kRowTwPerPrime * n_moduli);
    std::vector<PrimeConst<W>> pcs(n_moduli);
    for (int k = 0; k < n_moduli; k++) {
      const uint64_t q = moduli[k];
      host::PrimeTables t = host::build_prime_tables(q, log_n, word_bits);
      ctx->psi[k] = t.psi;
      // primes below 2^50 run their butterflies on doubles: the tables then hold the centred
      // twiddle and its correctly rounded quotient by q instead of the twiddle and its Shoup word
      const bool fp = word_bits == 64 && q < ((uint64_t)1 << 50) && ctx->allow_fp;
      auto fp_pair = [&](uint64_t w) {
        const double wd = host::centred(w, q);
        const double wq = wd / (double)q;
        uint64_t a, b;
        std::memcpy(&a, &wd, 8);
        std::memcpy(&b, &wq, 8);
        return WordTraits<W>::make((W)a, (W)b);
      };
      for (size_t i = 0; i < n; i++) {
        if (fp) {
          fwd[k * n + i] = fp_pair(t.w[i]);
          inv[k * n + i] = fp_pair(t.wi[i]);
        } else {
          fwd[k * n + i] = WordTraits<W>::make((W)t.w[i], (W)host::shoup(t.w[i], q, word_bits));
          inv[k * n + i] = WordTraits<W>::make((W)t.wi[i], (W)host::shoup(t.wi[i], q, word_bits));
        }
      }
      for (int h = 0; h < 256; h++)
        for (int t = 0; t < 4; t++)
          for (int g = 0; g < (1 << t); g++)
            for (int u = 0; u < 16; u++) {
              const size_t src = k * n + (((size_t)(4096 + 16 * h + u)) << t) + g;
              if (fp) {
                // twiddles only (the kernel computes their quotients), two per entry: double number
                // 2^t + g of the group's 16 (see lane_tw_fp)
                const int slot = (1 << t) + g;
                const size_t dst = (size_t)k * kRowTwPerPrime + ((size_t)h * 8 + (slot >> 1)) * 16 + u;
                if (slot & 1) {
                  rfwd[dst].y = fwd[src].x;
                  rinv[dst].y = inv[src].x;
                } else {
                  rfwd[dst].x = fwd[src].x;
                  rinv[dst].x = inv[src].x;
                }
              } else {
                const size_t dst = (size_t)k * kRowTwPerPrime + ((size_t)h * 15 + ((1 << t) - 1 + g)) * 16 + u;
                rfwd[dst] = fwd[src];
                rinv[dst] = inv[src];
              }
            }
      PrimeConst<W>& pc = pcs[k];
      std::memset(&pc, 0, sizeof(pc));
      pc.q = (W)q;
      pc.q2 = (W)(2 * q);
      pc.mu_hi = (W)t.mu_hi;
      pc.mu_lo = (W)t.mu_lo;
      pc.one_shoup = (W)host::shoup(1, q, word_bits);
      pc.ninv = (W)t.ninv;
      pc.ninv_shoup = (W)host::shoup(t.ninv, q, word_bits);
      const uint64_t w1 = host::mulmod(t.wi[1], t.ninv, q);
      pc.w1ninv = (W)w1;
      pc.w1ninv_shoup = (W)host::shoup(w1, q, word_bits);
      pc.lazy_ok = (W)((word_bits == 64 && q < ((uint64_t)1 << 52)) ? 1 : 0);
      ctx->fp_ok.push_back(fp ? 1 : 0);
      ctx->ninv.push_back(t.ninv);
      ctx->w1ninv.push_back(w1);
      if (fp) {
        const double qinv = 1.0 / (double)q;
        uint64_t bits;
        std::memcpy(&bits, &qinv, 8);
        pc.fp_ok = 1;
        pc.fp_qinv = (W)bits;
        const auto ni = fp_pair(t.ninv), w1 = fp_pair(host::mulmod(t.wi[1], t.ninv, q));
        pc.fp_ninv = ni.x;
        pc.fp_ninv_q = ni.y;
        pc.fp_w1ninv = w1.x;
        pc.fp_w1ninv_q = w1.y;
      }
    }
    CERIUM_CUDA(cudaMalloc(&ctx->d_tw_fwd, fwd.size() * sizeof(Pair)));
    CERIUM_CUDA(cudaMalloc(&ctx->d_tw_inv, inv.size() * sizeof(Pair)));
    CERIUM_CUDA(cudaMalloc(&ctx->d_pcs, pcs.size() * sizeof(PrimeConst<W>)));
    CERIUM_CUDA(cudaMalloc(&ctx->d_twr_fwd, rfwd.size() * sizeof(Pair)));
    CERIUM_CUDA(cudaMalloc(&ctx->d_twr_inv, rinv.size() * sizeof(Pair)));
    CERIUM_CUDA(cudaMalloc(reinterpret_cast<void**>(&ctx->d_status), 16));
    CERIUM_CUDA(cudaMemset(ctx->d_status, 0, 16));
    CERIUM_CUDA(cudaMemcpy(ctx->d_twr_fwd, rfwd.data(), rfwd.size() * sizeof(Pair), cudaMemcpyHostToDevice));
    CERIUM_CUDA(cudaMemcpy(ctx->d_twr_inv, rinv.data(), rinv.size() * sizeof(Pair), cudaMemcpyHostToDevice));
    CERIUM_CUDA(cudaMemcpy(ctx->d_tw_fwd, fwd.data(), fwd.size() * sizeof(Pair), cudaMemcpyHostToDevice));
    CERIUM_CUDA(cudaMemcpy(ctx->d_tw_inv, inv.data(), inv.size() * sizeof(Pair), cudaMemcpyHostToDevice));
    CERIUM_CUDA(cudaMemcpy(ctx->d_pcs, pcs.data(), pcs.size() * sizeof(PrimeConst<W>), cudaMemcpyHostToDevice));
    CERIUM_CUDA(uploads_done());
    return CERIUM_OK;
  });
  if (rc != CERIUM_OK) {
    cerium_context_destroy(ctx);
    return rc;
  }
  *out = ctx;
  return CERIUM_OK;
}

int cerium_context_destroy(cerium_context* ctx) {
  if (!ctx) return CERIUM_OK;
  DeviceGuard guard(ctx->device);
  cudaFree(ctx->d_tw_fwd);
  cudaFree(ctx->d_tw_inv);
  cudaFree(ctx->d_pcs);
  cudaFree(ctx->d_twr_fwd);
  cudaFree(ctx->d_twr_inv);
  cudaFree(ctx->d_status);
  delete ctx;
  return CERIUM_OK;
}

int cerium_context_check(cerium_context* ctx) {
  if (!ctx) return fail(CERIUM_ERR_INVALID, "context_check: null context");
  DeviceGuard guard(ctx->device);
  uint32_t st = 0;
  CERIUM_CUDA(cudaMemcpy(&st, ctx->d_status, sizeof(st), cudaMemcpyDeviceToHost));  // waits for the device's work
  if (st == 0) return CERIUM_OK;
  CERIUM_CUDA(cudaMemset(ctx->d_status, 0, sizeof(st)));
  CERIUM_CUDA(uploads_done());
  std::string msg = "context_check:";
  if (st & kStatusBconvShape) msg += " a base-conversion table entry exceeded the shape bounds of its launch (that conversion was skipped);";
  if (st & ~kStatusBconvShape) msg += " unknown status bits;";
  return fail(CERIUM_ERR_INVALID, msg);
}

int cerium_context_word_bits(const cerium_context* ctx) { return ctx ? ctx->word_bits : 0; }
int cerium_context_num_moduli(const cerium_context* ctx) { return ctx ? ctx->n_primes : 0; }
uint64_t cerium_context_modulus(const cerium_context* ctx, int k) {
  return (ctx && k >= 0 && k < ctx->n_primes) ? ctx->moduli[k] : 0;
}
uint64_t cerium_context_root(const cerium_context* ctx, int k) {
  return (ctx && k >= 0 && k < ctx->n_primes) ? ctx->psi[k] : 0;
}

static int ntt_common(cerium_context* ctx, bool forward, void* out, size_t out_stride, const void* in,
                      size_t in_stride, const uint32_t* prime_idx, int count, void* stream) {
  if (!ctx) return fail(CERIUM_ERR_INVALID, "ntt: null context");
  if (count < 0) return fail(CERIUM_ERR_INVALID, "ntt: negative count");
  if (count == 0) return CERIUM_OK;
  if (!prime_idx) return fail(CERIUM_ERR_INVALID, "ntt: null prime_idx");
  if (count > 65536) return fail(CERIUM_ERR_INVALID, "ntt: more than 65536 limbs in one call");
  if (int rc = check_stack(out, out_stride, ctx->word_bytes(), "ntt: out")) return rc;
  if (int rc = check_stack(in, in_stride, ctx->word_bytes(), "ntt: in")) return rc;
  DeviceGuard guard(ctx->device);
  NttCall c{in, out, in_stride, out_stride, nullptr, prime_idx, count};
  return forward ? launch_ntt_forward(ctx, c, (cudaStream_t)stream)
                 : launch_ntt_inverse(ctx, c, (cudaStream_t)stream);
}

int cerium_ntt_forward(cerium_context* ctx, void* out, size_t out_stride, const void* in, size_t in_stride,
                       const uint32_t* prime_idx, int count, void* stream) {
  return ntt_common(ctx, true, out, out_stride, in, in_stride, prime_idx, count, stream);
}

int cerium_ntt_inverse(cerium_context* ctx, void* out, size_t out_stride, const void* in, size_t in_stride,
                       const uint32_t* prime_idx, int count, void* stream) {
  return ntt_common(ctx, false, out, out_stride, in, in_stride, prime_idx, count, stream);
}

static int ntt_ptrs_common(cerium_context* ctx, bool forward, void* const* outs, const void* const* ins,
                           const uint32_t* bases, size_t num_bases, void* stream) {
  if (!ctx) return fail(CERIUM_ERR_INVALID, "ntt_ptrs: null context");
  if (num_bases == 0) return CERIUM_OK;
  if (!outs || !ins || !bases) return fail(CERIUM_ERR_INVALID, "ntt_ptrs: null table");
  if (num_bases > 65535) return fail(CERIUM_ERR_INVALID, "ntt_ptrs: more than 65535 limbs in one call");
  DeviceGuard guard(ctx->device);
  cudaStream_t s = (cudaStream_t)stream;
  return dispatch_word(ctx->word_bits, [&](auto tag) -> int {
    using W = decltype(tag);
    PointerBatch<W> pb{reinterpret_cast<W* const*>(outs), reinterpret_cast<const W* const*>(ins), bases, 1, 0};
    PointerBatch<W> inplace{reinterpret_cast<W* const*>(outs), reinterpret_cast<const W* const*>(outs), bases, 1, 0};
    const int cnt = (int)num_bases;
    if (forward) {
      launch_fwd_cols<W>(ctx, pb, PlainLoader<W>{}, cnt, s);
      launch_fwd_rows<W>(ctx, inplace, StoreEpilogue<W>{}, cnt, s);
    } else {
      launch_inv_rows<W>(ctx, pb, cnt, s);
      launch_inv_cols<W>(ctx, pb, InvScale<W>{}, cnt, s);
    }
    CERIUM_LAUNCH_CHECK("ntt_ptrs");
    return CERIUM_OK;
  });
}

int cerium_ntt_forward_ptrs(cerium_context* ctx, void* const* outs, const void* const* ins, const uint32_t* bases,
                            size_t num_bases, void* stream) {
  return ntt_ptrs_common(ctx, true, outs, ins, bases, num_bases, stream);
}

int cerium_ntt_inverse_ptrs(cerium_context* ctx, void* const* outs, const void* const* ins, const uint32_t* bases,
                            size_t num_bases, void* stream) {
  return ntt_ptrs_common(ctx, false, outs, ins, bases, num_bases, stream);
}

int cerium_sud_ptrs(cerium_context* ctx, void* const* outs, const void* const* ins, const uint32_t* bases,
                    size_t num_bases, const void* factors, void* stream) {
  if (!ctx) return fail(CERIUM_ERR_INVALID, "sud_ptrs: null context");
  if (num_bases == 0) return CERIUM_OK;
  if (!outs || !ins || !bases || !factors) return fail(CERIUM_ERR_INVALID, "sud_ptrs: null table");
  if (num_bases > 65535) return fail(CERIUM_ERR_INVALID, "sud_ptrs: more than 65535 limbs in one call");
  DeviceGuard guard(ctx->device);
  cudaStream_t s = (cudaStream_t)stream;
  return dispatch_word(ctx->word_bits, [&](auto tag) -> int {
    using W = decltype(tag);
    const int cnt = (int)num_bases;
    // column pass: second input of every entry -> output limb; row pass in place on the output
    PointerBatch<W> cols{reinterpret_cast<W* const*>(outs), reinterpret_cast<const W* const*>(ins), bases, 2, 1};
    PointerBatch<W> rows{reinterpret_cast<W* const*>(outs), reinterpret_cast<const W* const*>(outs), bases, 1, 0};
    PtrSudEpilogue<W> epi{reinterpret_cast<const W* const*>(ins), static_cast<const W*>(factors)};
    launch_fwd_cols<W>(ctx, cols, PlainLoader<W>{}, cnt, s);
    launch_fwd_rows<W>(ctx, rows, epi, cnt, s);
    CERIUM_LAUNCH_CHECK("sud_ptrs");
    return CERIUM_OK;
  });
}

int cerium_bconv_ptrs(cerium_context* ctx, void* const* outs, const size_t* n_out, const void* const* ins,
                      const size_t* n_in, const void* const* factors, const void* const* out_moduli,
                      size_t max_in, size_t max_out, size_t num_conversions, void* stream) {
  if (!ctx) return fail(CERIUM_ERR_INVALID, "bconv_ptrs: null context");
  if (num_conversions == 0) return CERIUM_OK;
  if (!outs || !n_out || !ins || !n_in || !factors || !out_moduli) return fail(CERIUM_ERR_INVALID, "bconv_ptrs: null table");
  if (max_in < 1 || max_out < 1 || max_in > 64 || max_out > 128) return fail(CERIUM_ERR_INVALID, "bconv_ptrs: bad shape bound");
  if (num_conversions > 65535) return fail(CERIUM_ERR_INVALID, "bconv_ptrs: more than 65535 conversions in one call");
  DeviceGuard guard(ctx->device);
  cudaStream_t s = (cudaStream_t)stream;
  return dispatch_word(ctx->word_bits, [&](auto tag) -> int {
    using W = decltype(tag);
    static bool smem_opt_in[kMaxDevices][2] = {};  // the attribute is per device
    // the shapes live on the device: size the shared memory for the caller's bounds (inputs staged per
    // thread when there are more than kBconvRegInputs of them)
    const size_t smem = bconv_smem_bytes<W>((int)max_in, (int)max_out);
    if (smem > 200 * 1024) return fail(CERIUM_ERR_UNSUPPORTED, "bconv_ptrs: conversion needs more than 200 KiB of shared memory");
    if (smem > 48 * 1024) {
      const int slot = sizeof(W) == 4 ? 0 : 1;
      const int dev = ctx->device;
      if (dev < 0 || dev >= kMaxDevices || !smem_opt_in[dev][slot]) {
        CERIUM_CUDA(cudaFuncSetAttribute(bconv_ptrs_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        if (dev >= 0 && dev < kMaxDevices) smem_opt_in[dev][slot] = true;
      }
    }
    auto kfn = bconv_ptrs_kernel<W>;
    CERIUM_LAUNCH(kfn, dim3(kBconvBlocks, (unsigned)num_conversions), kBconvThreads, smem, s,
                  reinterpret_cast<W* const*>(outs), n_out, reinterpret_cast<const W* const*>(ins), n_in,
                  reinterpret_cast<const W* const*>(factors), reinterpret_cast<const W* const*>(out_moduli),
                  max_in, max_out, smem, ctx->d_status);
    CERIUM_LAUNCH_CHECK("bconv_ptrs");
    return CERIUM_OK;
  });
}

int cerium_sud(cerium_context* ctx, void* out, size_t out_stride, const void* minuend, size_t minuend_stride,
               void* in_coeff, size_t in_stride, const void* addend, size_t addend_stride,
               const uint32_t* prime_idx, int count, const uint32_t* divide_primes, int n_divide, void* stream) {
  if (!ctx) return fail(CERIUM_ERR_INVALID, "sud: null context");
  if (count < 0 || n_divide < 1) return fail(CERIUM_ERR_INVALID, "sud: bad count");
  if (count == 0) return CERIUM_OK;
  if (!prime_idx || !divide_primes) return fail(CERIUM_ERR_INVALID, "sud: null index array");
  const size_t wb = ctx->word_bytes();
  if (int rc = check_stack(out, out_stride, wb, "sud: out")) return rc;
  if (int rc = check_stack(minuend, minuend_stride, wb, "sud: minuend")) return rc;
  if (int rc = check_stack(in_coeff, in_stride, wb, "sud: in_coeff")) return rc;
  if (addend)
    if (int rc = check_stack(addend, addend_stride, wb, "sud: addend")) return rc;
  std::vector<uint32_t> div(divide_primes, divide_primes + n_divide);
  for (uint32_t d : div)
    if (d >= (uint32_t)ctx->n_primes) return fail(CERIUM_ERR_INVALID, "sud: divide prime index out of range");
  std::vector<uint64_t> factor(count);
  for (int i = 0; i < count; i++) {
    if (prime_idx[i] >= (uint32_t)ctx->n_primes) return fail(CERIUM_ERR_INVALID, "sud: prime index out of range");
    const uint64_t q = ctx->moduli[prime_idx[i]];
    // a prime that divides the product has no inverse: factor 0, as compute_sud_factors leaves it
    factor[i] = 1 % q;
    for (uint32_t d : div) factor[i] = host::mulmod(factor[i], d == prime_idx[i] ? 0 : ctx->inverse(d, prime_idx[i]), q);
  }
  DeviceGuard guard(ctx->device);
  SudCall c{};
  c.src = in_coeff;
  c.src_stride = in_stride;
  c.work = in_coeff;
  c.work_stride = in_stride;
  c.dst = out;
  c.dst_stride = out_stride;
  c.minuend = minuend;
  c.minuend_stride = minuend_stride;
  c.addend = addend;
  c.addend_stride = addend_stride;
  c.prime = prime_idx;
  c.factor = factor.data();
  c.count = count;
  return launch_sud(ctx, c, (cudaStream_t)stream);
}

int cerium_ewise(cerium_context* ctx, int op, void* out, size_t out_stride, const void* a, size_t a_stride,
                 const void* b, size_t b_stride, const void* c, size_t c_stride, const uint64_t* scalars,
                 const uint32_t* prime_idx, int count, void* stream) {
  if (!ctx) return fail(CERIUM_ERR_INVALID, "ewise: null context");
  if (op < CERIUM_EW_ADD || op > CERIUM_EW_REDUCE) return fail(CERIUM_ERR_INVALID, "ewise: unknown op");
  if (count < 0) return fail(CERIUM_ERR_INVALID, "ewise: negative count");
  if (count == 0) return CERIUM_OK;
  if (!prime_idx) return fail(CERIUM_ERR_INVALID, "ewise: null prime_idx");
  const size_t wb = ctx->word_bytes();
  const bool need_b = op == CERIUM_EW_ADD || op == CERIUM_EW_SUB || op == CERIUM_EW_MUL || op == CERIUM_EW_MAD ||
                      op == CERIUM_EW_PMU;
  const bool need_c = op == CERIUM_EW_MAD;
  const bool need_s = op == CERIUM_EW_PMU || op == CERIUM_EW_MUL_SCALAR;
  if (int rc = check_stack(out, out_stride, wb, "ewise: out")) return rc;
  if (int rc = check_stack(a, a_stride, wb, "ewise: a")) return rc;
  if (need_b)
    if (int rc = check_stack(b, b_stride, wb, "ewise: b")) return rc;
  if (need_c)
    if (int rc = check_stack(c, c_stride, wb, "ewise: c")) return rc;
  if (need_s && !scalars) return fail(CERIUM_ERR_INVALID, "ewise: null scalars");
  for (int i = 0; i < count; i++)
    if (prime_idx[i] >= (uint32_t)ctx->n_primes) return fail(CERIUM_ERR_INVALID, "ewise: prime index out of range");
  DeviceGuard guard(ctx->device);
  cudaStream_t s = (cudaStream_t)stream;
  return dispatch_word(ctx->word_bits, [&](auto tag) -> int {
    using W = decltype(tag);
    using V = Vec16<W>;
    const PrimeConst<W>* pcs = static_cast<const PrimeConst<W>*>(ctx->d_pcs);
    for (int first = 0; first < count; first += kEwMaxLimbs) {
      const int cnt = std::min(kEwMaxLimbs, count - first);
      EwArgs<W> g{};
      EwScalars<W> sc;
      g.out = {static_cast<W*>(out) + (size_t)first * out_stride, out_stride};
      g.a = {const_cast<W*>(static_cast<const W*>(a)) + (size_t)first * a_stride, a_stride};
      if (need_b) g.b = {const_cast<W*>(static_cast<const W*>(b)) + (size_t)first * b_stride, b_stride};
      if (need_c) g.c = {const_cast<W*>(static_cast<const W*>(c)) + (size_t)first * c_stride, c_stride};
      for (int k = 0; k < cnt; k++) {
        g.prime[k] = (uint8_t)prime_idx[first + k];
        if (need_s) {
          const uint64_t q = ctx->moduli[prime_idx[first + k]];
          const uint64_t sv = scalars[first + k] % q;
          sc.scalar[k] = (W)sv;
          sc.scalar_shoup[k] = (W)host::shoup(sv, q, ctx->word_bits);
        }
      }
      const dim3 grid(kN / (kEwThreads * V::kLanes), cnt);
      switch (op) {
        case CERIUM_EW_ADD: { auto kfn = ewise_kernel<W, kEwAdd>; CERIUM_LAUNCH(kfn, grid, kEwThreads, 0, s, g, EwNone{}, pcs); } break;
        case CERIUM_EW_SUB: { auto kfn = ewise_kernel<W, kEwSub>; CERIUM_LAUNCH(kfn, grid, kEwThreads, 0, s, g, EwNone{}, pcs); } break;
        case CERIUM_EW_NEG: { auto kfn = ewise_kernel<W, kEwNeg>; CERIUM_LAUNCH(kfn, grid, kEwThreads, 0, s, g, EwNone{}, pcs); } break;
        case CERIUM_EW_MUL: { auto kfn = ewise_kernel<W, kEwMul>; CERIUM_LAUNCH(kfn, grid, kEwThreads, 0, s, g, EwNone{}, pcs); } break;
        case CERIUM_EW_MAD: { auto kfn = ewise_kernel<W, kEwMad>; CERIUM_LAUNCH(kfn, grid, kEwThreads, 0, s, g, EwNone{}, pcs); } break;
        case CERIUM_EW_PMU: { auto kfn = ewise_kernel<W, kEwPmu>; CERIUM_LAUNCH(kfn, grid, kEwThreads, 0, s, g, sc, pcs); } break;
        case CERIUM_EW_REDUCE: { auto kfn = ewise_kernel<W, kEwReduce>; CERIUM_LAUNCH(kfn, grid, kEwThreads, 0, s, g, EwNone{}, pcs); } break;
        default: { auto kfn = ewise_kernel<W, kEwMulScalar>; CERIUM_LAUNCH(kfn, grid, kEwThreads, 0, s, g, sc, pcs); } break;
      }
    }
    CERIUM_LAUNCH_CHECK("ewise");
    return CERIUM_OK;
  });
}

int cerium_mul_plain_periodic(cerium_context* ctx, void* out, size_t out_stride, const void* a, size_t a_stride,
                              const void* pt, size_t pt_stride, int log2_repeat, const void* addend, size_t addend_stride,
                              const uint32_t* prime_idx, int count, void* stream) {
  if (!ctx) return fail(CERIUM_ERR_INVALID, "mul_plain_periodic: null context");
  if (count < 0) return fail(CERIUM_ERR_INVALID, "mul_plain_periodic: negative count");
  if (log2_repeat < 0 || log2_repeat > ctx->logn) return fail(CERIUM_ERR_INVALID, "mul_plain_periodic: repeat count out of range");
  if (count == 0) return CERIUM_OK;
  if (!prime_idx) return fail(CERIUM_ERR_INVALID, "mul_plain_periodic: null prime_idx");
  const size_t wb = ctx->word_bytes();
  if (int rc = check_stack(out, out_stride, wb, "mul_plain_periodic: out")) return rc;
  if (int rc = check_stack(a, a_stride, wb, "mul_plain_periodic: a")) return rc;
  if (!pt) return fail(CERIUM_ERR_INVALID, "mul_plain_periodic: null plaintext");
  if (pt_stride < ((size_t)kN >> log2_repeat)) return fail(CERIUM_ERR_INVALID, "mul_plain_periodic: plaintext stride is smaller than one period");
  if (addend)
    if (int rc = check_stack(addend, addend_stride, wb, "mul_plain_periodic: addend")) return rc;
  for (int i = 0; i < count; i++)
    if (prime_idx[i] >= (uint32_t)ctx->n_primes) return fail(CERIUM_ERR_INVALID, "mul_plain_periodic: prime index out of range");
  DeviceGuard guard(ctx->device);
  cudaStream_t s = (cudaStream_t)stream;
  return dispatch_word(ctx->word_bits, [&](auto tag) -> int {
    using W = decltype(tag);
    using V = Vec16<W>;
    const PrimeConst<W>* pcs = static_cast<const PrimeConst<W>*>(ctx->d_pcs);
    for (int first = 0; first < count; first += kEwMaxLimbs) {
      const int cnt = std::min(kEwMaxLimbs, count - first);
      EwArgs<W> g{};
      g.out = {static_cast<W*>(out) + (size_t)first * out_stride, out_stride};
      g.a = {const_cast<W*>(static_cast<const W*>(a)) + (size_t)first * a_stride, a_stride};
      g.b = {const_cast<W*>(static_cast<const W*>(pt)) + (size_t)first * pt_stride, pt_stride};
      if (addend) g.c = {const_cast<W*>(static_cast<const W*>(addend)) + (size_t)first * addend_stride, addend_stride};
      g.shift = log2_repeat;
      for (int k = 0; k < cnt; k++) g.prime[k] = (uint8_t)prime_idx[first + k];
      const dim3 grid(kN / (kEwThreads * V::kLanes), cnt);
      if (addend) { auto kfn = ewise_kernel<W, kEwMadPeriodic>; CERIUM_LAUNCH(kfn, grid, kEwThreads, 0, s, g, EwNone{}, pcs); }
      else { auto kfn = ewise_kernel<W, kEwMulPeriodic>; CERIUM_LAUNCH(kfn, grid, kEwThreads, 0, s, g, EwNone{}, pcs); }
    }
    CERIUM_LAUNCH_CHECK("mul_plain_periodic");
    return CERIUM_OK;
  });
}

int cerium_tensor(cerium_context* ctx, void* d0, void* d1, void* d2, const void* a0, const void* a1,
                  const void* b0, const void* b1, size_t stride, const uint32_t* prime_idx, int count,
                  void* stream) {
  if (!ctx) return fail(CERIUM_ERR_INVALID, "tensor: null context");
  if (count < 0) return fail(CERIUM_ERR_INVALID, "tensor: negative count");
  if (count == 0) return CERIUM_OK;
  if (!prime_idx) return fail(CERIUM_ERR_INVALID, "tensor: null prime_idx");
  const size_t wb = ctx->word_bytes();
  const void* ptrs[7] = {d0, d1, d2, a0, a1, b0, b1};
  for (const void* p : ptrs)
    if (int rc = check_stack(p, stride, wb, "tensor: operand")) return rc;
  for (int i = 0; i < count; i++)
    if (prime_idx[i] >= (uint32_t)ctx->n_primes) return fail(CERIUM_ERR_INVALID, "tensor: prime index out of range");
  DeviceGuard guard(ctx->device);
  return dispatch_word(ctx->word_bits, [&](auto tag) -> int {
    using W = decltype(tag);
    using V = Vec16<W>;
    for (int first = 0; first < count; first += kEwMaxLimbs) {
      const int cnt = std::min(kEwMaxLimbs, count - first);
      const size_t off = (size_t)first * stride;
      auto mk = [&](const void* p) { return Limbs<W>{const_cast<W*>(static_cast<const W*>(p)) + off, stride}; };
      TensorArgs<W> g{};
      g.a0 = mk(a0); g.a1 = mk(a1); g.b0 = mk(b0); g.b1 = mk(b1);
      g.d0 = mk(d0); g.d1 = mk(d1); g.d2 = mk(d2);
      for (int k = 0; k < cnt; k++) g.prime[k] = (uint8_t)prime_idx[first + k];
      { auto kfn = tensor_kernel<W>; CERIUM_LAUNCH(kfn, dim3(kN / (kEwThreads * V::kLanes), cnt), kEwThreads, 0, (cudaStream_t)stream, g, static_cast<const PrimeConst<W>*>(ctx->d_pcs)); }
    }
    CERIUM_LAUNCH_CHECK("tensor");
    return CERIUM_OK;
  });
}

uint32_t cerium_galois_elt_from_step(int step, int log_n) {
  if (log_n < 1 || log_n > 30) return 0;
  const uint64_t n = (uint64_t)1 << log_n, m = 2 * n;
  if (step == 0) return (uint32_t)(m - 1);
  const uint64_t a = step < 0 ? (uint64_t)(-(int64_t)step) : (uint64_t)step;
  if (a >= (n >> 1)) return 0;  // "step count too large" in the reference
  uint64_t s = step < 0 ? (n >> 1) - a : a;
  uint64_t e = 1, g = 5;
  for (; s; s >>= 1) {
    if (s & 1) e = (e * g) & (m - 1);
    g = (g * g) & (m - 1);
  }
  return (uint32_t)e;
}

int cerium_automorph(cerium_context* ctx, void* out, size_t out_stride, const void* in, size_t in_stride,
                     uint32_t galois_elt, int count, void* stream) {
  if (!ctx) return fail(CERIUM_ERR_INVALID, "automorph: null context");
  if (count < 0) return fail(CERIUM_ERR_INVALID, "automorph: negative count");
  if (!(galois_elt & 1) || galois_elt >= 2u * kN) return fail(CERIUM_ERR_INVALID, "automorph: Galois element is not valid");
  if (count == 0) return CERIUM_OK;
  if (count > 65535) return fail(CERIUM_ERR_INVALID, "automorph: more than 65535 limbs in one call");
  const size_t wb = ctx->word_bytes();
  if (int rc = check_stack(out, out_stride, wb, "automorph: out")) return rc;
  if (int rc = check_stack(in, in_stride, wb, "automorph: in")) return rc;
  if (out == in) return fail(CERIUM_ERR_INVALID, "automorph: result cannot alias the operand");
  DeviceGuard guard(ctx->device);
  return dispatch_word(ctx->word_bits, [&](auto tag) -> int {
    using W = decltype(tag);
    AutomorphArgs<W> g{};
    g.out = {static_cast<W*>(out), out_stride};
    g.in = {const_cast<W*>(static_cast<const W*>(in)), in_stride};
    g.split = count;
    g.elt = galois_elt;
    { auto kfn = automorph_kernel<W>; CERIUM_LAUNCH(kfn, dim3(kN / kEwThreads, count), kEwThreads, 0, (cudaStream_t)stream, g); }
    CERIUM_LAUNCH_CHECK("automorph");
    return CERIUM_OK;
  });
}

}  // extern "C"

namespace cerium {
// Automorphism of two polynomials of `count` limbs each (stride N) in one launch.
int launch_automorph_pair(cerium_context* ctx, void* out_a, const void* in_a, void* out_b, const void* in_b,
                          uint32_t galois_elt, int count, cudaStream_t stream) {
  return dispatch_word(ctx->word_bits, [&](auto tag) -> int {
    using W = decltype(tag);
    AutomorphArgs<W> g{};
    g.out = {static_cast<W*>(out_a), (size_t)kN};
    g.in = {const_cast<W*>(static_cast<const W*>(in_a)), (size_t)kN};
    g.out2 = {static_cast<W*>(out_b), (size_t)kN};
    g.in2 = {const_cast<W*>(static_cast<const W*>(in_b)), (size_t)kN};
    g.split = count;
    g.elt = galois_elt;
    { auto kfn = automorph_kernel<W>; CERIUM_LAUNCH(kfn, dim3(kN / kEwThreads, 2 * count), kEwThreads, 0, stream, g); }
    CERIUM_LAUNCH_CHECK("automorph");
    return CERIUM_OK;
  });
}
}  // namespace cerium

extern "C" {

int cerium_resolve2(cerium_context* ctx, void* lo, void* hi, const void* x0, const void* x1, size_t stride,
                    uint32_t prime0, uint32_t prime1, int count, void* stream) {
  if (!ctx) return fail(CERIUM_ERR_INVALID, "resolve2: null context");
  if (count < 0 || count > 65535) return fail(CERIUM_ERR_INVALID, "resolve2: bad count");
  if (count == 0) return CERIUM_OK;
  if (prime0 >= (uint32_t)ctx->n_primes || prime1 >= (uint32_t)ctx->n_primes || prime0 == prime1)
    return fail(CERIUM_ERR_INVALID, "resolve2: need two different prime indices of the context");
  const size_t wb = ctx->word_bytes();
  const void* ptrs[4] = {lo, hi, x0, x1};
  for (const void* p : ptrs)
    if (int rc = check_stack(p, stride, wb, "resolve2: operand")) return rc;
  const uint64_t m0 = ctx->moduli[prime0], m1 = ctx->moduli[prime1];
  const uint64_t inv = ctx->inverse(prime0, prime1);
  DeviceGuard guard(ctx->device);
  return dispatch_word(ctx->word_bits, [&](auto tag) -> int {
    using W = decltype(tag);
    using V = Vec16<W>;
    auto mk = [&](const void* p) { return Limbs<W>{const_cast<W*>(static_cast<const W*>(p)), stride}; };
    Rsv2Args<W> g{};
    g.x0 = mk(x0); g.x1 = mk(x1); g.lo = mk(lo); g.hi = mk(hi);
    g.m0 = (W)m0;
    g.inv = (W)inv;
    g.inv_shoup = (W)host::shoup(inv, m1, ctx->word_bits);
    g.prime1 = prime1;
    { auto kfn = rsv2_kernel<W>; CERIUM_LAUNCH(kfn, dim3(kN / (kEwThreads * V::kLanes), count), kEwThreads, 0, (cudaStream_t)stream, g, static_cast<const PrimeConst<W>*>(ctx->d_pcs)); }
    CERIUM_LAUNCH_CHECK("resolve2");
    return CERIUM_OK;
  });
}

int cerium_mod2(cerium_context* ctx, void* out, size_t out_stride, const void* lo, const void* hi,
                const uint32_t* prime_idx, int count, void* stream) {
  if (!ctx) return fail(CERIUM_ERR_INVALID, "mod2: null context");
  if (count < 0) return fail(CERIUM_ERR_INVALID, "mod2: negative count");
  if (count == 0) return CERIUM_OK;
  if (!prime_idx) return fail(CERIUM_ERR_INVALID, "mod2: null prime_idx");
  const size_t wb = ctx->word_bytes();
  if (int rc = check_stack(out, out_stride, wb, "mod2: out")) return rc;
  if (int rc = check_stack(lo, kN, wb, "mod2: lo")) return rc;
  if (int rc = check_stack(hi, kN, wb, "mod2: hi")) return rc;
  for (int i = 0; i < count; i++)
    if (prime_idx[i] >= (uint32_t)ctx->n_primes) return fail(CERIUM_ERR_INVALID, "mod2: prime index out of range");
  DeviceGuard guard(ctx->device);
  return dispatch_word(ctx->word_bits, [&](auto tag) -> int {
    using W = decltype(tag);
    using V = Vec16<W>;
    for (int first = 0; first < count; first += kEwMaxLimbs) {
      const int cnt = std::min(kEwMaxLimbs, count - first);
      Mod2Args<W> g{};
      g.lo = static_cast<const W*>(lo);
      g.hi = static_cast<const W*>(hi);
      g.out = {static_cast<W*>(out) + (size_t)first * out_stride, out_stride};
      for (int k = 0; k < cnt; k++) g.prime[k] = (uint8_t)prime_idx[first + k];
      { auto kfn = mod2_kernel<W>; CERIUM_LAUNCH(kfn, dim3(kN / (kEwThreads * V::kLanes), cnt), kEwThreads, 0, (cudaStream_t)stream, g, static_cast<const PrimeConst<W>*>(ctx->d_pcs)); }
    }
    CERIUM_LAUNCH_CHECK("mod2");
    return CERIUM_OK;
  });
}

int cerium_bconv_create(cerium_context* ctx, cerium_bconv** out, int mode, const uint32_t* in_primes, int n_in,
                        const uint32_t* out_primes, int n_out) {
  return create_bconv(ctx, out, mode, in_primes, n_in, out_primes, n_out, BconvOptions{});
}

int cerium_bconv_destroy(cerium_bconv* bc) {
  if (!bc) return CERIUM_OK;
  DeviceGuard guard(bc->ctx->device);
  cudaFree(bc->d_block);
  delete bc;
  return CERIUM_OK;
}

int cerium_bconv_apply(cerium_bconv* bc, void* out, size_t out_stride, const void* in, size_t in_stride,
                       void* stream) {
  if (!bc) return fail(CERIUM_ERR_INVALID, "bconv_apply: null converter");
  const size_t wb = bc->ctx->word_bytes();
  if (int rc = check_stack(out, out_stride, wb, "bconv_apply: out")) return rc;
  if (int rc = check_stack(in, in_stride, wb, "bconv_apply: in")) return rc;
  DeviceGuard guard(bc->ctx->device);
  BconvCall c{bc, out, out_stride, in, in_stride};
  return launch_bconv(bc->ctx, &c, 1, (cudaStream_t)stream);
}

int cerium_bconv_apply_batch(cerium_bconv* const* bcs, void* const* outs, const void* const* ins, int count,
                             size_t out_stride, size_t in_stride, void* stream) {
  if (count < 0) return fail(CERIUM_ERR_INVALID, "bconv_apply_batch: negative count");
  if (count == 0) return CERIUM_OK;
  if (!bcs || !outs || !ins) return fail(CERIUM_ERR_INVALID, "bconv_apply_batch: null array");
  std::vector<BconvCall> calls(count);
  for (int k = 0; k < count; k++) {
    if (!bcs[k]) return fail(CERIUM_ERR_INVALID, "bconv_apply_batch: null converter");
    if (bcs[k]->ctx != bcs[0]->ctx) return fail(CERIUM_ERR_INVALID, "bconv_apply_batch: converters of different contexts");
    const size_t wb = bcs[k]->ctx->word_bytes();
    if (int rc = check_stack(outs[k], out_stride, wb, "bconv_apply_batch: out")) return rc;
    if (int rc = check_stack(ins[k], in_stride, wb, "bconv_apply_batch: in")) return rc;
    calls[k] = BconvCall{bcs[k], outs[k], out_stride, ins[k], in_stride};
  }
  DeviceGuard guard(bcs[0]->ctx->device);
  return launch_bconv(bcs[0]->ctx, calls.data(), count, (cudaStream_t)stream);
}

}  // extern "C"
