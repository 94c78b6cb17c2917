// Entry points of the encoder / decoder side: residues of integer-valued doubles, and the exact CRT
// composition of coefficient-form limbs back to doubles (kernels in client_kernels.cuh).
#include <cstring>

#include "client_kernels.cuh"
#include "internal.h"

using namespace cerium;

struct cerium_compose {
  cerium_context* ctx = nullptr;
  int limbs = 0, words = 0;
  char* d_block = nullptr;   // qinv | inv, Shoup companions, moduli | Qhat_i words, Q words
  size_t o_inv = 0, o_table = 0;
};

namespace {

// little-endian 32-bit words of the product of the moduli, leaving out one of them (skip < 0: none)
std::vector<uint32_t> product_words(const std::vector<uint64_t>& q, int skip, size_t words) {
  std::vector<uint32_t> p(words, 0);
  p[0] = 1;
  for (int k = 0; k < (int)q.size(); k++) {
    if (k == skip) continue;
    uint64_t carry = 0;
    for (size_t w = 0; w < words; w++) {
      carry += (uint64_t)p[w] * q[k];
      p[w] = (uint32_t)carry;
      carry >>= 32;
    }
  }
  return p;
}

using u128 = unsigned __int128;
uint64_t pcg64_output(u128 s) {
  const uint64_t hi = (uint64_t)(s >> 64), x = hi ^ (uint64_t)s;
  const unsigned r = (unsigned)(hi >> 58);
  return x >> r | x << (-r & 63u);
}
// The next n outputs of the generator.  Four states a step apart advance four steps at a time: one state at a time waits for its
// 128-bit product (17 limbs of 2^16 words: numpy 4.6 ms, here 1.8 on the same core).
void pcg64_fill(u128& state, u128 inc, uint64_t* out, size_t n) {
  const u128 m = (u128)0x2360ED051FC65DA4ull << 64 | 0x4385DF649FCCF645ull, m2 = m * m, m4 = m2 * m2;
  const u128 c4 = inc * (1 + m + m2 + m2 * m);
  u128 s[4];
  s[0] = state * m + inc;
  for (int k = 1; k < 4; k++) s[k] = s[k - 1] * m + inc;
  size_t i = 0;
  for (; i + 4 < n; i += 4)
    for (int k = 0; k < 4; k++) {
      out[i + k] = pcg64_output(s[k]);
      s[k] = s[k] * m4 + c4;
    }
  for (int k = 0; i < n; i++, k++) {
    out[i] = pcg64_output(s[k]);
    state = s[k];
  }
}

}  // namespace

extern "C" {

int cerium_pcg64_uniform(uint64_t state[4], uint32_t buffered[2], uint32_t below, uint32_t* out, size_t count) {
  if (!state || !buffered || (!out && count != 0)) return fail(CERIUM_ERR_INVALID, "pcg64_uniform: null argument");
  if (below == 0) return fail(CERIUM_ERR_INVALID, "pcg64_uniform: no word is below 0");
  if (below == 1) {  // nothing to draw
    for (size_t i = 0; i < count; i++) out[i] = 0;
    return CERIUM_OK;
  }
  u128 s = (u128)state[0] << 64 | state[1];
  const u128 inc = (u128)state[2] << 64 | state[3];
  const uint32_t reject = (0u - below) % below;  // fractions below this belong to values that come once more often
  size_t i = 0;
  constexpr size_t kBlock = 128;
  uint64_t block[kBlock];
  uint32_t draws[2 * kBlock];
  while (i < count) {
    // as many outputs as are used whatever is rejected
    const bool waiting = buffered[0] != 0;
    const size_t want = (count - i + 1) / 2, n = waiting ? 0 : want < kBlock ? want : kBlock;
    pcg64_fill(s, inc, block, n);
    draws[0] = buffered[1];
    for (size_t k = 0; k < n; k++) {
      draws[2 * k] = (uint32_t)block[k];
      draws[2 * k + 1] = (uint32_t)(block[k] >> 32);
    }
    const size_t have = waiting ? 1 : 2 * n, use = have < count - i ? have : count - i;
    uint32_t rejected = 0;
    for (size_t k = 0; k < use; k++) {
      const uint64_t m = (uint64_t)draws[k] * below;
      out[i + k] = (uint32_t)(m >> 32);
      rejected |= (uint32_t)m < reject ? 1u : 0u;
    }
    size_t used = use;
    if (rejected == 0) {
      i += use;
    } else {  // again, one by one
      for (used = 0; used < have && i < count; used++) {
        const uint64_t m = (uint64_t)draws[used] * below;
        if ((uint32_t)m >= reject) out[i++] = (uint32_t)(m >> 32);
      }
    }
    buffered[0] = used < have ? 1 : 0;  // at most the last half is left
    buffered[1] = draws[have - 1];
  }
  state[0] = (uint64_t)(s >> 64);
  state[1] = (uint64_t)s;
  return CERIUM_OK;
}

int cerium_residues(cerium_context* ctx, void* out, size_t out_stride, const double* values, const int32_t* small,
                    const uint32_t* prime_idx, int count, void* stream) {
  if (!ctx || !out || !values || !prime_idx) return fail(CERIUM_ERR_INVALID, "residues: null argument");
  if (count < 0) return fail(CERIUM_ERR_INVALID, "residues: negative count");
  if (out_stride < (size_t)kN) return fail(CERIUM_ERR_INVALID, "residues: stride is smaller than N");
  for (int i = 0; i < count; i++)
    if (prime_idx[i] >= (uint32_t)ctx->n_primes) return fail(CERIUM_ERR_INVALID, "residues: prime index out of range");
  DeviceGuard guard(ctx->device);
  return dispatch_word(ctx->word_bits, [&](auto tag) -> int {
    using W = decltype(tag);
    for (int first = 0; first < count; first += kClientMaxLimbs) {
      const int cnt = count - first < kClientMaxLimbs ? count - first : kClientMaxLimbs;
      ResidueArgs<W> g{};
      g.values = values;
      g.small = small;
      g.out = static_cast<W*>(out) + (size_t)first * out_stride;
      g.out_stride = out_stride;
      for (int k = 0; k < cnt; k++) g.prime[k] = (uint8_t)prime_idx[first + k];
      auto kfn = residues_kernel<W>;
      CERIUM_LAUNCH(kfn, dim3(kN / kClientThreads, cnt), kClientThreads, 0, (cudaStream_t)stream, g, static_cast<const PrimeConst<W>*>(ctx->d_pcs));
    }
    CERIUM_LAUNCH_CHECK("residues");
    return CERIUM_OK;
  });
}

int cerium_compose_create(cerium_context* ctx, cerium_compose** out, const uint32_t* prime_idx, int count) {
  if (!ctx || !out || !prime_idx) return fail(CERIUM_ERR_INVALID, "compose_create: null argument");
  if (ctx->word_bits != 32) return fail(CERIUM_ERR_UNSUPPORTED, "compose_create: 32-bit contexts");
  if (count < 1 || count > kComposeMaxLimbs) return fail(CERIUM_ERR_UNSUPPORTED, "compose_create: 1..255 limbs");
  std::vector<uint64_t> q(count);
  for (int i = 0; i < count; i++) {
    if (prime_idx[i] >= (uint32_t)ctx->n_primes) return fail(CERIUM_ERR_INVALID, "compose_create: prime index out of range");
    q[i] = ctx->moduli[prime_idx[i]];
    for (int j = 0; j < i; j++)
      if (q[j] == q[i]) return fail(CERIUM_ERR_INVALID, "compose_create: a prime appears twice");
  }
  std::vector<uint32_t> big_q = product_words(q, -1, count + 1);  // moduli are below 2^30
  size_t bits = big_q.size() * 32;
  while (!(big_q[(bits - 1) / 32] >> ((bits - 1) % 32) & 1u)) bits--;
  const size_t words = (bits + 1 + 31) / 32;  // one bit more: the centred value has a sign
  std::vector<uint32_t> table, inv(3 * (size_t)count);
  std::vector<double> qinv(count);
  for (int i = 0; i < count; i++) {
    std::vector<uint32_t> t = product_words(q, i, words);
    table.insert(table.end(), t.begin(), t.end());
    uint64_t hat = 1 % q[i];
    for (int j = 0; j < count; j++)
      if (j != i) hat = host::mulmod(hat, q[j] % q[i], q[i]);
    const uint64_t h = host::invmod(hat, q[i]);
    inv[i] = (uint32_t)h;
    inv[count + i] = (uint32_t)host::shoup(h, q[i], 32);
    inv[2 * count + i] = (uint32_t)q[i];
    qinv[i] = 1.0 / (double)q[i];
  }
  big_q.resize(words);
  table.insert(table.end(), big_q.begin(), big_q.end());
  DeviceGuard guard(ctx->device);
  if (!guard.ok) return fail(CERIUM_ERR_CUDA, "compose_create: cannot select device");
  auto* c = new cerium_compose();
  c->ctx = ctx;
  c->limbs = count;
  c->words = (int)words;
  c->o_inv = qinv.size() * sizeof(double);
  c->o_table = c->o_inv + inv.size() * 4;
  std::vector<char> bytes(c->o_table + table.size() * 4);
  std::memcpy(bytes.data(), qinv.data(), qinv.size() * sizeof(double));
  std::memcpy(bytes.data() + c->o_inv, inv.data(), inv.size() * 4);
  std::memcpy(bytes.data() + c->o_table, table.data(), table.size() * 4);
  if (cudaMalloc(&c->d_block, bytes.size()) != cudaSuccess ||
      cudaMemcpy(c->d_block, bytes.data(), bytes.size(), cudaMemcpyHostToDevice) != cudaSuccess || uploads_done() != cudaSuccess) {
    cerium_compose_destroy(c);
    return fail(CERIUM_ERR_CUDA, "compose_create: table upload failed");
  }
  *out = c;
  return CERIUM_OK;
}

int cerium_compose_destroy(cerium_compose* c) {
  if (!c) return CERIUM_OK;
  DeviceGuard guard(c->ctx->device);
  cudaFree(c->d_block);
  delete c;
  return CERIUM_OK;
}

int cerium_compose_apply(cerium_compose* c, double* out, const void* in, size_t in_stride, void* stream) {
  if (!c || !out || !in) return fail(CERIUM_ERR_INVALID, "compose_apply: null argument");
  if (in_stride < (size_t)kN) return fail(CERIUM_ERR_INVALID, "compose_apply: stride is smaller than N");
  DeviceGuard guard(c->ctx->device);
  ComposeArgs g{};
  g.in = static_cast<const uint32_t*>(in);
  g.in_stride = in_stride;
  g.out = out;
  g.qinv = reinterpret_cast<const double*>(c->d_block);
  g.inv = reinterpret_cast<const uint32_t*>(c->d_block + c->o_inv);
  g.table = reinterpret_cast<const uint32_t*>(c->d_block + c->o_table);
  g.limbs = c->limbs;
  g.words = c->words;
  const size_t smem = (size_t)(c->limbs + c->words) * kComposeThreads * 4;
  if (smem > 48 * 1024) CERIUM_CUDA(cudaFuncSetAttribute(compose_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024));
  { auto kfn = compose_kernel; CERIUM_LAUNCH(kfn, dim3(kN / kComposeThreads), kComposeThreads, smem, (cudaStream_t)stream, g); }
  CERIUM_LAUNCH_CHECK("compose");
  return CERIUM_OK;
}

}  // extern "C"
