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

}  // namespace

extern "C" {

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
