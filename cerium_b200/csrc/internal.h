// Internal host-side structures behind the opaque handles of include/cerium_b200.h.
#pragma once
#if defined(CERIUM_EMU)
#include "emu_cuda.h"  // test-only host stand-ins; the shipped library is never built this way
#else
#include <cuda_runtime.h>
#endif

#include <atomic>
#include <cstdint>
#include <cstdio>
#include <map>
#include <memory>
#include <string>
#include <utility>
#include <vector>

#include "../../include/cerium_b200.h"
#include "bconv_kernels.cuh"
#include "bconv_mma.cuh"
#include "bsgs_kernels.cuh"
#include "ewise_kernels.cuh"
#include "host_math.h"
#include "ntt_kernels.cuh"
#include "ntt_radix8.cuh"
#include "raised_inner.cuh"

namespace cerium {

constexpr int kMaxDevices = 64;  // per-device host-side caches are indexed by the CUDA device ordinal

void set_error(const std::string& msg);
int fail(int code, const std::string& msg);

#define CERIUM_CUDA(call)                                                              \
  do {                                                                                 \
    cudaError_t e__ = (call);                                                          \
    if (e__ != cudaSuccess)                                                            \
      return ::cerium::fail(CERIUM_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e__)); \
  } while (0)

#define CERIUM_LAUNCH_CHECK(what)                                                      \
  do {                                                                                 \
    cudaError_t e__ = cudaGetLastError();                                              \
    if (e__ != cudaSuccess)                                                            \
      return ::cerium::fail(CERIUM_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e__)); \
  } while (0)

// Kernels for which something has been set on a device.  Threads that come first together set it once each.
class KernelTable {
  static constexpr size_t kSlots = 1024;  // open addressing; a full table only means that it is set again
  std::atomic<uintptr_t> seen_[kSlots] = {};

 public:
  template <typename Set>
  cudaError_t once(const void* kfn, Set&& set) {
    int device = 0;
    if (cudaError_t e = cudaGetDevice(&device); e != cudaSuccess) return e;
    const uintptr_t key = reinterpret_cast<uintptr_t>(kfn) * kMaxDevices + (uintptr_t)device;
    bool done = false;
    for (size_t k = 0, h = key / kMaxDevices / 16 % kSlots; k < kSlots; k++, h = (h + 1) % kSlots) {
      uintptr_t at = seen_[h].load(std::memory_order_acquire);
      if (at == key) return cudaSuccess;
      if (at != 0) continue;
      if (!done)
        if (cudaError_t e = set(); e != cudaSuccess) return e;
      done = true;
      if (seen_[h].compare_exchange_strong(at, key, std::memory_order_acq_rel) || at == key) return cudaSuccess;
    }
    return done ? cudaSuccess : set();
  }
};

// Lets a kernel be launched with up to `bytes` of dynamic shared memory.  The limit belongs to the kernel and not to a
// launch, so `bytes` is the most that any of its launches needs: one that lowered it would fail another thread's.
template <typename Kernel>
inline cudaError_t allow_smem(Kernel kfn, size_t bytes) {
  static KernelTable seen;
  return seen.once(reinterpret_cast<const void*>(kfn), [&] {
    return cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  });
}

constexpr size_t kSplitSmem = 164 * 1024;  // shared memory of an SM, as every kernel asks for it (kCarveoutPercent)
// Kernel launch through a function pointer (template-ids with commas stay out of the macro).
#if defined(CERIUM_EMU)
#define CERIUM_LAUNCH(kfn, grid, block, smem, stream, ...) \
  ::cerium_emu::launch((grid), (block), (smem), [=]() { kfn(__VA_ARGS__); })
#else
// All kernels ask for one split of the SM's memory, 164 KB shared and 64 KB L1 (71 % of the 228 KB rounds up to it): what
// four CTAs of a transform's row pass need.  Left to the driver every kernel gets the split that suits it alone, an SM
// has to drain before it changes from one to the next, and the overlap of dependent launches is lost at every such
// boundary (a rotation of 12 limbs, 11 launches: 132 us; 127 with one split of 132 KB, then 119.5; 115.7 with 164 KB,
// where the next kernel's CTAs find more room beside those that finish).  With 228 KB the transforms lose the L1 that
// holds their twiddles (384 limbs: 212 us against 188).  The attribute is set at a kernel's first launch on a device.
constexpr int kCarveoutPercent = 71;
inline void prefer_carveout(const void* kfn) {
  static KernelTable seen;
  seen.once(kfn, [&] {
    cudaFuncSetAttribute(kfn, cudaFuncAttributePreferredSharedMemoryCarveout, kCarveoutPercent);  // a hint
    return cudaSuccess;
  });
}
// Every kernel is launched with programmatic stream serialisation (see grid_dependency_wait in
// modarith.cuh): its CTAs may be placed while the previous kernel of the stream drains.
template <typename... KArgs, typename... Args>
inline void launch_dependent(void (*kfn)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                             Args&&... args) {
  prefer_carveout(reinterpret_cast<const void*>(kfn));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kfn, std::forward<Args>(args)...);  // errors surface in CERIUM_LAUNCH_CHECK
}
#define CERIUM_LAUNCH(kfn, grid, block, smem, stream, ...) \
  ::cerium::launch_dependent(kfn, dim3(grid), dim3(block), (size_t)(smem), (stream), __VA_ARGS__)
#endif

// Runs fn(W{}) with W = uint32_t or uint64_t according to the context's word size.
template <typename F>
inline int dispatch_word(int word_bits, F&& fn) {
  if (word_bits == 32) return fn(uint32_t{});
  return fn(uint64_t{});
}

// The end of every call that makes a handle: what it copied from pageable memory, or set, is in place.  cudaMemcpy may
// return when the bytes have left the caller's buffer, with the copy to the device still queued on the default
// stream, and a stream created without blocking does not wait for that one.
inline cudaError_t uploads_done() { return cudaStreamSynchronize(nullptr); }

// RAII switch to the context's device for the duration of a call.
struct DeviceGuard {
  int prev = -1;
  bool ok = true;
  explicit DeviceGuard(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) ok = false;
    if (ok && prev != dev && cudaSetDevice(dev) != cudaSuccess) ok = false;
    if (prev == dev) prev = -1;
  }
  ~DeviceGuard() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

}  // namespace cerium

struct cerium_context {
  int device = 0;
  int logn = 0;
  int word_bits = 0;
  int n_primes = 0;
  std::vector<uint64_t> moduli;
  std::vector<uint64_t> psi;
  std::vector<uint64_t> ninv, w1ninv;  // N^-1, psi^-(N/2) N^-1
  void* d_tw_fwd = nullptr;  // Pair[n_primes][N], bit-reversed powers of psi
  void* d_tw_inv = nullptr;  // Pair[n_primes][N], bit-reversed powers of psi^-1
  void* d_twr_fwd = nullptr; // Pair[n_primes][256][15][16], lane-interleaved level-3 twiddles (row pass)
  void* d_twr_inv = nullptr; // same for the inverse transform
  void* d_pcs = nullptr;     // PrimeConst<W>[n_primes]
  uint32_t* d_status = nullptr;  // device status word: kernels that skip a malformed work item set a bit here
  // 64-bit primes below 2^50 transform on the FP64 pipe unless the environment variable
  // CERIUM_B200_NTT_ARITH is "int" when the context is created (for comparisons)
  bool allow_fp = true;
  int sm_count = 1;  // SMs of the device (launch shapes are sized in multiples of it)
  std::vector<uint8_t> fp_ok;  // primes whose transforms run on doubles (host copy)
  size_t word_bytes() const { return (size_t)word_bits / 8; }
  // q_a^-1 mod q_b, found once per pair (the extended Euclid of a rescale's factors was most of its host time): a table
  // of n_primes^2 words, 0 = not known yet; concurrent calls at worst find the same value twice
  std::unique_ptr<std::atomic<uint64_t>[]> inverses;
  uint64_t inverse(uint32_t a, uint32_t b) const {
    std::atomic<uint64_t>& e = inverses[(size_t)a * n_primes + b];
    uint64_t v = e.load(std::memory_order_relaxed);
    if (v == 0) {
      v = cerium::host::invmod(moduli[a] % moduli[b], moduli[b]);
      e.store(v, std::memory_order_relaxed);
    }
    return v;
  }
};

struct cerium_bconv {
  cerium_context* ctx = nullptr;
  int mode = 0;
  int I = 0, O = 0;
  std::vector<uint32_t> in_primes;
  // one device allocation holding every table below
  void* d_block = nullptr;
  int steps = 0;                // steps of 32 input bytes of the products
  bool all_wide = true;         // every output prime is in the quotient class of the lazy kernel
  void* d_table = nullptr;      // fragments of the tensor cores (bconv_mma.cuh)
  void* d_outc = nullptr;       // BconvMmaOut<W>[O]
  void* d_inv = nullptr;        // W[I] (exact mode, unless the caller pre-scales)
  void* d_inv_shoup = nullptr;  // W[I]
  uint32_t* d_in_prime = nullptr;
  uint32_t* d_in_pos = nullptr;   // or null
  // rounding (round_half): what the caller adds to the inputs, modulo q_i, before they are converted
  std::vector<uint64_t> in_add_host;
  bool lazy_out = false;
  std::vector<uint64_t> inv_host;  // [Qhat_i^-1]_{q_i}
};

// Communicator of the limb collectives: the ranks of one job, one GPU each.  The transport is NCCL
// (loaded at run time) or a set of caller-provided functions.
struct cerium_comm {
  int rank = 0, world = 1, device = 0;
  void* nccl = nullptr;  // ncclComm_t when the transport is NCCL
  cerium_comm_callbacks cb = {};
  bool has_cb = false;
  std::map<int, cerium_comm*> subgroups;  // communicators of `size` consecutive ranks holding this rank (owned)
};

namespace cerium {

// Collectives on raw device buffers, enqueued on `stream`.  `send` of the all-gather may be the
// rank's own block of `recv` (in place).  Sums are plain word additions (no modular reduction).
int comm_allgather(cerium_comm* comm, void* recv, const void* send, size_t bytes_per_rank, cudaStream_t stream);
int comm_reducescatter_sum(cerium_comm* comm, void* recv, const void* send, size_t words_per_rank, int word_bits,
                           cudaStream_t stream);
int comm_allreduce_sum(cerium_comm* comm, void* recv, const void* send, size_t words, int word_bits, cudaStream_t stream);
int comm_broadcast(cerium_comm* comm, void* buf, size_t bytes, int root, cudaStream_t stream);
// The communicator of the `size` consecutive ranks [rank / size * size, ...) that hold this rank (`comm` itself
// when size is its world); created on first use - a collective call: every rank of `comm` makes it, in the
// same order - and owned by `comm`.
int comm_subgroup(cerium_comm* comm, int size, cerium_comm** out);

// Options of create_bconv beyond the public entry point.
struct BconvOptions {
  bool prescaled = false;            // exact mode, inputs already multiplied by [Qhat_i^-1]
  bool round_half = false;           // the inputs come with floor(prod_in/2) added (in_add_host): subtract it from outputs
  std::vector<uint32_t> out_pos;     // output limb slots (empty = 0..O-1)
  std::vector<uint32_t> in_pos;      // input limb slots (empty = 0..I-1)
  bool lazy_out = false;             // outputs feed the forward NTT directly: skip the final corrections
  int inputs_together = 0;           // most inputs of the conversions that may share a launch with this one (0: those of this one)
};

int create_bconv(cerium_context* ctx, cerium_bconv** out, int mode, const uint32_t* in_primes, int n_in,
                 const uint32_t* out_primes, int n_out, const BconvOptions& opt);

// One entry of a batched conversion launch.
struct BconvCall {
  cerium_bconv* bc;
  void* out;
  size_t out_stride;
  const void* in;
  size_t in_stride;
};
int launch_bconv(cerium_context* ctx, const BconvCall* calls, int count, cudaStream_t stream);

// Batched transforms with explicit limb slots (pos[b]) and prime indices.
struct NttCall {
  const void* in;
  void* out;
  size_t in_stride, out_stride;
  const uint32_t* pos;    // count entries, or null for 0..count-1
  const uint32_t* prime;  // count entries
  int count;
  // forward transform: entry b reads limb src_pos[b] of `in`, residues of another modulus, and
  // reduces them to its own prime on the way in (null: reads limb pos[b], already reduced).
  // inverse transform: entry b reads limb src_pos[b] of `in` (same modulus) instead of limb pos[b]
  const uint32_t* src_pos = nullptr;
  // with src_pos: prime index of the modulus the words of entry b are residues of (null: unknown)
  const uint32_t* src_prime = nullptr;
  // forward transform only: the input words are what a base conversion with lazy_out left, without a rounding term or with one
  // (kFpRaisedIn, kFpLoweredIn), instead of canonical
  bool raised_in = false, lowered_in = false;
  // inverse transform only, not 0: the input limbs are read through the Galois automorphism of this element
  uint32_t in_galois = 0;
  // inverse transform only: the input is the product with the limbs of this stack, which lie as those of `in` do
  const void* factor = nullptr;
  // forward transform only: the column pass alone; raised_inner_kernel does the rows
  bool cols_only = false;
};
// lazy_out: leave the results below 4q instead of canonical (internal buffers read by the inner product only)
int launch_ntt_forward(cerium_context* ctx, const NttCall& c, cudaStream_t stream, bool lazy_out = false);
// last: device array of four words per batch entry (inverse_last_words: the results times a scale), or null.
// add: device array of one word per batch entry, added to the results modulo q, or null.
int launch_ntt_inverse(cerium_context* ctx, const NttCall& c, cudaStream_t stream, const void* last = nullptr,
                       const void* add = nullptr);
// The four words by which the last layer of an inverse transform of prime `k` scales its results by `scale` / N.
void inverse_last_words(const cerium_context* ctx, int k, uint64_t scale, uint64_t (&out)[4]);

// SuD over `count` limbs (count <= kSudMaxBatch per launch; chunked internally).
struct SudCall {
  const void* src;       // coefficient-form source; src_stride == 0 broadcasts one limb
  size_t src_stride;
  void* work;            // column-pass output / row-pass input (may equal src when src_stride != 0)
  size_t work_stride;
  void* dst;
  size_t dst_stride;
  const void* minuend;
  size_t minuend_stride;
  const void* addend;    // or null
  size_t addend_stride;
  const uint32_t* prime;  // count prime indices
  const uint64_t* factor; // count canonical residues (host)
  int count;
  // optional second polynomial in the same launch: entries [split, count) write dst2 and read
  // minuend2 / addend2 at index (b - split); src / work stay one stack of `count` limbs
  int split = 0;          // 0 = one polynomial
  void* dst2 = nullptr;
  const void* minuend2 = nullptr;
  const void* addend2 = nullptr;
  bool lazy_src = false;  // the source words are what a base conversion with lazy_out left (kFpLoweredIn) instead of canonical
  bool cols_done = false;  // `work` holds the column pass's results already
  // source re-reduction (only when reduce_src): residues of modulus src_q, optional rounding
  bool reduce_src = false;
  uint64_t src_q = 0;
  uint64_t pre_add = 0;
  const uint64_t* post_sub = nullptr;  // count residues (host) or null
  // only with reduce_src: entry b reads limb src_pos[b] of src (null: limb b, or the one limb
  // when src_stride == 0)
  const uint32_t* src_pos = nullptr;
  // not 0: addend / addend2 are read through the Galois automorphism of this element
  uint32_t addend_galois = 0;
  // not 0: word i of every result limb is stored at pi(i) (index map of this element); dst / dst2 must
  // then not overlap minuend, addend or work
  uint32_t store_galois = 0;
};
int launch_sud(cerium_context* ctx, const SudCall& c, cudaStream_t stream);
int launch_automorph_pair(cerium_context* ctx, void* out_a, const void* in_a, void* out_b, const void* in_b,
                          uint32_t galois_elt, int count, cudaStream_t stream);

}  // namespace cerium
