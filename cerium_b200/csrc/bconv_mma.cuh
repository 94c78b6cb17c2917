// Fast base conversion on the tensor cores.
//
// out_j[c] = ( sum_i y_i[c] * F[j][i] ) mod p_j is a matrix product whose entries are too wide for a tensor core,
// so it is taken byte by byte: with y_i = sum_k y_ik 2^8k and G[j][i][k] = F[j][i] 2^8k mod p_j (a table),
//   out_j = sum_m 2^8m ( sum_ik byte_m(G[j][i][k]) * y_ik )   mod p_j,
// i.e. an unsigned 8-bit product [8 O x 8 I] x [8 I x coefficients] into 32-bit sums (4 in place of 8 for 32-bit
// words), and per output ONE recombination of its 8 (4) byte planes and one reduction of a value that exceeds p_j by
// 2^14 or so: the quotient is a 32-bit high product, the remainder two multiply-adds.  The words of the inputs
// are their own bytes, so the right-hand operand is read as it lies in memory.
//
// A multiply-add on 64-bit words costs this chip's integer pipe four wide products of four cycles each (5 inputs: 73
// instructions an output before, 13 inputs of 32-bit words ~35); here an output costs ~13 instructions whatever
// the number of inputs, beside 14 / 128 of an m16n8k32 product per step of 32 input bytes.
//
// Mapping: a CTA owns kMmaStage coefficients of one conversion and stages their input words in shared memory (cp.async).  Each of
// its warps owns a group of outputs and walks over tiles of 8 coefficients.  The 16 rows of a product are two byte planes of 8
// outputs (64-bit words) or one plane of 16 (32-bit words; two planes where at most 8 are left), so the accumulators of all
// planes give a thread every byte of its own (output, coefficient) pairs and nothing is exchanged.  The table's fragments
// stay in the warp's registers (kSteps <= 2 for 64-bit words, <= 4 for 32-bit ones, i.e. up to 8 and 32 inputs;
// beyond that they are read again for every tile), and so do the constants of the thread's outputs.
// Bound by the latencies of product and recombination (tensor pipe 43 % of its cycles, multiply pipe 39 %, issue slots 40 % for 7
// conversions 5 -> 35 of 64-bit words), so many small CTAs that are in different phases do better than the walk over five to
// ten stages through three buffers that was here before, whose warps met at a barrier for each stage and whose grid ended in a part of a
// round: rotation of 35 limbs 275.1 -> 267.6 us, of 51 limbs of 32-bit words 173.3 -> 165.4, multiplication of 30 limbs 242.6 ->
// 232.9, 12 limbs 99.0 / 98.4 (with the next kernel let in late, see grid_dependency_launch).  64 coefficients: 35 limbs 272.0,
// 256: 268.8; 64 registers instead of 80: 267.5.
// Where the inputs end in the first 16 bytes of a step the product is taken for those alone (35 limbs 278.7 -> 275.1).
// Measured before: warps that read the words from global memory themselves waited for them half of the time, and 16 outputs to
// a warp took 152 registers (56 us against 48).
// The kernel was first built on tcgen05 (M = 128 coefficients, accumulators in TMEM): with K = 64 the product is over
// in tens of cycles, and the round through barrier, commit, wait and TMEM load of every 8 outputs left the SM at 43 %
// of its issue slots: 48 us for 7 conversions 5 -> 35 against 22 us of memory traffic.
//
// Replaces convert<I,O> (cerium/compiler/backend/kernels/fhe_bconv.cuh:98-151).
#pragma once
#include <type_traits>

#include "bconv_kernels.cuh"
#include "ntt_kernels.cuh"

namespace cerium {

constexpr int kMmaMaxWarps = 8;                   // groups of one CTA
constexpr int kMmaStage = 128;                    // coefficients of a CTA
template <typename W>
constexpr int kMmaRows = sizeof(W) == 8 ? 8 : 16;  // outputs of a group
constexpr int kMmaTile = 8;                       // coefficients of a tile
// Most steps whose fragments a warp keeps in registers.
template <typename W>
constexpr int kMmaRegSteps = sizeof(W) == 8 ? 2 : 4;
constexpr int kMmaMaxBatch = 24;                  // conversions per launch (descriptors travel as parameters)
constexpr int kMmaMaxInputs = 64;                 // of a conversion
constexpr int kMmaPairInputs = 32;                // 64-bit inputs whose plane pairs c + 2^8 c' stay below 2^32:
                                                  // 8 I 255^2 257 < 2^32 (32-bit words: 4 I, so all 64 do)

// What a thread needs for one output.
//
// The quotient c of the recombined sum x <= 255 b I (q - 1) (b = bytes of a word) comes from the bits of x above
// 2^base, t, times floor(2^(base + 32 + shift) / q):
//   64-bit words, wide    q >= 2^48, base = 48, shift = 0: x - c q is below 2.3 q, and taken modulo 2^64 (x itself may pass it)
//   64-bit words, narrow  2^40 <= q < 2^48, base = 32 (x fits 64 bits up to kMmaPairInputs inputs; beyond them base = 34,
//                         from the plane sums): below 1.1 q
//   64-bit words, tiny    q < 2^40: 64-bit high product with floor(2^64 / q); below 4 q
//   32-bit words          base = 16, shift = 0: q > 2^17, so below 1.3 q
template <typename W>
struct alignas(16) BconvMmaOut {
  W nq;              // -q modulo the word
  W mu;              // the factor above
  W add;             // q - rounding term, or 0
  uint32_t pos;      // limb slot of the output
  uint16_t shift;
  uint16_t cls;
};
enum : int { kMmaWide = 0, kMmaNarrow = 1, kMmaTiny = 2 };

// The constants of an output of modulus q (its slot aside); sub = rounding term that leaves the result.
template <typename W>
inline BconvMmaOut<W> bconv_mma_constants(uint64_t q, uint64_t sub) {
  BconvMmaOut<W> o{};
  o.nq = (W)0 - (W)q;
  o.add = sub != 0 ? (W)(q - sub) : (W)0;
  o.cls = sizeof(W) == 4 || q >= ((uint64_t)1 << 48) ? kMmaWide : q >= ((uint64_t)1 << 40) ? kMmaNarrow : kMmaTiny;
  if (o.cls == kMmaTiny) {
    o.mu = (W)(((unsigned __int128)1 << 64) / q);
  } else if (o.cls == kMmaNarrow) {
    uint64_t mu = 0;
    while ((mu = (uint64_t)(((unsigned __int128)1 << (64 + o.shift)) / q)) < ((uint64_t)1 << 31)) o.shift++;
    o.mu = (W)mu;
  } else {
    o.mu = (W)(((unsigned __int128)1 << (sizeof(W) == 8 ? 80 : 48)) / q);
  }
  return o;
}

template <typename W>
struct BconvMmaDesc {
  const W* in;
  W* out;
  size_t in_stride, out_stride;
  const W* inv;              // [I] or null: inputs are multiplied by it first (exact mode, unless the caller has)
  const W* inv_shoup;
  const uint32_t* in_prime;
  const uint32_t* in_pos;    // limb slots of the inputs, or null
  const uint4* table;        // fragments [group][plane or pair of planes][step][lane]
  const BconvMmaOut<W>* outc;
  int I, O;
  int steps;                 // steps of 32 input bytes
};

template <typename W>
struct BconvMmaBatch {
  BconvMmaDesc<W> d[kMmaMaxBatch];
};

template <typename W>
__host__ __device__ inline int bconv_mma_groups(int outs) { return (outs + kMmaRows<W> - 1) / kMmaRows<W>; }
// fragments of a group: one per plane, or per pair of planes when it has at most 8 outputs
template <typename W>
__host__ __device__ inline int bconv_mma_frags(int outs) { return outs <= 8 ? (int)sizeof(W) / 2 : (int)sizeof(W); }
// first uint4 entry of a group (all before it are full)
template <typename W>
__host__ __device__ inline size_t bconv_mma_entry(int group, int steps) {
  return (size_t)group * bconv_mma_frags<W>(kMmaRows<W>) * steps * 32;
}
template <typename W>
__host__ __device__ inline size_t bconv_mma_table_entries(int outs, int steps) {
  const int full = bconv_mma_groups<W>(outs) - 1;
  return bconv_mma_entry<W>(full, steps) + (size_t)bconv_mma_frags<W>(outs - full * kMmaRows<W>) * steps * 32;
}

// How a launch finishes its outputs.
//   kMmaLazy     every q of the batch wide (64-bit words) and every consumer content with values below 4q: no
//                case distinctions; kMmaLazyAdd: the same with rounding terms
//   kMmaGeneral  any q, canonical results
//   kMmaBig      general with more than kMmaPairInputs inputs: plane pairs kept in 64 bits
enum : int { kMmaLazy = 0, kMmaLazyAdd = 1, kMmaGeneral = 2, kMmaBig = 3 };

template <int kFinish>
__device__ __forceinline__ uint64_t bconv_mma_finish(const uint32_t (&c)[8], const BconvMmaOut<uint64_t>& o) {
  using Sum = std::conditional_t<kFinish == kMmaBig, uint64_t, uint32_t>;
  const Sum a = c[0] + ((Sum)c[1] << 8), b = c[2] + ((Sum)c[3] << 8), cc = c[4] + ((Sum)c[5] << 8), d = c[6] + ((Sum)c[7] << 8);
  // x modulo 2^64 = low word of `low`, u + 2^16 d above it; pairs of up to kMmaPairInputs inputs leave u the room of the carry
  const uint64_t low = (uint64_t)a + ((uint64_t)b << 16);
  const Sum u = cc + (Sum)(low >> 32);
  const uint64_t x = (uint64_t)(uint32_t)low | (uint64_t)(uint32_t)(u + (d << 16)) << 32;
  if (kFinish <= kMmaLazyAdd) {
    const uint32_t t = (uint32_t)(d + (u >> 16));
    const uint64_t r = x + (uint64_t)__umulhi(t, (uint32_t)o.mu) * o.nq;
    return kFinish == kMmaLazy ? r : r + o.add;  // below 2.3 q, 3.3 q
  }
  const uint64_t q = 0 - o.nq;
  uint64_t r;
  if (o.cls == kMmaTiny) {
    r = x + mulhi_approx64(x, o.mu) * o.nq;
  } else {
    // narrow, more than kMmaPairInputs inputs: x may pass 2^64 (below 2^65), so the bits above 2^32 come from the sums,
    // two fewer of them
    const uint32_t t = o.cls == kMmaWide     ? (uint32_t)(d + (u >> 16))
                       : kFinish == kMmaBig ? (uint32_t)((u + (d << 16)) >> 2)
                                            : (uint32_t)(x >> 32);
    const int shift = kFinish == kMmaBig && o.cls == kMmaNarrow ? o.shift - 2 : o.shift;  // narrow: at least 7
    r = x + (uint64_t)(__umulhi(t, (uint32_t)o.mu) >> shift) * o.nq;
  }
  r = csub<uint64_t>(csub<uint64_t>(r, q + q), q);
  return csub<uint64_t>(r + o.add, q);
}
template <int kFinish>
__device__ __forceinline__ uint32_t bconv_mma_finish(const uint32_t (&c)[4], const BconvMmaOut<uint32_t>& o) {
  const uint32_t a = c[0] + (c[1] << 8), b = c[2] + (c[3] << 8);
  const uint32_t r = a + (b << 16) + __umulhi(b + (a >> 16), o.mu) * o.nq;
  if (kFinish <= kMmaLazyAdd) return kFinish == kMmaLazy ? r : r + o.add;  // below 1.3 q, 2.3 q
  const uint32_t q = 0u - o.nq;
  return csub<uint32_t>(csub<uint32_t>(r, q) + o.add, q);
}

#if !defined(CERIUM_EMU)
__device__ __forceinline__ void mma_u8(uint32_t (&c)[4], const uint4& a, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
// The first 16 of 32 input bytes alone, with the same fragments.
__device__ __forceinline__ void mma_u8_half(uint32_t (&c)[4], const uint4& a, uint32_t b0) {
  asm("mma.sync.aligned.m16n8k16.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a.x), "r"(a.y), "r"(b0));
}
__device__ __forceinline__ void mma_u8_half_first(uint32_t (&c)[4], const uint4& a, uint32_t b0) {
  asm("mma.sync.aligned.m16n8k16.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
      : "r"(a.x), "r"(a.y), "r"(b0), "r"(0));
}
__device__ __forceinline__ void mma_u8_first(uint32_t (&c)[4], const uint4& a, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1), "r"(0));
}
#endif

// Bytes between the staged limbs: a product's lanes read 8 coefficients of 2 limbs (64-bit words, both
// halves) or 4 limbs (32-bit words), which the padding spreads over all 32 banks.
template <typename W>
constexpr int kMmaPitch = kMmaStage * (int)sizeof(W) + (sizeof(W) == 8 ? 64 : 32);
template <typename W>
__host__ __device__ inline size_t bconv_mma_smem_bytes(int inputs) {
  return (size_t)inputs * kMmaPitch<W>;
}

// Byte offset of the 32-bit piece that holds input bytes 4 piece .. 4 piece + 3 of coefficient 0.  A
// piece past the last input is read from the last one: its table entries are zero.
template <typename W>
__device__ __forceinline__ int bconv_mma_piece(int piece, int inputs) {
  constexpr int kPerWord = sizeof(W) / 4;
  const int i = piece / kPerWord < inputs ? piece / kPerWord : inputs - 1;
  return i * kMmaPitch<W> + piece % kPerWord * 4;
}

// Stages kMmaStage coefficients from `first` on of every input limb.
template <typename W, bool kPrepare>
__device__ __forceinline__ void bconv_mma_stage(const BconvMmaDesc<W>& d, const PrimeConst<W>* __restrict__ pcs,
                                                unsigned char* buf, int first) {
  constexpr int kWords = 16 / (int)sizeof(W), kVecs = kMmaStage / kWords;
  using Vec = typename RowVec<W>::Vec;
  for (int k = threadIdx.x; k < d.I * kVecs; k += blockDim.x) {
    const int i = k / kVecs, v = k % kVecs;
    const W* src = d.in + (size_t)(d.in_pos != nullptr ? d.in_pos[i] : (uint32_t)i) * d.in_stride + first + v * kWords;
    unsigned char* dst = buf + i * kMmaPitch<W> + v * 16;
    if (kPrepare && d.inv != nullptr) {
      const W q = pcs[d.in_prime[i]].q, f = d.inv[i], fs = d.inv_shoup[i];
      W w[kWords];
      vec_unpack(*reinterpret_cast<const Vec*>(src), w);
#pragma unroll
      for (int e = 0; e < kWords; e++) w[e] = csub<W>(mul_shoup_lazy<W>(w[e], f, fs, q), q);
      *reinterpret_cast<Vec*>(dst) = vec_pack(w);
    } else {
#if defined(CERIUM_EMU)
      *reinterpret_cast<Vec*>(dst) = *reinterpret_cast<const Vec*>(src);
#else
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
#endif
    }
  }
}

#if defined(CERIUM_EMU)
// Sum of one byte plane of one output and coefficient, from the fragments as the tensor core would read them.
template <typename W>
inline uint32_t bconv_mma_emulate(const unsigned char* buf, const uint4* frag, int steps, int inputs, int row, int coeff) {
  uint32_t sum = 0;
  for (int s = 0; s < steps; s++)
    for (int piece = 0; piece < 8; piece++) {
      const uint4& f = frag[s * 32 + (row % 8) * 4 + piece % 4];
      const uint32_t a = piece < 4 ? (row < 8 ? f.x : f.y) : (row < 8 ? f.z : f.w);
      const uint32_t b = *reinterpret_cast<const uint32_t*>(buf + bconv_mma_piece<W>(s * 8 + piece, inputs) + coeff * (int)sizeof(W));
      for (int e = 0; e < 32; e += 8) sum += (a >> e & 0xff) * (b >> e & 0xff);
    }
  return sum;
}
#endif

// Warps that an SM holds: of 128 registers a thread or of 80.
template <typename W, int kSteps, bool kPrepare>
constexpr int kMmaWarpsPerSm = (sizeof(W) == 4 && kSteps == 4) || kPrepare ? 16 : 24;

// The CTA's coefficients from `first` on; this warp's group starts at output j0 (none: it only helps to stage).  kPair: the group
// has at most 8 outputs, its fragments hold two planes.  kSteps = 0: any number of steps, fragments read for every tile.  kHalf: no
// input has more than 16 bytes in the last step.
template <typename W, int kSteps, int kFinish, bool kPrepare, bool kHalf, bool kPair>
__device__ __forceinline__ void bconv_mma_group(const BconvMmaDesc<W>& d, const uint4* frag, int j0, int first, unsigned char* buf,
                                                const PrimeConst<W>* __restrict__ pcs, bool late_next) {
  constexpr int kPlanes = sizeof(W);
  constexpr int kFrags = kPair ? kPlanes / 2 : kPlanes;
  constexpr int kRows = kPair ? 1 : 2;             // outputs of a thread
  constexpr int kRegSteps = kSteps > 0 ? kSteps : 1;
  using Two = std::conditional_t<sizeof(W) == 8, ulonglong2, uint2>;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int steps = kSteps > 0 ? kSteps : d.steps;
  const bool busy = j0 < d.O;
  BconvMmaOut<W> o[kRows];
  W* dst[kRows];
  bool live[kRows];
#pragma unroll
  for (int r = 0; r < kRows; r++) {
    const int j = j0 + g + 8 * r;
    live[r] = j < d.O;
    o[r] = d.outc[live[r] ? j : 0];
    dst[r] = d.out + (size_t)o[r].pos * d.out_stride + first + 2 * t;
  }
  uint4 a[kSteps > 0 ? kFrags : 1][kRegSteps];
  if (kSteps > 0 && busy) {
#pragma unroll
    for (int p = 0; p < kFrags; p++)
#pragma unroll
      for (int s = 0; s < kRegSteps; s++) a[kSteps > 0 ? p : 0][s] = __ldg(frag + (p * kSteps + s) * 32 + lane);
  }
  int piece[kRegSteps][2];
#pragma unroll
  for (int s = 0; s < kRegSteps; s++)
#pragma unroll
    for (int h = 0; h < 2; h++) piece[s][h] = bconv_mma_piece<W>(s * 8 + h * 4 + t, d.I) + g * (int)sizeof(W);
  grid_dependency_wait();  // the tables above never change; the input limbs below come from the previous kernel
  if (!late_next) grid_dependency_launch();
  bconv_mma_stage<W, kPrepare>(d, pcs, buf, first);
#if !defined(CERIUM_EMU)
  asm volatile("cp.async.wait_all;" ::: "memory");
#endif
  __syncthreads();
  if (late_next) grid_dependency_launch();
  if (!busy) return;
#if defined(CERIUM_EMU)
  for (int base = 0; base < kMmaStage; base += kMmaTile)
    for (int r = 0; r < kRows; r++)
      for (int e = 0; e < 2; e++) {
        uint32_t c[kPlanes];
        for (int m = 0; m < kPlanes; m++)
          c[m] = bconv_mma_emulate<W>(buf, frag + (size_t)(kPair ? m / 2 : m) * steps * 32, steps, d.I,
                                      kPair ? g + 8 * (m & 1) : g + 8 * r, base + 2 * t + e);
        if (live[r]) dst[r][base + e] = bconv_mma_finish<kFinish>(c, o[r]);
      }
#else
#pragma unroll 2
  for (int base = 0; base < kMmaStage; base += kMmaTile) {
    const unsigned char* tile = buf + base * (int)sizeof(W);
    uint32_t c[kFrags][4];
    if (kSteps > 0) {
#pragma unroll
      for (int s = 0; s < kRegSteps; s++) {
        const uint32_t b0 = *reinterpret_cast<const uint32_t*>(tile + piece[s][0]);
        if (kHalf && s == kRegSteps - 1) {
#pragma unroll
          for (int p = 0; p < kFrags; p++) {
            if (s == 0) mma_u8_half_first(c[p], a[kSteps > 0 ? p : 0][s], b0);
            else mma_u8_half(c[p], a[kSteps > 0 ? p : 0][s], b0);
          }
          continue;
        }
        const uint32_t b1 = *reinterpret_cast<const uint32_t*>(tile + piece[s][1]);
#pragma unroll
        for (int p = 0; p < kFrags; p++) {
          if (s == 0) mma_u8_first(c[p], a[kSteps > 0 ? p : 0][s], b0, b1);
          else mma_u8(c[p], a[kSteps > 0 ? p : 0][s], b0, b1);
        }
      }
    } else {
#pragma unroll
      for (int p = 0; p < kFrags; p++) c[p][0] = c[p][1] = c[p][2] = c[p][3] = 0;
      for (int s = 0; s < steps; s++) {
        const uint32_t b0 = *reinterpret_cast<const uint32_t*>(tile + bconv_mma_piece<W>(s * 8 + t, d.I) + g * (int)sizeof(W));
        const uint32_t b1 = *reinterpret_cast<const uint32_t*>(tile + bconv_mma_piece<W>(s * 8 + 4 + t, d.I) + g * (int)sizeof(W));
#pragma unroll
        for (int p = 0; p < kFrags; p++) mma_u8(c[p], __ldg(frag + ((size_t)p * steps + s) * 32 + lane), b0, b1);
      }
    }
#pragma unroll
    for (int r = 0; r < kRows; r++) {
      W v[2];
#pragma unroll
      for (int e = 0; e < 2; e++) {
        uint32_t bytes[kPlanes];
#pragma unroll
        for (int m = 0; m < kPlanes; m++) bytes[m] = kPair ? c[m / 2][2 * (m & 1) + e] : c[kPair ? 0 : m][2 * r + e];
        v[e] = bconv_mma_finish<kFinish>(bytes, o[r]);
      }
      if (live[r]) *reinterpret_cast<Two*>(dst[r] + base) = Two{v[0], v[1]};
    }
  }
#endif
}

// grid = (N / kMmaStage, conversions, ceil(groups / warps)), block = 32 * warps, dynamic smem = bconv_mma_smem_bytes of the largest
// number of inputs.  late_next: see grid_dependency_launch.
template <typename W, int kSteps, int kFinish, bool kPrepare, bool kHalf = false, int kWarpsPerSm = kMmaWarpsPerSm<W, kSteps, kPrepare>>
__global__ void __launch_bounds__(32 * kMmaMaxWarps, kWarpsPerSm / kMmaMaxWarps)
    bconv_mma_kernel(const bool late_next, const BconvMmaBatch<W> batch, const PrimeConst<W>* __restrict__ pcs) {
  CERIUM_DYN_SMEM(smem);
  const BconvMmaDesc<W>& d = batch.d[blockIdx.y];
  const int group = blockIdx.z * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int j0 = group * kMmaRows<W>, first = blockIdx.x * kMmaStage;
  if ((int)(blockIdx.z * (blockDim.x / 32)) * kMmaRows<W> >= d.O) return;
  const uint4* frag = d.table + bconv_mma_entry<W>(group, d.steps);
  if (sizeof(W) == 8 || d.O - j0 <= 8) bconv_mma_group<W, kSteps, kFinish, kPrepare, kHalf, true>(d, frag, j0, first, smem, pcs, late_next);
  else bconv_mma_group<W, kSteps, kFinish, kPrepare, kHalf, sizeof(W) == 8>(d, frag, j0, first, smem, pcs, late_next);
}

}  // namespace cerium
