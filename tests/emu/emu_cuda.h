// Host stand-ins for the CUDA built-ins and the few runtime calls the library uses, so that
// the kernel sources and the host glue compile with g++ and run on the CPU.  TEST
// INFRASTRUCTURE ONLY: it exists to check index arithmetic, barrier placement and host
// orchestration on a machine without a GPU.  The shipped library is never built with
// CERIUM_EMU and has no CPU path.
//
// Execution model: a launch runs its thread blocks one after another (spread over OpenMP
// threads); the threads of a block are ucontext fibers on one OS thread, scheduled round
// robin, and __syncthreads() yields to the next fiber.  Because every fiber runs to its next
// barrier before any fiber continues, barriers that all threads of a block reach (the only
// kind the kernels use) behave as on the device.  __syncwarp() holds only the 32 fibers of a warp
// together; warps otherwise run one after another as far as they can, so code that needs a
// block barrier where it only has a warp barrier computes wrong results here too.  __shared__ variables become
// static thread_local, i.e. one copy per OS thread = per running block.
#pragma once
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <functional>

struct uint2 { unsigned x, y; };
struct uint3 { unsigned x, y, z; };
struct alignas(16) uint4 { unsigned x, y, z, w; };
struct alignas(16) ulonglong2 { unsigned long long x, y; };
struct alignas(16) double2 { double x, y; };
static inline double2 make_double2(double a, double b) { return double2{a, b}; }
struct dim3 {
  unsigned x, y, z;
  dim3(unsigned x_ = 1, unsigned y_ = 1, unsigned z_ = 1) : x(x_), y(y_), z(z_) {}
};
static inline uint2 make_uint2(unsigned a, unsigned b) { return uint2{a, b}; }
static inline uint4 make_uint4(unsigned a, unsigned b, unsigned c, unsigned d) { return uint4{a, b, c, d}; }
static inline ulonglong2 make_ulonglong2(unsigned long long a, unsigned long long b) { return ulonglong2{a, b}; }

#define __global__
#define __device__
#define __host__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __restrict__
#define __shared__ static thread_local
#define __align__(n) __attribute__((aligned(n)))

namespace cerium_emu {
extern thread_local uint3 t_threadIdx, t_blockIdx;
extern thread_local dim3 t_blockDim, t_gridDim;
unsigned char* dyn_smem();
void sync_threads();
void sync_warp();
void launch(dim3 grid, dim3 block, size_t smem_bytes, const std::function<void()>& body);
long launches();  // number of launches so far (tests use it to see that kernels ran)
void set_smem_limit(const void* kernel, int bytes);
void default_stream(bool pending);  // something was queued on the default stream / the host has waited for it
}  // namespace cerium_emu

#define threadIdx (::cerium_emu::t_threadIdx)
#define blockIdx (::cerium_emu::t_blockIdx)
#define blockDim (::cerium_emu::t_blockDim)
#define gridDim (::cerium_emu::t_gridDim)

static inline void __syncthreads() { ::cerium_emu::sync_threads(); }
static inline void __syncwarp() { ::cerium_emu::sync_warp(); }
static inline unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)(((uint64_t)a * b) >> 32); }
static inline unsigned long long __umul64hi(unsigned long long a, unsigned long long b) {
  return (unsigned long long)(((unsigned __int128)a * b) >> 64);
}
static inline double __dmul_rn(double a, double b) { return a * b; }
static inline double __dadd_rn(double a, double b) { return a + b; }
static inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
static inline long long __double2ll_rn(double x) { return std::llrint(x); }  // default rounding mode: to nearest even
static inline double __ll2double_rn(long long x) { return (double)x; }
static inline double __ull2double_rn(unsigned long long x) { return (double)x; }
static inline double __longlong_as_double(long long x) { double d; std::memcpy(&d, &x, 8); return d; }
static inline long long __double_as_longlong(double d) { long long x; std::memcpy(&x, &d, 8); return x; }
static inline unsigned __brev(unsigned x) {
  unsigned r = 0;
  for (int i = 0; i < 32; i++) { r = (r << 1) | (x & 1); x >>= 1; }
  return r;
}
static inline int __clzll(long long x) { return x == 0 ? 64 : __builtin_clzll((unsigned long long)x); }
static inline unsigned __funnelshift_r(unsigned lo, unsigned hi, unsigned s) { return (unsigned)(((uint64_t)hi << 32 | lo) >> (s & 31)); }
static inline int __clz(int x) { return x == 0 ? 32 : __builtin_clz((unsigned)x); }
template <typename T>
static inline T __ldg(const T* p) { return *p; }
template <typename T>
static inline T __ldcs(const T* p) { return *p; }
static inline unsigned atomicOr(unsigned* p, unsigned v) { return __atomic_fetch_or(p, v, __ATOMIC_RELAXED); }

// ---- runtime API subset ----
typedef int cudaError_t;
typedef void* cudaStream_t;
typedef void* cudaEvent_t;
enum { cudaSuccess = 0, cudaErrorMemoryAllocation = 2 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2, cudaMemcpyDeviceToDevice = 3 };
enum cudaFuncAttribute { cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
static inline cudaError_t cudaMalloc(void** p, size_t n) {
  *p = std::aligned_alloc(256, (n + 255) / 256 * 256);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
template <typename T>
static inline cudaError_t cudaMalloc(T** p, size_t n) { return cudaMalloc(reinterpret_cast<void**>(p), n); }
static inline cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
static inline cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind kind) {
  std::memcpy(d, s, n);
  ::cerium_emu::default_stream(kind == cudaMemcpyHostToDevice);
  return cudaSuccess;
}
static inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memmove(d, s, n); return cudaSuccess; }
static inline cudaError_t cudaMemset(void* d, int v, size_t n) {
  std::memset(d, v, n);
  ::cerium_emu::default_stream(true);
  return cudaSuccess;
}
static inline cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
static inline cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  if (s == nullptr) ::cerium_emu::default_stream(false);
  return cudaSuccess;
}
static inline cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
enum cudaDeviceAttr { cudaDevAttrMultiProcessorCount = 16 };
static inline cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 2; return cudaSuccess; }
static inline cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
static inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
static inline cudaError_t cudaGetLastError() { return cudaSuccess; }
static inline const char* cudaGetErrorString(cudaError_t) { return "emulated"; }
enum { cudaStreamNonBlocking = 1, cudaEventDisableTiming = 2 };
static inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)1; return cudaSuccess; }
static inline cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
static inline cudaError_t cudaDeviceGetStreamPriorityRange(int* lo, int* hi) { *lo = 0; *hi = 0; return cudaSuccess; }
static inline cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) { *s = (cudaStream_t)1; return cudaSuccess; }
static inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)1; return cudaSuccess; }
static inline cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
static inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
static inline cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
template <typename T>
static inline cudaError_t cudaGetSymbolAddress(void** p, T& symbol) { *p = (void*)&symbol; return cudaSuccess; }
template <typename F>
static inline cudaError_t cudaFuncSetAttribute(F kernel, cudaFuncAttribute, int bytes) {
  ::cerium_emu::set_smem_limit(reinterpret_cast<const void*>(kernel), bytes);
  return cudaSuccess;
}
