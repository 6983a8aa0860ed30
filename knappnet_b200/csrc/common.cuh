// Shared device and host helpers of the knappnet B200 library.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <map>
#include <mutex>
#include <stdexcept>
#include <string>
#include <tuple>
#include <type_traits>

namespace knb {

// ---------------------------------------------------------------- errors
// Every failure below the C ABI is a C++ exception carrying the message the
// ABI writes into the caller's err buffer.
struct Error : std::runtime_error {
  explicit Error(const std::string& m) : std::runtime_error(m) {}
};

inline void cuda_check(cudaError_t e, const char* what) {
  if (e != cudaSuccess)
    throw Error(std::string("CUDA error in ") + what + ": " + cudaGetErrorString(e));
}
#define KNB_CUDA(x) ::knb::cuda_check((x), #x)
#define KNB_LAUNCH(what) ::knb::cuda_check(cudaGetLastError(), what)

constexpr int WARP = 32;

// ---------------------------------------------------------------- L2 cache policy
// Streamed arrays (column indices, arc values) are read once per sweep and
// should not push the gathered iterate out of the 126 MB L2; the iterate
// should stay. createpolicy builds the 64-bit L2 cache-policy operands.
__device__ __forceinline__ uint64_t policy_evict_first() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t policy_evict_last() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// Loads with an L2 policy (L2::cache_hint). ld_stream is for arrays that are
// laid out once and read-only while a kernel lives (ld.global.nc, not volatile:
// the compiler may move them). ld_keep and ld_keep_na gather the iterate, which
// the kernel before may still be writing when a chained kernel starts: ordinary
// loads, which no volatile asm, chain_wait's among them, is moved across. Sweeps
// take the same time either way (FP64 Katz on 2^24 arcs 7.8 to 7.9 ms a call,
// R-MAT with 2^28 arcs 23.8; a pointer made to depend on the wait instead costs
// its registers, Katz 8.1).
__device__ __forceinline__ uint32_t ld_stream(const uint32_t* p, uint64_t pol) {
  uint32_t v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.u32 %0, [%1], %2;"
               : "=r"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ float ld_stream(const float* p, uint64_t pol) {
  float v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.f32 %0, [%1], %2;"
               : "=f"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ double ld_stream(const double* p, uint64_t pol) {
  double v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.f64 %0, [%1], %2;"
               : "=d"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ float ld_keep(const float* p, uint64_t pol) {
  float v;
  asm volatile("ld.global.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ double ld_keep(const double* p, uint64_t pol) {
  double v;
  asm volatile("ld.global.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol));
  return v;
}

// 16-byte streamed loads (four u32 / f32, or two f64); the address must be
// 16-byte aligned.
__device__ __forceinline__ void ld_stream4(const uint32_t* p, uint64_t pol, uint32_t (&o)[4]) {
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
      : "=r"(o[0]), "=r"(o[1]), "=r"(o[2]), "=r"(o[3]) : "l"(p), "l"(pol));
}
__device__ __forceinline__ void ld_stream4(const float* p, uint64_t pol, float (&o)[4]) {
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
      : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]) : "l"(p), "l"(pol));
}
__device__ __forceinline__ void ld_stream4(const double* p, uint64_t pol, double (&o)[4]) {
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;"
      : "=d"(o[0]), "=d"(o[1]) : "l"(p), "l"(pol));
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;"
      : "=d"(o[2]), "=d"(o[3]) : "l"(p + 2), "l"(pol));
}

// Gathers that skip L1 allocation (the L2 policy still applies).
__device__ __forceinline__ float ld_keep_na(const float* p, uint64_t pol) {
  float v;
  asm volatile("ld.global.L1::no_allocate.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ double ld_keep_na(const double* p, uint64_t pol) {
  double v;
  asm volatile("ld.global.L1::no_allocate.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol));
  return v;
}

// ---------------------------------------------------------------- reductions
template <class T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Sums of K <= 4 per-lane values over a warp by a reduce-scatter butterfly:
// the first two exchanges also halve the number of values a lane carries,
// so the K sums cost 2 + 1 + 3 shuffles instead of 5 K. Returns, in every
// lane, the warp sum of value lane / 8 (lanes 8 K and up return a sum of
// zeros). The association is fixed, so results are identical run to run.
template <int K>
__device__ __forceinline__ double warp_sum_scatter(const double* v, int lane) {
  static_assert(K >= 1 && K <= 4, "at most 4 values");
  constexpr unsigned F = 0xffffffffu;
  const double v0 = v[0], v1 = K > 1 ? v[1] : 0.0, v2 = K > 2 ? v[2] : 0.0,
               v3 = K > 3 ? v[3] : 0.0;
  const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0;
  // lanes 0-15 keep values 0 and 1, lanes 16-31 values 2 and 3
  const double a0 = __shfl_xor_sync(F, h16 ? v0 : v2, 16);
  const double a1 = __shfl_xor_sync(F, h16 ? v1 : v3, 16);
  const double k0 = (h16 ? v2 : v0) + a0;
  const double k1 = (h16 ? v3 : v1) + a1;
  // then lanes with bit 3 clear keep the even value of the pair, set the odd
  const double b = __shfl_xor_sync(F, h8 ? k0 : k1, 8);
  double m = (h8 ? k1 : k0) + b;
  m += __shfl_xor_sync(F, m, 4);
  m += __shfl_xor_sync(F, m, 2);
  m += __shfl_xor_sync(F, m, 1);
  return m;
}

// Epilogues whose per-tile scalars are all plain sums declare SUMS = true.
template <class E, class = void>
struct EpiSums {
  static constexpr bool value = false;
};
template <class E>
struct EpiSums<E, std::void_t<decltype(E::SUMS)>> {
  static constexpr bool value = E::SUMS;
};

template <class T>
__device__ __forceinline__ T warp_max(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide sum in a fixed order (warp butterflies, then warp 0 over the
// warp totals), so the result is the same on every run. `scratch` holds at
// least blockDim.x / 32 values. The total is returned to every thread.
template <class T>
__device__ __forceinline__ T block_sum(T v, T* scratch) {
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[w] = v;
  __syncthreads();
  T t = lane < nw ? scratch[lane] : T(0);
  t = warp_sum(t);
  return t;
}
template <class T>
__device__ __forceinline__ T block_max(T v, T* scratch) {
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) scratch[w] = v;
  __syncthreads();
  T t = lane < nw ? scratch[lane] : T(-1e308);
  t = warp_max(t);
  return t;
}

// ---------------------------------------------------------------- launch helpers
// Sets a kernel attribute on the current device unless this process already
// set it to the same value there: cudaFuncSetAttribute acts on the current
// device only, and graph handles may live on any device, so the record is
// kept per (kernel, device, attribute), under a lock shared by all threads.
inline void set_func_attr(const void* fn, cudaFuncAttribute attr, int value) {
  static std::mutex mu;
  static std::map<std::tuple<const void*, int, int>, int> applied;
  int dev = 0;
  cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
  std::lock_guard<std::mutex> lock(mu);
  const auto key = std::make_tuple(fn, dev, (int)attr);
  auto it = applied.find(key);
  if (it != applied.end() && it->second == value) return;
  cuda_check(cudaFuncSetAttribute(fn, attr, value), "cudaFuncSetAttribute");
  applied[key] = value;
}

// Chains of short kernels: a kernel launched with launch_chained may be set up
// while the one before it on the stream still runs, and waits in chain_wait
// for that one's end before it touches memory; every kernel launched this way
// calls chain_wait first. It hides most of the 3 to 4 us that a kernel boundary
// costs between sweeps of a few microseconds. Launched the ordinary way,
// chain_wait returns at once. What the kernel before writes (iterates, partials,
// the state) is not read-only while a chained kernel lives: it takes no
// `const __restrict__` pointer to it, which would let the compiler read it
// through the non-coherent path or before the wait.
__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... K, class... A>
inline void launch_chained(void (*fn)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                           A&&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cuda_check(cudaLaunchKernelEx(&cfg, fn, static_cast<K>(args)...), "launch_chained");
}

inline unsigned grid_for(uint64_t work, unsigned block, unsigned cap = 148u * 32u) {
  uint64_t g = (work + block - 1) / block;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return (unsigned)g;
}

// Device memory comes from a pool of the library, one per device, that keeps
// up to POOL_KEEP bytes of what was freed for the next allocation and gives the
// rest back to the driver (a call that allocates its buffers spent most of its
// time in cudaMalloc and cudaFree, which also wait for the whole device: 16 of
// 47 ms of building a 4.2M-edge graph, 7 of 18 ms of strong components).
// device_pool_trim gives everything that is free back. Blocks of more than
// POOL_BLOCK bytes come from cudaMalloc: beyond what the pool keeps, mapping
// and unmapping through it costs more (building an R-MAT 24 graph: 375 ms with
// cudaMalloc, 545 ms with every block from the pool).
//
// Allocations and frees are ordered on the calling thread's stream
// (thread_stream), where all work on the memory runs; a block freed on one
// thread's stream reaches another thread's only once that stream's work on it
// is done. Memory that work on other streams uses (PlainMemory in scope) comes
// from cudaMalloc and goes back through cudaFree.
constexpr size_t POOL_KEEP = size_t(512) << 20;
constexpr size_t POOL_BLOCK = size_t(64) << 20;
struct DeviceBlock {
  void* p = nullptr;
  int device = 0;
  bool pooled = false;
};
DeviceBlock device_alloc(size_t bytes);      // throws Error when there is no memory
void device_free(const DeviceBlock& b) noexcept;
void device_pool_trim();                     // the current device's pool

struct PlainMemory {
  PlainMemory();
  ~PlainMemory();
  PlainMemory(const PlainMemory&) = delete;
};

// Page-locked host memory for a call's small copies (a copy from or to pageable
// memory costs about 10 us and waits). The lower half is for copies to the
// device, the upper for copies back, and whoever holds it waits for its copies
// before it lets go. Blocks are shared by all threads: there are as many as calls
// have held at once, of which STAGING_KEEP stay for the next ones until
// host_staging_trim.
constexpr size_t STAGING_HALF = size_t(512) << 10;
constexpr size_t STAGING_KEEP = 4;
struct HostStaging {
  unsigned char* p = nullptr;  // null where none could be had
  HostStaging();
  ~HostStaging();
  HostStaging(const HostStaging&) = delete;
};
void host_staging_trim();

// Device memory owned by RAII.
template <class T>
struct DevBuf {
  T* p = nullptr;
  size_t n = 0;
  DeviceBlock block;
  DevBuf() = default;
  explicit DevBuf(size_t count) { alloc(count); }
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  DevBuf(DevBuf&& o) noexcept { take(o); }
  DevBuf& operator=(DevBuf&& o) noexcept {
    if (this != &o) {
      release();
      take(o);
    }
    return *this;
  }
  ~DevBuf() { release(); }
  void alloc(size_t count) {
    release();
    if (count) {
      block = device_alloc(count * sizeof(T));
      p = static_cast<T*>(block.p);
    }
    n = count;
  }
  void release() {
    if (p) device_free(block);
    p = nullptr;
    n = 0;
    block = DeviceBlock{};
  }
  T* get() const { return p; }
  size_t bytes() const { return n * sizeof(T); }

 private:
  void take(DevBuf& o) {
    p = o.p;
    n = o.n;
    block = o.block;
    o.p = nullptr;
    o.n = 0;
    o.block = DeviceBlock{};
  }
};

}  // namespace knb
