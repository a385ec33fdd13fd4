// Shared host/device helpers of the flb200 kernel library (sm_100a only).
#pragma once

#include <type_traits>
#include <cuda_runtime.h>

#include <cstring>
#include <cuda_fp16.h>
#include <cuda_bf16.h>

#include <atomic>
#include <cstdarg>
#include <cstdint>
#include <cstdio>

#include "flb200.h"

namespace flb200 {

// ---------------------------------------------------------------- errors
// One message buffer per host thread; the C ABI never throws.
char* last_error_buffer();
int fail(int status, const char* fmt, ...);
extern std::atomic<long long> g_kernel_launches;

// Device facts are read once per device (SM count, opt-in shared memory).
struct DeviceInfo {
  int sm_count = 148;
  int max_smem_optin = 0;
  int cc_major = 0;
  int cc_minor = 0;
};
const DeviceInfo& device_info();

// A thread's last answers to a question that its Key (plain bytes) decides, as the scratch queries are: an
// operator asks several, and weighing the plans behind one takes 0.3 us each, up to sixteen of them.
template <typename Key, typename Value, int N = 256>
class Memo {
 public:
  // The answer kept for `key`, or null; put() then keeps one in its place.
  const Value* find(const Key& key) {
    unsigned long long h = 1469598103934665603ull;
    const unsigned char* p = reinterpret_cast<const unsigned char*>(&key);
    for (size_t i = 0; i + 4 <= sizeof(Key); i += 4) {
      unsigned w;
      memcpy(&w, p + i, 4);
      h = (h ^ w) * 1099511628211ull;
    }
    at_ = &entries_[(h ^ (h >> 32)) % N];
    return at_->used && memcmp(&at_->key, &key, sizeof(Key)) == 0 ? &at_->value : nullptr;
  }
  const Value& put(const Key& key, const Value& value) {
    memcpy(&at_->key, &key, sizeof(Key));
    at_->value = value;
    at_->used = true;
    return at_->value;
  }

 private:
  struct Entry { bool used; Key key; Value value; };
  Entry entries_[N] = {};
  Entry* at_ = nullptr;
};

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Kernels of one stream, one after the other, with little of the gap between them (1.0 to 1.4 us): the next
// one is launched as the last CTAs of this one end (programmatic stream serialization), and each begins with
// chain_begin(), which waits until the kernel before it has ended and its writes are visible, before it
// touches any memory or tensor memory.  No kernel triggers the next one earlier: with a trigger behind
// chain_begin() the next kernel's CTAs crowd the SMs that are free first (ResNet-50 scoring 29 images in
// fp32: 5770 us unchained, 5910 so, 5390 without; a 12-layer Transformer step 7840, 6980, 6695).  What
// is launched without launch_chained waits for the kernel before it as ever.
__device__ __forceinline__ void chain_begin() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <typename... Params, typename... A>
inline void launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                           A&&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);  // FLB200_AFTER_LAUNCH reads the error
}

// Checks the launch error of the kernel just issued and counts the launch.
#define FLB200_AFTER_LAUNCH(name)                                                      \
  do {                                                                                 \
    ::flb200::g_kernel_launches.fetch_add(1, std::memory_order_relaxed);               \
    cudaError_t e__ = cudaGetLastError();                                              \
    if (e__ != cudaSuccess)                                                            \
      return ::flb200::fail(FLB200_LAUNCH_FAILURE, "%s: %s", name, cudaGetErrorString(e__)); \
  } while (0)

#define FLB200_CUDA_CHECK(expr)                                                        \
  do {                                                                                 \
    cudaError_t e__ = (expr);                                                          \
    if (e__ != cudaSuccess)                                                            \
      return ::flb200::fail(FLB200_LAUNCH_FAILURE, "%s: %s", #expr, cudaGetErrorString(e__)); \
  } while (0)

#define FLB200_REQUIRE(cond, ...)                                                      \
  do {                                                                                 \
    if (!(cond)) return ::flb200::fail(FLB200_INVALID_ARG, __VA_ARGS__);               \
  } while (0)

// Grid for a grid-stride kernel: enough CTAs to cover `work_items` at
// `per_cta` items each, capped at `waves` full waves of the device
// (148 SMs x resident CTAs), so big tensors run as a few persistent waves.
inline int grid_for(long long work_items, int per_cta, int ctas_per_sm = 8, int waves = 4) {
  long long need = (work_items + per_cta - 1) / per_cta;
  long long cap = 1LL * device_info().sm_count * ctas_per_sm * waves;
  if (need < 1) need = 1;
  return static_cast<int>(need < cap ? need : cap);
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// ------------------------------------------------------------ device side
template <typename T> struct Num;
template <> struct Num<float> {
  __device__ static float to_f(float v) { return v; }
  __device__ static float from_f(float v) { return v; }
};
template <> struct Num<__half> {
  __device__ static float to_f(__half v) { return __half2float(v); }
  __device__ static __half from_f(float v) { return __float2half_rn(v); }
};
template <> struct Num<__nv_bfloat16> {
  __device__ static float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }
  __device__ static __nv_bfloat16 from_f(float v) { return __float2bfloat16_rn(v); }
};

// 16-byte vector of T (4 floats or 8 halves) moved with one 128-bit access.
template <typename T> struct alignas(16) Vec16 {
  static constexpr int N = 16 / sizeof(T);
  T v[N];
};

template <typename T>
__device__ __forceinline__ Vec16<T> load16(const T* p) {
  Vec16<T> r;
  *reinterpret_cast<uint4*>(&r) = *reinterpret_cast<const uint4*>(p);
  return r;
}
template <typename T>
__device__ __forceinline__ void store16(T* p, const Vec16<T>& r) {
  *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(&r);
}

// Its values as fp32 and back; 16-bit values are converted two at a time.
template <typename T>
__device__ __forceinline__ void unpack16(const Vec16<T>& r, float* v) {
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = r.v[j];
  } else {
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      float2 f;
      if constexpr (std::is_same<T, __half>::value)
        f = __half22float2(*reinterpret_cast<const __half2*>(r.v + j));
      else
        f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(r.v + j));
      v[j] = f.x;
      v[j + 1] = f.y;
    }
  }
}
template <typename T>
__device__ __forceinline__ Vec16<T> pack16(const float* v) {
  Vec16<T> r;
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int j = 0; j < 4; ++j) r.v[j] = v[j];
  } else {
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      if constexpr (std::is_same<T, __half>::value)
        *reinterpret_cast<__half2*>(r.v + j) = __floats2half2_rn(v[j], v[j + 1]);
      else
        *reinterpret_cast<__nv_bfloat162*>(r.v + j) = __floats2bfloat162_rn(v[j], v[j + 1]);
    }
  }
  return r;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sum over a CTA of up to 1024 threads; every thread gets the result.
// `scratch` must hold 32 values of T and is reusable after the call returns.
template <typename T>
__device__ __forceinline__ T block_sum(T v, T* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();  // scratch may still be read from a previous call
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  T r = (lane < nwarps) ? scratch[lane] : T(0);
  r = warp_sum(r);
  return r;
}

}  // namespace flb200
