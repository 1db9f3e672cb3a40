// Shared helpers for the sm_100a MoE kernels: error plumbing for the C ABI,
// element-type traits and 128-bit vector access.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <atomic>
#include <utility>

#include "../../include/b200moe.h"

namespace b200moe {

// Records a message for b200moe_last_error() and returns `code`.
int fail(int code, const char* fmt, ...);

#define B200_CHECK_ARG(cond, ...)                                   \
  do {                                                              \
    if (!(cond)) return ::b200moe::fail(B200MOE_E_BADARG, __VA_ARGS__); \
  } while (0)

// An error that a call returns also stays behind as the thread's last error, which the next
// B200_LAUNCH_OK would take for its own: it is cleared where it is reported.
#define B200_CUDA_OK(expr)                                                     \
  do {                                                                         \
    cudaError_t e__ = (expr);                                                  \
    if (e__ != cudaSuccess) {                                                  \
      (void)cudaGetLastError();                                                \
      return ::b200moe::fail(B200MOE_E_CUDA, "%s failed: %s", #expr,          \
                             cudaGetErrorString(e__));                         \
    }                                                                          \
  } while (0)

#define B200_LAUNCH_OK(name)                                                   \
  do {                                                                         \
    cudaError_t e__ = cudaGetLastError();                                      \
    if (e__ != cudaSuccess)                                                    \
      return ::b200moe::fail(B200MOE_E_CUDA, "launch of %s failed: %s", name, \
                             cudaGetErrorString(e__));                         \
  } while (0)

// Launch of a kernel that calls pdl_wait() before it touches global memory.  `early`: with
// programmatic stream serialisation, i.e. the kernel may be launched while its predecessor in the
// stream still runs, so that its set-up (and the launch itself) is off the critical path; the wait
// ends when every earlier kernel of the stream has completed (each of them waited for its own
// predecessor) and its writes are visible.  A decode step is a chain of few-microsecond kernels and
// gains 0.5 to 1 us per launch, a chain of nine at a few thousand rows as much.  Kernels of many waves lose
// (blocks that wait take the place of blocks that work).  Layer calls with plain launches from 2048 rows on / with
// early ones, single bursts, us: qwen3 fp8 8000 rows 191 / 179; one of 8 DeepSeek ranks at 4096 rows 270 / 261, 8192 rows
// 278 / 271; small 16-bit layer 4096 rows 127 / 118, 8192 rows 171 / 161; Mixtral 16-bit 4096 rows 1306 / 1294, 8192 rows
// 2209 / 2180, int4 1386 / 1377 and 2481 / 2480; DeepSeek of 256 experts 4800 rows no difference, 8000 rows 1627 / 1645 (the
// one that loses), 32768 rows 3279 / 3410, 65536 rows 5 % slower; gpt-oss MXFP4 4096 rows 508 / 499, 8192 rows 678 / 665
// (its GEMM apart, which has a line of its own: gemm_tc_mx.cu), 16384 rows 1419 / 1481.
constexpr int64_t kEarlyLaunchRows = 8192;   // routed rows up to which a layer's kernels launch early
template <typename... Params, typename... Args>
inline cudaError_t launch_pdl(bool early, void (*kern)(Params...), dim3 grid, dim3 block, size_t smem,
                              cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = early ? 1 : 0;
  cfg.attrs = attr; cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, Params(std::forward<Args>(args))...);
}
// Every thread that touches global memory calls the wait (what an earlier kernel of the stream writes is read with plain
// loads behind it: __ldg is for weights and their scales, which stay as they are while a kernel runs); the trigger lets the next kernel of the
// stream be launched (it holds its own wait until this one has completed).  The grouped GEMMs
// trigger when a CTA's last tile is done, everything else at once.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#define B200_LAUNCHED(name, ...)                                               \
  do {                                                                         \
    cudaError_t e__ = (__VA_ARGS__);                                           \
    if (e__ != cudaSuccess) {                                                  \
      (void)cudaGetLastError();                                                \
      return ::b200moe::fail(B200MOE_E_CUDA, "launch of %s failed: %s", name, \
                             cudaGetErrorString(e__));                         \
    }                                                                          \
  } while (0)

constexpr int kMaxDevices = 64;

inline int current_device() {
  int dev = 0;
  cudaGetDevice(&dev);
  return (dev >= 0 && dev < kMaxDevices) ? dev : 0;
}

// SM count of the current device (cached per device: a process may drive several).
inline int sm_count() {
  static std::atomic<int> n[kMaxDevices];
  const int dev = current_device();
  int v = n[dev].load(std::memory_order_relaxed);
  if (v == 0) {
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    if (v <= 0) v = 148;
    n[dev].store(v, std::memory_order_relaxed);
  }
  return v;
}

inline cudaStream_t as_stream(b200moe_stream s) { return (cudaStream_t)s; }

inline int dtype_bytes(b200moe_dtype t) {
  switch (t) {
    case B200MOE_F32: case B200MOE_I32: case B200MOE_U32: return 4;
    case B200MOE_F16: case B200MOE_BF16: return 2;
    case B200MOE_I64: return 8;
    default: return 1;
  }
}

// ---- scalar conversions --------------------------------------------------
template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// e4m3fn round-to-nearest-even with saturation to +-448 (NaN stays NaN).
__device__ __forceinline__ uint8_t f32_to_e4m3(float v) {
  return (uint8_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
}
// Two at once (one conversion instruction), x in the low byte.
__device__ __forceinline__ uint32_t f32x2_to_e4m3x2(float x, float y) {
  return __nv_cvt_float2_to_fp8x2(make_float2(x, y), __NV_SATFINITE, __NV_E4M3);
}
__device__ __forceinline__ float2 e4m3x2_to_f32x2(uint32_t v) {
  const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)v, __NV_E4M3);
  return __half22float2(*reinterpret_cast<const __half2*>(&h));
}
__device__ __forceinline__ float e4m3_to_f32(uint8_t v) {
  __half_raw h = __nv_cvt_fp8_to_halfraw(v, __NV_E4M3);
  return __half2float(*reinterpret_cast<__half*>(&h));
}

// e5m2 is the upper byte of an IEEE half.
__device__ __forceinline__ float e5m2_to_f32(uint8_t v) {
  __half_raw h;
  h.x = (unsigned short)((unsigned short)v << 8);
  return __half2float(*reinterpret_cast<__half*>(&h));
}

// e2m1 code (4 bits) -> float: {0,.5,1,1.5,2,3,4,6} with sign bit 3.
__device__ __forceinline__ float e2m1_to_f32(uint32_t code) {
  const float mag[8] = {0.f, 0.5f, 1.f, 1.5f, 2.f, 3.f, 4.f, 6.f};
  float m = mag[code & 7];
  return (code & 8) ? -m : m;
}
// e8m0 byte -> 2^(b-127) (b = 0 gives 2^-127, a subnormal float; 255 = NaN).
__device__ __forceinline__ float e8m0_to_f32(uint32_t b) {
  if (b == 255) return __uint_as_float(0x7fc00000u);
  if (b == 0) return __uint_as_float(0x00400000u);
  return __uint_as_float(b << 23);
}

// ---- 16-byte vector load/store ---------------------------------------------
struct alignas(16) vec16 { uint32_t w[4]; };

__device__ __forceinline__ vec16 ld16(const void* p) {
  return *reinterpret_cast<const vec16*>(p);
}
__device__ __forceinline__ void st16(void* p, const vec16& v) {
  *reinterpret_cast<vec16*>(p) = v;
}

// Dispatch a lambda-like macro body on a 16/32-bit float element type.
#define B200_DISPATCH_FLOAT(DTYPE, NAME, ...)                                  \
  switch (DTYPE) {                                                             \
    case B200MOE_F32: { using scalar_t = float; __VA_ARGS__; break; }          \
    case B200MOE_F16: { using scalar_t = __half; __VA_ARGS__; break; }         \
    case B200MOE_BF16: { using scalar_t = __nv_bfloat16; __VA_ARGS__; break; } \
    default:                                                                   \
      return ::b200moe::fail(B200MOE_E_BADARG,                                 \
                             "%s: only float32, float16 and bfloat16 are "     \
                             "supported", NAME);                               \
  }

}  // namespace b200moe
