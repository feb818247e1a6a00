// Shared host/device helpers of the hybrid MX linear library (sm_100a only).
#pragma once
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <cstdint>
#include <stdexcept>
#include <string>
#include <utility>

#include "../../include/hygemm.h"

namespace hg {

// Thread-local message behind hg_last_error(); the error convention follows
// integrations/vllm/native/runtime.cu:15-18 of the reference.
std::string& last_error();

inline void check(cudaError_t e, const char* what = "CUDA") {
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

#define HG_TRY try {
#define HG_CATCH                                   \
  }                                                \
  catch (std::exception const& e) {                \
    hg::last_error() = e.what();                   \
    return -1;                                     \
  }                                                \
  return 0;

// Bytes of the padded E8M0 buffer: 512-byte atoms of 128 rows x 4 K32 groups.
__host__ __device__ inline int64_t scale_size(int rows, int k) {
  return rows <= 0 || k <= 0 ? 0 : int64_t((rows + 127) / 128) * (k / 128) * 512;
}

// Byte offset of the 32-bit word holding the four K32 scales of (row, K128 block kb).
__host__ __device__ inline int64_t scale_word_offset(int row, int kb, int k) {
  return (int64_t(row / 128) * (k / 128) + kb) * 512 + (row % 32) * 16 + ((row % 128) / 32) * 4;
}

// For calls that end with a host-side result: 256 bytes each of pinned memory that kernels can write (a copy from device
// memory, through a pageable buffer above all, costs more than the wait itself) and of device memory, zeroed in the order
// of the stream, that a kernel leaves zeroed.  A call holds a pair of its own for its duration.  Pairs go back to a pool, as many
// as calls were ever under way at once on a device (at most kHostResultsKept wait there), once the stream has been
// waited for; one whose stream cannot be waited for stays out of use.  They are allocated and freed in relaxed capture mode, so
// that another thread's capture is not disturbed.
constexpr size_t kHostResultsKept = 16;
class HostResult {
 public:
  explicit HostResult(cudaStream_t stream);
  ~HostResult();
  HostResult(const HostResult&) = delete;
  void wait(const char* what);   // for the stream; `host` is complete then
  void* host = nullptr;
  void* device = nullptr;
 private:
  cudaStream_t stream_;
  int ordinal_ = 0;
  bool waited_ = false;
};

#ifdef __CUDACC__
// Programmatic dependent launch.  Every kernel of the library is launched with the
// programmatic-stream-serialization attribute (unless HYGEMM_PDL=0): it may start while its
// predecessor in the stream drains, does its set-up and any work that does not depend on the
// predecessor, and calls pdl_wait() before it reads the predecessor's output or writes global memory.
// pdl_trigger() lets the next kernel in the stream do the same.  Without the attribute both are no-ops.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

bool pdl_enabled();

template <typename... KernelArgs, typename... Args>
inline cudaError_t launch_kernel(void (*kernel)(KernelArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                 Args&&... args) {
  cudaLaunchConfig_t config{};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[0].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attribute;
  config.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&config, kernel, KernelArgs(std::forward<Args>(args))...);
}

// Smallest e with amax * 2^-e <= MAX (448 for E4M3, 6 for E2M1), clamped to
// [-127,127]; e = 0 for an all-zero block.  Equals ceil(log2(amax/MAX)) of
// integrations/vllm/native/runtime.cu:71-72 for every 16-bit input without a
// transcendental (the CPU tests compare this formula, restated in the oracle,
// for all of them; the GPU tests quantise every one as the maximum of a group).
template <bool FP4>
__device__ __forceinline__ int mx_exponent(float amax) {
  const uint32_t b = __float_as_uint(amax);
  if (b == 0) return 0;
  // The mantissa carries into the exponent when it lies above that of MAX (1.5 x 2^2, 1.75 x 2^8).
  return max(-127, FP4 ? int((b + 0x3fffffu) >> 23) - 129 : int((b + 0x1fffffu) >> 23) - 135);
}

// 2^-e as an fp32 factor (e in [-127,127]; 2^-127 is a subnormal constant).
__device__ __forceinline__ float mx_inverse_scale(int e) {
  return __uint_as_float(max(uint32_t(127 - e) << 23, 0x00400000u));
}

// Two floats -> two E4M3 bytes (lo in bits 0-7), round-to-nearest-even, saturating.
__device__ __forceinline__ uint32_t cvt_e4m3x2(float lo, float hi) {
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  return r;
}

// Eight floats -> eight E2M1 nibbles (element 0 in the lowest nibble).
__device__ __forceinline__ uint32_t cvt_e2m1x8(const float (&v)[8]) {
  uint32_t r;
  asm("{\n"
      ".reg .b8 b0, b1, b2, b3;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n"
      "mov.b32 %0, {b0, b1, b2, b3};\n"
      "}"
      : "=r"(r)
      : "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]));
  return r;
}

template <typename T> __device__ __forceinline__ float to_float(uint16_t bits);
template <> __device__ __forceinline__ float to_float<__half>(uint16_t bits) {
  return __half2float(__ushort_as_half(bits));
}
template <> __device__ __forceinline__ float to_float<__nv_bfloat16>(uint16_t bits) {
  return __uint_as_float(uint32_t(bits) << 16);
}
template <typename T> __device__ __forceinline__ uint16_t from_float(float v);
template <> __device__ __forceinline__ uint16_t from_float<__half>(float v) {
  return __half_as_ushort(__float2half_rn(v));
}
template <> __device__ __forceinline__ uint16_t from_float<__nv_bfloat16>(float v) {
  return __bfloat16_as_ushort(__float2bfloat16_rn(v));
}

// Pairs of 16-bit values in a word.
template <typename T> struct Packed;
template <> struct Packed<__half> {
  static __device__ __forceinline__ uint32_t min(uint32_t a, uint32_t b) {   // skips NaNs
    const __half2 m = __hmin2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
    return *reinterpret_cast<const uint32_t*>(&m);
  }
  static __device__ __forceinline__ uint32_t max_abs(uint32_t a, uint32_t b) {   // a is a maximum already
    const __half2 m = __hmax2(*reinterpret_cast<const __half2*>(&a), __habs2(*reinterpret_cast<const __half2*>(&b)));
    return *reinterpret_cast<const uint32_t*>(&m);
  }
  static __device__ __forceinline__ float2 widen(uint32_t v) { return __half22float2(*reinterpret_cast<const __half2*>(&v)); }
  static __device__ __forceinline__ uint32_t swiglu(float2 act, uint32_t up) {   // (up + 0) as in silu8
    const __half2 p = __hmul2(__floats2half2_rn(act.x, act.y), __hadd2(*reinterpret_cast<const __half2*>(&up), __float2half2_rn(0.f)));
    return *reinterpret_cast<const uint32_t*>(&p);
  }
};
template <> struct Packed<__nv_bfloat16> {
  static __device__ __forceinline__ uint32_t min(uint32_t a, uint32_t b) {   // skips NaNs
    const __nv_bfloat162 m = __hmin2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&m);
  }
  static __device__ __forceinline__ uint32_t max_abs(uint32_t a, uint32_t b) {
    const __nv_bfloat162 m = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&a), __habs2(*reinterpret_cast<const __nv_bfloat162*>(&b)));
    return *reinterpret_cast<const uint32_t*>(&m);
  }
  static __device__ __forceinline__ float2 widen(uint32_t v) { return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u)); }
  static __device__ __forceinline__ uint32_t swiglu(float2 act, uint32_t up) {
    const __nv_bfloat162 p = __hmul2(__floats2bfloat162_rn(act.x, act.y), __hadd2(*reinterpret_cast<const __nv_bfloat162*>(&up), __float2bfloat162_rn(0.f)));
    return *reinterpret_cast<const uint32_t*>(&p);
  }
};

// Two fp32 operations per instruction.
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n mul.rn.f32x2 z, x, y;\n mov.b64 {%0, %1}, z;\n}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n add.rn.f32x2 z, x, y;\n mov.b64 {%0, %1}, z;\n}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n .reg .b64 x, y, z, w;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n mov.b64 z, {%6, %7};\n fma.rn.f32x2 w, x, y, z;\n mov.b64 {%0, %1}, w;\n}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
#endif  // __CUDACC__

}  // namespace hg
