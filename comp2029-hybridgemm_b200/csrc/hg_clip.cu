// Offline MXFP4 weight quantiser with an exponent search per K32 group (load-time work).
//
// Follows integrations/vllm/allocation/fp4_quant.py:28-58 of the reference (`quantize`): the
// round-to-nearest result of hg_pack is the baseline; for every non-zero offset, in the order given, the
// group's scale byte is moved by the offset (clamped to [0,254]), the 32 values are re-rounded to E2M1 at
// that scale (saturating at 6, i.e. clipped when the scale shrinks) and the candidate replaces the best
// so far if its importance-weighted squared error is strictly smaller.  The reference runs this as a
// chain of torch ops over whole tensors (several full-size fp32 temporaries per offset); here one pass
// reads each 16-bit weight once and writes 4.25 bits per weight.
//
// Layout as mx_quant_kernel: sixteen threads own one (row, K128 block), four threads one K32 group, eight
// consecutive values per thread.  The error sum has a fixed order (eight terms left to right per thread,
// then a two-step butterfly over the four threads) so that the CPU oracle reproduces every decision.
//
// The statistics of the search (errors before and after, how far the scales moved) and the checks on its inputs are
// gathered in the same pass: the values, codes and both scales are in registers here, and as torch ops they were a
// dozen passes over full-size fp32 tensors and ten host synchronisations (4096 x 3584: 1660 us a call, 65 us now, of which
// the kernel is 43).  The kernel is bound by its arithmetic, so only the winning candidate is encoded and the offsets are read
// from the constant bank.  An item's eight terms are added in fp32, everything above that in fp64: a thread has 12 items of a
// 4096 x 3584 matrix and 590 of a 37888 x 18944 one, over which fp32 sums drift (they took 42.3 us here).
#include <algorithm>

#include "hg_common.cuh"

namespace hg {

constexpr int kMaxClipOffsets = 8;
struct ClipOffsets {
  int count;
  int value[kMaxClipOffsets];
};

// A pair of values rounded to E2M1 (nearest, ties to the even code, saturating) and back; exact in half precision.
__device__ __forceinline__ float2 e2m1_round(float x, float y) {
  uint32_t halves;
  asm("{\n"
      ".reg .b8 b;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b, %2, %1;\n"
      "cvt.rn.f16x2.e2m1x2 %0, b;\n"
      "}"
      : "=r"(halves) : "f"(x), "f"(y));
  return __half22float2(*reinterpret_cast<const __half2*>(&halves));
}

// The thread's part of the squared error of eight values at scale 2^e, weighted and plain.  (A code's value times a power of
// two is exact, so the fused multiply-add rounds once where a product and a difference would.)
__device__ __forceinline__ float clip_candidate(const float (&v)[8], const float (&weight)[8], int e, float& plain_error) {
  const float inv = mx_inverse_scale(e);
  // 2^e as a factor: e in [-127,127]; 2^-127 is the subnormal 0x00400000.
  const float scale = e == -127 ? __uint_as_float(0x00400000u) : __uint_as_float(uint32_t(e + 127) << 23);
  float sum = 0.f, plain = 0.f;
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    const float2 q = e2m1_round(v[i] * inv, v[i + 1] * inv);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float diff = __fmaf_rn(j ? q.y : q.x, scale, -v[i + j]);
      const float square = __fmul_rn(diff, diff);
      plain = __fadd_rn(plain, square);
      sum = __fadd_rn(sum, __fmul_rn(square, weight[i + j]));
    }
  }
  plain_error = plain;
  return sum;
}

// Slots of the statistics (doubles, added to): squared errors, flags, then one count per offset.
enum : int { kWeightedBefore = 0, kWeightedAfter = 1, kPlainBefore = 2, kPlainAfter = 3, kNotFinite = 4, kBadImportance = 5,
             kErrorGrew = 6, kTicket = 7, kShiftCounts = 8, kClipStats = 16 };

template <typename T, bool STATS>
__global__ void __launch_bounds__(256, 4)
mx_clip_search_kernel(const uint16_t* __restrict__ in, const float* __restrict__ importance, uint8_t* __restrict__ q4,
                      uint8_t* __restrict__ scales, int rows, int k, const __grid_constant__ ClipOffsets offsets, double* stats, double* __restrict__ host_stats) {
  const int per_row = k >> 3;
  const int64_t threads = int64_t(rows) * per_row, stride = int64_t(gridDim.x) * blockDim.x;
  const uint32_t mask = 0xfu << (threadIdx.x & 28);   // the four threads of this K32 group (groups never straddle the tail)
  double sums[4] = {0., 0., 0., 0.};
  int moved[kMaxClipOffsets] = {}, flags = 0;
  for (int64_t thread = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; thread < threads; thread += stride) {   // whole groups leave together
    const int row = threads < (int64_t(1) << 31) ? int(uint32_t(thread) / uint32_t(per_row)) : int(thread / per_row);
    const int col = int(thread - int64_t(row) * per_row) << 3;
    const uint4 raw = *reinterpret_cast<const uint4*>(in + int64_t(row) * k + col);
    const uint32_t words[4] = {raw.x, raw.y, raw.z, raw.w};
    float v[8], weight[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = to_float<T>(uint16_t(words[i] & 0xffffu));
      v[2 * i + 1] = to_float<T>(uint16_t(words[i] >> 16));
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) weight[i] = 1.f;
    if (importance && (reinterpret_cast<uintptr_t>(importance) & 15)) {
#pragma unroll
      for (int i = 0; i < 8; ++i) weight[i] = importance[col + i];
    } else if (importance) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(importance + col)), b = __ldg(reinterpret_cast<const float4*>(importance + col) + 1);
      weight[0] = a.x; weight[1] = a.y; weight[2] = a.z; weight[3] = a.w;
      weight[4] = b.x; weight[5] = b.y; weight[6] = b.z; weight[7] = b.w;
    }
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
    amax = fmaxf(amax, __shfl_xor_sync(mask, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(mask, amax, 2));
    const int base = mx_exponent<true>(amax);

    auto group_error = [&](float part) {
      part = __fadd_rn(part, __shfl_xor_sync(mask, part, 1));
      return __fadd_rn(part, __shfl_xor_sync(mask, part, 2));
    };
    float plain, part = clip_candidate(v, weight, base, plain);
    float best = group_error(part), best_part = part, best_plain = plain;
    const float first = best;
    if constexpr (STATS) {
      sums[kWeightedBefore] += part;
      sums[kPlainBefore] += plain;
    }
    int best_e = base;
    for (int o = 0; o < offsets.count; ++o) {
      if (offsets.value[o] == 0) continue;
      const int e = max(-127, min(127, base + offsets.value[o]));
      part = clip_candidate(v, weight, e, plain);
      const float error = group_error(part);
      if (error < best) { best = error; best_e = e; best_part = part; best_plain = plain; }
    }
    float scaled[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) scaled[i] = v[i] * mx_inverse_scale(best_e);
    *reinterpret_cast<uint32_t*>(q4 + (int64_t(row) * k + col) / 2) = cvt_e2m1x8(scaled);
    if ((col & 31) == 0) scales[int64_t(row) * (k >> 5) + (col >> 5)] = uint8_t(best_e + 127);
    if constexpr (STATS) {
      sums[kWeightedAfter] += best_part;
      sums[kPlainAfter] += best_plain;
      float zero = 0.f;   // stays zero unless a value is infinite or NaN
#pragma unroll
      for (int i = 0; i < 8; ++i) zero = fmaf(v[i], 0.f, zero);
      if (!(zero == 0.f)) flags |= 1;
      if (row == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (!(weight[i] >= 0.f) || !isfinite(weight[i])) flags |= 2;
      }
      if (!(best <= first * (1.f + 1e-6f) + 1e-25f)) flags |= 4;
      if ((col & 31) == 0) {
#pragma unroll
        for (int o = 0; o < kMaxClipOffsets; ++o)
          if (o < offsets.count && best_e - base == offsets.value[o]) ++moved[o];
      }
    }
  }
  if constexpr (STATS) {
    __shared__ double block_sum[8][kClipStats];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto over_warp = [&](double value, int slot) {
#pragma unroll
      for (int d = 16; d; d >>= 1) value += __shfl_xor_sync(0xffffffffu, value, d);
      if (lane == 0) block_sum[warp][slot] = value;
    };
#pragma unroll
    for (int i = 0; i < 4; ++i) over_warp(sums[i], i);
#pragma unroll
    for (int i = 0; i < 3; ++i) over_warp(double((flags >> i) & 1), kNotFinite + i);
    if (lane == 0) block_sum[warp][7] = 0.;
#pragma unroll
    for (int o = 0; o < kMaxClipOffsets; ++o) over_warp(double(moved[o]), kShiftCounts + o);
    __syncthreads();
    if (threadIdx.x < kClipStats) {   // half a warp
      double total = 0.;
      for (int w = 0; w < 8; ++w) total += block_sum[w][threadIdx.x];
      if (total != 0.) atomicAdd(stats + threadIdx.x, total);
      // The last block to arrive writes the totals to the host's buffer.
      __threadfence();
      __syncwarp(0xffffu);
      double arrived = threadIdx.x == 0 ? atomicAdd(stats + kTicket, 1.) + 1. : 0.;
      arrived = __shfl_sync(0xffffu, arrived, 0);
      if (arrived == double(gridDim.x)) {
        __threadfence();
        host_stats[threadIdx.x] = threadIdx.x == kTicket ? 0. : __ldcg(stats + threadIdx.x);
        __syncwarp(0xffffu);
        stats[threadIdx.x] = 0.;   // ready for the next call
      }
    }
  }
}

static void clip_pack(const void* in, const float* importance, void* q4, void* scales, int rows, int k, const int* offsets, int n_offsets,
                      int dtype, double* stats, double* host_stats, cudaStream_t s) {
  if (!in || !q4 || !scales || rows <= 0 || k <= 0 || k % 128) throw std::runtime_error("Invalid MX clip-pack arguments");
  if (n_offsets < 0 || n_offsets > kMaxClipOffsets || (n_offsets && !offsets)) throw std::runtime_error("At most 8 exponent offsets");
  if (dtype != HG_DTYPE_F16 && dtype != HG_DTYPE_BF16) throw std::runtime_error("Unknown input dtype");
  if ((reinterpret_cast<uintptr_t>(in) & 15) || (reinterpret_cast<uintptr_t>(q4) & 3)) throw std::runtime_error("Weights must be 16-byte aligned");
  ClipOffsets list{};
  list.count = n_offsets;
  for (int i = 0; i < n_offsets; ++i) {
    if (offsets[i] < -254 || offsets[i] > 254) throw std::runtime_error("Exponent offset out of range");
    list.value[i] = offsets[i];
  }
  const int64_t blocks = (int64_t(rows) * (k / 8) + 255) / 256;
  // With statistics every block ends in sixteen atomics, so the grid is about what the machine holds at once.
  const dim3 grid(unsigned(stats ? std::min<int64_t>(blocks, 148 * 4) : blocks)), block(256);
  const auto* src = static_cast<const uint16_t*>(in);
  auto* codes = static_cast<uint8_t*>(q4);
  auto* bytes = static_cast<uint8_t*>(scales);
  if (stats) {
    if (dtype == HG_DTYPE_BF16) mx_clip_search_kernel<__nv_bfloat16, true><<<grid, block, 0, s>>>(src, importance, codes, bytes, rows, k, list, stats, host_stats);
    else mx_clip_search_kernel<__half, true><<<grid, block, 0, s>>>(src, importance, codes, bytes, rows, k, list, stats, host_stats);
  } else {
    if (dtype == HG_DTYPE_BF16) mx_clip_search_kernel<__nv_bfloat16, false><<<grid, block, 0, s>>>(src, importance, codes, bytes, rows, k, list, nullptr, nullptr);
    else mx_clip_search_kernel<__half, false><<<grid, block, 0, s>>>(src, importance, codes, bytes, rows, k, list, nullptr, nullptr);
  }
  check(cudaGetLastError(), "clip-pack launch");
}

}  // namespace hg

extern "C" int hg_clip_pack(const void* in, const float* importance, void* q4, void* scales, int rows, int k,
                            const int* offsets, int n_offsets, int dtype, void* stream) {
  HG_TRY
  hg::clip_pack(in, importance, q4, scales, rows, k, offsets, n_offsets, dtype, nullptr, nullptr, static_cast<cudaStream_t>(stream));
  HG_CATCH
}

extern "C" int hg_clip_pack_stats(const void* in, const float* importance, void* q4, void* scales, int rows, int k,
                                  const int* offsets, int n_offsets, int dtype, double* host_stats, void* stream) {
  HG_TRY
  if (!host_stats) throw std::runtime_error("Invalid MX clip-pack arguments");
  const auto s = static_cast<cudaStream_t>(stream);
  hg::HostResult result(s);
  hg::clip_pack(in, importance, q4, scales, rows, k, offsets, n_offsets, dtype, static_cast<double*>(result.device), static_cast<double*>(result.host), s);
  result.wait("clip-pack");
  std::copy(static_cast<double*>(result.host), static_cast<double*>(result.host) + hg::kClipStats, host_stats);
  HG_CATCH
}
