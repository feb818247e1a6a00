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
// Four threads own one K32 group, eight consecutive values per thread.  The error sum has a fixed order (eight terms left
// to right per thread, then a two-step butterfly over the four threads) so that the CPU oracle reproduces every decision.
//
// The statistics of the search (errors before and after, how far the scales moved) and the checks on its inputs are
// gathered in the same pass: the values, codes and both scales are in registers here, and as torch ops they were a
// dozen passes over full-size fp32 tensors and ten host synchronisations (4096 x 3584: 1660 us a call, 48 us now, of which
// the kernel is 30).  The kernel is bound by its arithmetic, 300 instructions per eight values with three candidates; 580 with
// one value to an instruction, every candidate evaluated in full, a division per item and a counter per offset (call 65 us,
// kernel 43).  Of its issue slots it uses two thirds: candidates are chains of dependent instructions, so the first two run
// side by side (33.7 -> 30.6 us).  An item's eight terms are added in fp32, everything above that in fp64: a thread has 13
// items of a 4096 x 3584 matrix and 590 of a 37888 x 18944 one, over which fp32 sums drift.
#include <algorithm>
#include <type_traits>

#include "hg_common.cuh"

namespace hg {

constexpr int kMaxClipOffsets = 8;
struct ClipOffsets {
  int count, tried;                // as given; those that are not zero
  int value[kMaxClipOffsets], trial[kMaxClipOffsets];
};

// A pair of values rounded to E2M1 (nearest, ties to the even code, saturating) and back; exact in half precision.
__device__ __forceinline__ float2 e2m1_round(float2 x) {
  uint32_t halves;
  asm("{\n"
      ".reg .b8 b;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b, %2, %1;\n"
      "cvt.rn.f16x2.e2m1x2 %0, b;\n"
      "}"
      : "=r"(halves) : "f"(x.x), "f"(x.y));
  return __half22float2(*reinterpret_cast<const __half2*>(&halves));
}

// 2^e as a factor; e in [-127,127], 2^-127 is the subnormal 0x00400000.
__device__ __forceinline__ float clip_scale(int e) { return __uint_as_float(max(uint32_t(e + 127) << 23, 0x00400000u)); }

// The thread's part of the squared error of its eight values at scale 2^e: plain (x) and weighted (y).  (A code's value times a
// power of two is exact, so the fused multiply-add rounds once where a product and a difference would.)  Two values to an
// instruction up to their squares, which are added one after the other.
template <bool WEIGHTED>
__device__ __forceinline__ float2 clip_candidate(const float2 (&v)[4], const float2 (&weight)[4], int e) {
  const float inv = mx_inverse_scale(e), scale = clip_scale(e);
  const float2 invs = make_float2(inv, inv), minus = make_float2(-scale, -scale);
  float plain = 0.f, sum = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 d = fma2(e2m1_round(mul2(v[i], invs)), minus, v[i]);
    const float2 square = mul2(d, d);
    plain = __fadd_rn(__fadd_rn(plain, square.x), square.y);
    if constexpr (WEIGHTED) {
      const float2 term = mul2(square, weight[i]);
      sum = __fadd_rn(__fadd_rn(sum, term.x), term.y);
    }
  }
  return make_float2(plain, WEIGHTED ? sum : plain);
}
// Slots of the statistics (doubles, added to): squared errors, flags, then one count per offset.
enum : int { kWeightedBefore = 0, kWeightedAfter = 1, kPlainBefore = 2, kPlainAfter = 3, kNotFinite = 4, kBadImportance = 5,
             kErrorGrew = 6, kTicket = 7, kShiftCounts = 8, kClipStats = 16 };

// Which offset a group moved by is counted in a table of all differences of two exponents.
constexpr int kShiftTable = 2 * 254 + 1;

// A warp owns the K32 groups of one 32-column block in eight rows, four lanes to a group, and walks down the rows: the
// importance of its columns stays in registers, addresses only grow, and a block's eight warps read 512 contiguous bytes of a row.
// Where K is 128 mod 256, half of the last column block's warps have nothing to do, and without offsets round-to-nearest is evaluated
// twice: 15 million weights with importance and offsets 0, -1, -2 take 22.8 us at K = 384, 20.7 at 640 and 18.1 at 3584 (26.7 each with
// sixteen threads to a K128 block), without offsets 16.9 at 384 (16.9) and 13.9 at 3584 (16.7).
template <typename T, bool WEIGHTED, bool STATS>
__global__ void __launch_bounds__(256, 4)
mx_clip_search_kernel(const uint16_t* __restrict__ in, const float* __restrict__ importance, uint8_t* __restrict__ q4,
                      uint8_t* __restrict__ scales, int rows, int k, const __grid_constant__ ClipOffsets offsets, double* stats, double* __restrict__ host_stats) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int column_blocks = (k + 255) >> 8, walkers = gridDim.x / column_blocks;
  const int column_block = blockIdx.x % column_blocks, walker = blockIdx.x / column_blocks;
  const int col = column_block * 256 + warp * 32 + (lane & 3) * 8;
  __shared__ int moved[STATS ? kShiftTable : 1];
  if constexpr (STATS) {
    for (int i = threadIdx.x; i < kShiftTable; i += 256) moved[i] = 0;
    __syncthreads();
  }
  double sums[4] = {0., 0., 0., 0.};
  int flags = 0;
  if (col < k) {   // whole warps: k is a multiple of 128
    float2 weight[4] = {};
    float least = 1.f;
    if constexpr (WEIGHTED) {
      bool usable = true;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float one = importance[col + i];
        (i & 1 ? weight[i >> 1].y : weight[i >> 1].x) = one;
        least = i ? fminf(least, one) : one;
        usable = usable && one >= 0.f;
        if (!(one >= 0.f) || !isfinite(one)) flags |= 2;
      }
      // A candidate is only ruled out by one of its terms where all terms of the group are non-negative.
      const unsigned good = __ballot_sync(0xffffffffu, usable) >> (lane & 28);
      if ((good & 15u) != 15u) least = -INFINITY;
    }
    const int row_step = walkers * 8, row0 = walker * 8 + (lane >> 2);
    const int64_t src_step = int64_t(row_step) * k * 2, codes_step = int64_t(row_step) * (k >> 1), scale_step = int64_t(row_step) * (k >> 5);
    const char* src = reinterpret_cast<const char*>(in + int64_t(row0) * k + col);
    uint8_t *codes = q4 + (int64_t(row0) * k + col) / 2, *scale_byte = scales + int64_t(row0) * (k >> 5) + (col >> 5);
    int left = rows - row0;   // rows from this lane's to the end
    uint4 raw = left > 0 ? __ldcs(reinterpret_cast<const uint4*>(src)) : make_uint4(0u, 0u, 0u, 0u);
    for (; __any_sync(0xffffffffu, left > 0); left -= row_step) {
      const bool inside = left > 0;
      const uint32_t words[4] = {raw.x, raw.y, raw.z, raw.w};
      src += src_step;
      raw = left > row_step ? __ldcs(reinterpret_cast<const uint4*>(src)) : make_uint4(0u, 0u, 0u, 0u);   // the next rows'
      float2 v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = Packed<T>::widen(words[i]);
      uint32_t top = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) top = Packed<T>::max_abs(top, words[i]);
      const float2 mine = Packed<T>::widen(top);
      const float largest = fmaxf(fmaxf(0.f, mine.x), mine.y);   // NaNs are skipped
      float amax = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, 1));
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
      const int base = mx_exponent<true>(amax);

      auto group_error = [&](float part) {
        part = __fadd_rn(part, __shfl_xor_sync(0xffffffffu, part, 1));
        return __fadd_rn(part, __shfl_xor_sync(0xffffffffu, part, 2));
      };
      auto candidate_exponent = [&](int o) { return max(-127, min(127, base + offsets.trial[o])); };
      auto consider = [&](float error, float2 part, int e, float& best, float2& best_part, int& best_e) {
        if (error < best) { best = error; best_part = part; best_e = e; }
      };
      // Rounding to nearest and the first candidate side by side: two chains of dependent instructions instead of one.
      const int e1 = offsets.tried ? candidate_exponent(0) : base;
      const float2 first_part = clip_candidate<WEIGHTED>(v, weight, base), part1 = clip_candidate<WEIGHTED>(v, weight, e1);
      const float first = group_error(first_part.y), error1 = group_error(part1.y);
      float2 best_part = first_part;
      float best = first;
      int best_e = base;
      consider(error1, part1, e1, best, best_part, best_e);
      for (int o = 1; o < offsets.tried; ++o) {
        const int e = candidate_exponent(o);
        // A value beyond 6 x 2^e is clipped, and its term alone is a lower bound of the candidate's error in the very arithmetic
        // of the sum (adding what is not negative never makes it less).  From two binades down on that settles nearly every
        // group that holds no column of outstanding importance.
        if (offsets.trial[o] <= -2) {
          const float d = fminf(__fmaf_rn(6.f, clip_scale(e), -largest), 0.f);
          unsigned out = __ballot_sync(0xffffffffu, __fmul_rn(__fmul_rn(d, d), least) >= best);
          out |= out >> 1;
          out |= out >> 2;
          if ((out & 0x11111111u) == 0x11111111u) continue;
        }
        const float2 part = clip_candidate<WEIGHTED>(v, weight, e);
        consider(group_error(part.y), part, e, best, best_part, best_e);
      }
      if (inside) {
        const float inv = mx_inverse_scale(best_e);
        float scaled[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 s = mul2(v[i], make_float2(inv, inv));
          scaled[2 * i] = s.x;
          scaled[2 * i + 1] = s.y;
        }
        *reinterpret_cast<uint32_t*>(codes) = cvt_e2m1x8(scaled);
        if ((lane & 3) == 0) {
          *scale_byte = uint8_t(best_e + 127);
          if constexpr (STATS) atomicAdd(moved + best_e - base + 254, 1);
        }
        if constexpr (STATS) {
          sums[kPlainBefore] += first_part.x;
          sums[kPlainAfter] += best_part.x;
          if constexpr (WEIGHTED) {
            sums[kWeightedBefore] += first_part.y;
            sums[kWeightedAfter] += best_part.y;
          }
          float zero = 0.f;   // stays zero unless a value is infinite or NaN
          float2 zeros = make_float2(0.f, 0.f);
#pragma unroll
          for (int i = 0; i < 4; ++i) zeros = fma2(v[i], make_float2(0.f, 0.f), zeros);
          zero = zeros.x + zeros.y;
          if (!(zero == 0.f)) flags |= 1;
          if (!(best <= first * (1.f + 1e-6f) + 1e-25f)) flags |= 4;
        }
      }
      codes += codes_step;
      scale_byte += scale_step;
    }
    if constexpr (STATS && !WEIGHTED) {
      sums[kWeightedBefore] = sums[kPlainBefore];
      sums[kWeightedAfter] = sums[kPlainAfter];
    }
  }
  if constexpr (STATS) {
    __shared__ double block_sum[8][kClipStats];
    auto over_warp = [&](double value, int slot) {
#pragma unroll
      for (int d = 16; d; d >>= 1) value += __shfl_xor_sync(0xffffffffu, value, d);
      if (lane == 0) block_sum[warp][slot] = value;
    };
#pragma unroll
    for (int i = 0; i < 4; ++i) over_warp(sums[i], i);
#pragma unroll
    for (int i = 0; i < 3; ++i) over_warp(double((flags >> i) & 1), kNotFinite + i);
    __syncthreads();   // `moved` is complete
    if (lane == 0) {
      block_sum[warp][kTicket] = 0.;
#pragma unroll
      for (int o = 0; o < kMaxClipOffsets; ++o) block_sum[warp][kShiftCounts + o] = warp == 0 && o < offsets.count ? moved[offsets.value[o] + 254] : 0;
    }
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
    if (offsets[i]) list.trial[list.tried++] = offsets[i];
  }
  // About what the machine holds at once (with statistics every block ends in sixteen atomics), the same number for every 256 columns.
  const int64_t column_blocks = (int64_t(k) + 255) / 256, row_groups = (int64_t(rows) + 7) / 8;
  const int64_t walkers = std::max<int64_t>(1, std::min(row_groups, 148 * 4 / column_blocks));
  const dim3 grid(unsigned(column_blocks * walkers)), block(256);
  const auto* src = static_cast<const uint16_t*>(in);
  auto* codes = static_cast<uint8_t*>(q4);
  auto* bytes = static_cast<uint8_t*>(scales);
  auto launch = [&](auto type, auto weighted) {
    using T = decltype(type);
    constexpr bool kWeighted = decltype(weighted)::value;
    if (stats) mx_clip_search_kernel<T, kWeighted, true><<<grid, block, 0, s>>>(src, importance, codes, bytes, rows, k, list, stats, host_stats);
    else mx_clip_search_kernel<T, kWeighted, false><<<grid, block, 0, s>>>(src, importance, codes, bytes, rows, k, list, nullptr, nullptr);
  };
  auto launch_typed = [&](auto type) {
    if (importance) launch(type, std::true_type());
    else launch(type, std::false_type());
  };
  if (dtype == HG_DTYPE_BF16) launch_typed(__nv_bfloat16());
  else launch_typed(__half());
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
