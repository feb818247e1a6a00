// MXFP8 / MXFP4 quantiser and fused SwiGLU+MXFP8 producer (memory-bound kernels).
//
// One kernel family replaces the reference's pack_mx / pack_mx_vector
// (integrations/vllm/native/runtime.cu:46-113) and silu_mx
// (integrations/vllm/native/producer.cu:10-45).  Sixteen threads own one
// (row, K128 block): each loads 8 contiguous 16-bit values with one 16-byte
// load, four neighbouring threads reduce the K32 amax with two shuffles, and
// the sixteen threads emit the block's four E8M0 bytes as ONE aligned 32-bit
// word of the 512-byte scale atom.  Threads past the real work write the 0x7f
// padding words of the last 128-row scale block, so no memset node precedes
// the kernel and every byte of the scale buffer is rewritten on every call.
#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <type_traits>
#include <vector>

#include "hg_common.cuh"

namespace hg {

std::string& last_error() {
  static thread_local std::string message;
  return message;
}

namespace {

struct HostPair { void* host; void* device; };

struct HostPool {
  std::mutex mutex;
  std::vector<HostPair> idle[64];
};
HostPool& host_pool() {
  static HostPool* const pool = new HostPool;   // not destroyed: at exit the driver may be gone before it
  return *pool;
}

struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};
constexpr size_t kHostResultBytes = 256;

}  // namespace

HostResult::HostResult(cudaStream_t stream) : stream_(stream) {
  check(cudaGetDevice(&ordinal_), "cudaGetDevice");
  if (ordinal_ < 0 || ordinal_ >= 64) throw std::runtime_error("Device ordinals 0..63 are supported");
  HostPool& pool = host_pool();
  {
    std::lock_guard<std::mutex> lock(pool.mutex);
    std::vector<HostPair>& idle = pool.idle[ordinal_];
    if (!idle.empty()) {
      host = idle.back().host;
      device = idle.back().device;
      idle.pop_back();
      return;
    }
  }
  const RelaxedCapture relaxed;
  check(cudaHostAlloc(&host, kHostResultBytes, cudaHostAllocPortable | cudaHostAllocMapped), "pinned buffer");
  cudaError_t e = cudaMalloc(&device, kHostResultBytes);
  if (e != cudaSuccess) cudaFreeHost(host);
  check(e, "result buffer");
  check(cudaMemsetAsync(device, 0, kHostResultBytes, stream), "result buffer");
}

void HostResult::wait(const char* what) {
  check(cudaStreamSynchronize(stream_), what);
  waited_ = true;
}

HostResult::~HostResult() {
  if (!waited_ && cudaStreamSynchronize(stream_) != cudaSuccess) return;   // an error before the wait: work may be in flight
  HostPool& pool = host_pool();
  {
    std::lock_guard<std::mutex> lock(pool.mutex);
    std::vector<HostPair>& idle = pool.idle[ordinal_];
    if (idle.size() < kHostResultsKept) {
      idle.push_back({host, device});
      return;
    }
  }
  const RelaxedCapture relaxed;
  cudaFreeHost(host);
  cudaFree(device);
}

bool pdl_enabled() {
  static const bool enabled = [] {
    const char* v = std::getenv("HYGEMM_PDL");
    return !(v && v[0] == '0');
  }();
  return enabled;
}

template <typename T>
__device__ __forceinline__ void widen8(const uint4& raw, float (&v)[8]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = to_float<T>(uint16_t(w[i >> 1] >> ((i & 1) * 16)));
}

// SwiGLU of one (gate, up) pair with the roundings of SiluAndMul.
template <typename T, int MATH>
__device__ __forceinline__ uint16_t silu1(float g, float u) {
  const float e = MATH == 0 ? expf(-g) : __expf(-g);
  const float act = MATH == 1 ? __fdividef(g, 1.f + e) : g / (1.f + e);
  // The consumer this replaces adds a zero beta to `up` before multiplying;
  // keeping the addition preserves +0 + -0 -> +0 and with it the sign bit
  // of a zero product (integrations/vllm/native/producer.cu:30-32).
  return from_float<T>(to_float<T>(from_float<T>(act)) * __fadd_rn(u, 0.f));
}

// SwiGLU of eight (gate, up) pairs; `product` receives the 16-bit products.
template <typename T, int MATH>
__device__ __forceinline__ void silu8(const uint4& g4, const uint4& u4, float (&v)[8], uint4& product) {
  float g[8], u[8];
  widen8<T>(g4, g);
  widen8<T>(u4, u);
  uint32_t dw[4] = {0, 0, 0, 0};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint16_t p16 = silu1<T, MATH>(g[i], u[i]);
    v[i] = to_float<T>(p16);
    dw[i >> 1] |= uint32_t(p16) << ((i & 1) * 16);
  }
  product = make_uint4(dw[0], dw[1], dw[2], dw[3]);
}

__device__ __forceinline__ float exp2_fast(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float reciprocal_fast(float x) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }

// 2 N SwiGLU products by approximate exponentials and reciprocals, bit for bit silu8's.
//
// The gate's activation is rounded to 16 bits, so an fp32 value that is only nearly silu8's gives the same bits unless a
// rounding boundary lies in between.  Pairs with a value near one are computed as in silu8: over all gates of both types the two
// differ by at most 8 fp32 units down to -6 and 13 down to -16 (the error of the exponent's argument grows with it), and lanes
// whose gates all lie above -6 take a window of 10 units instead of 20.  So are gates below -16, and fp16 activations below the
// normal range, whose boundaries lie elsewhere.  up + 0 and the product are rounded once in the 16-bit type, as they are in fp32: a
// product of two fp16 values is exact in fp32, one of two bf16 values down to 2^-126 (the caller leaves values near that to silu8).
//
// Doubtful pairs are collected and computed one after the other at the end, all lanes' first ones together: a warp takes the exact
// functions once or twice for its 32 x 2 N values, and not up to N times (fp16: of sixteen pairs of a warp four had a value in
// doubt).  IN_PLACE: each behind a branch of its own, which needs fewer registers (see in_place).
constexpr uint32_t kDoubt = 20, kDoubtNear = 10;
constexpr float kNearGate = -6.f;
template <typename T, bool IN_PLACE = false, int N>
__device__ __forceinline__ void silu_fast(const uint32_t (&gate)[N], const uint32_t (&up)[N], uint32_t (&product)[N]) {
  constexpr bool kHalf = std::is_same<T, __half>::value;
  constexpr int kShift = kHalf ? 19 : 16;                        // brings the bits below the 16-bit mantissa to the top
  uint32_t least = gate[0];
#pragma unroll
  for (int i = 1; i < N; ++i) least = Packed<T>::min(least, gate[i]);
  const float2 ends = Packed<T>::widen(least);
  const float lowest = fminf(ends.x, ends.y);
  const uint32_t window = (lowest < kNearGate ? kDoubt : kDoubtNear) << kShift, boundary = 0x80000000u - window;
  uint32_t doubtful = 0;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const float2 g = Packed<T>::widen(gate[i]);
    const float2 t = mul2(g, make_float2(-1.44269504f, -1.44269504f));
    const float2 s = add2(make_float2(exp2_fast(t.x), exp2_fast(t.y)), make_float2(1.f, 1.f));
    float2 act = mul2(g, make_float2(reciprocal_fast(s.x), reciprocal_fast(s.y)));
    const uint32_t x = __float_as_uint(act.x) * (1u << kShift) - boundary, y = __float_as_uint(act.y) * (1u << kShift) - boundary;
    bool doubt = min(x, y) <= 2 * window;
    if constexpr (kHalf)   // below 2^-14; zeros, which are exact, wrap round
      doubt |= min((__float_as_uint(act.x) & 0x7fffffffu) - 1u, (__float_as_uint(act.y) & 0x7fffffffu) - 1u) < 0x38800000u - 1u;
    if constexpr (IN_PLACE) {
      if (__builtin_expect(doubt || fminf(g.x, g.y) < -16.f, 0)) act = make_float2(g.x / (1.f + expf(-g.x)), g.y / (1.f + expf(-g.y)));
    } else if (doubt) {
      doubtful |= 1u << i;
    }
    product[i] = Packed<T>::swiglu(act, up[i]);
  }
  if (!IN_PLACE && __builtin_expect(doubtful != 0 || lowest < -16.f, 0)) {
    if (lowest < -16.f) {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const float2 g = Packed<T>::widen(gate[i]);
        if (fminf(g.x, g.y) < -16.f) doubtful |= 1u << i;
      }
    }
#pragma unroll 1
    while (doubtful) {
      const int at = __ffs(int(doubtful)) - 1;
      doubtful &= doubtful - 1;
      uint32_t gate_at = gate[0], up_at = up[0];
#pragma unroll
      for (int i = 1; i < N; ++i)
        if (i == at) { gate_at = gate[i]; up_at = up[i]; }
      const float2 g = Packed<T>::widen(gate_at);
      const uint32_t exact = Packed<T>::swiglu(make_float2(g.x / (1.f + expf(-g.x)), g.y / (1.f + expf(-g.y))), up_at);
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (i == at) product[i] = exact;
    }
  }
}

template <typename T, bool FP4, bool SILU, int MATH, bool IN_PLACE = false>
__global__ void __launch_bounds__(256, IN_PLACE ? 8 : 0)
mx_quant_kernel(const uint16_t* __restrict__ in, uint8_t* __restrict__ out, uint8_t* __restrict__ sf,
                uint16_t* __restrict__ debug, int rows, int k) {
  pdl_trigger();
  // All that does not depend on the input comes before the wait: behind a kernel that releases its dependents early, as this
  // library's do, this one is resident while that one still runs, and what follows the wait is the chain that a decode step is made
  // of.  Behind one that does not (an engine's norm or attention) there is no wait to hide work in: over 110 layers of up to 128
  // tokens calls became 13 % faster back to back with all changes of that time, and 5 % behind an elementwise kernel of torch.
  const int kblocks = k >> 7;
  const int64_t real = int64_t(rows) * kblocks * 16;
  const int64_t tid = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (tid >= real) {
    // Padding words of the last 128-row scale block (rows .. roundup128(rows)-1).
    const int pad_rows = ((rows + 127) & ~127) - rows;
    const int64_t p = tid - real;
    if (pad_rows == 0 || p >= int64_t(pad_rows) * kblocks) return;
    const int kb = int(uint32_t(p) / uint32_t(pad_rows)), row = rows + int(p) - kb * pad_rows;   // p is below k
    uint32_t* const word = reinterpret_cast<uint32_t*>(sf + scale_word_offset(row, kb, k));
    pdl_wait();
    *word = 0x7f7f7f7fu;
    return;
  }
  const int lane = threadIdx.x & 31;
  const unsigned mask = 0xffffu << (lane & 16);        // the 16 threads of this (row, K128 block)
  const int sub = int(tid & 15);
  const int64_t item = tid >> 4;
  const int row = item < (int64_t(1) << 31) ? int(uint32_t(item) / uint32_t(kblocks)) : int(item / kblocks), kb = int(item - int64_t(row) * kblocks);
  const int col = kb * 128 + sub * 8;
  const uint16_t* const src = in + int64_t(row) * (SILU ? 2 * k : k) + col;
  void* const to = out + (int64_t(row) * k + col) / (FP4 ? 2 : 1);
  uint32_t* const scale_word = reinterpret_cast<uint32_t*>(sf + scale_word_offset(row, kb, k));
  // The previous kernel's output is in L2, and the prefetch does nothing; an older input comes in during the wait.  Layer calls on old
  // inputs take 0.2 % longer without it on average (23 shapes), behind a kernel that writes the input the same.
  asm volatile("prefetch.global.L2 [%0];" ::"l"(src) : "memory");
  if constexpr (SILU) asm volatile("prefetch.global.L2 [%0];" ::"l"(src + k) : "memory");
  pdl_wait();

  float v[8];
  if constexpr (SILU) {
    const uint4 g4 = *reinterpret_cast<const uint4*>(src);
    const uint4 u4 = *reinterpret_cast<const uint4*>(src + k);
    bool exact = MATH != 0 || debug;
    if (!exact) {
      const uint32_t g[4] = {g4.x, g4.y, g4.z, g4.w}, u[4] = {u4.x, u4.y, u4.z, u4.w};
      uint32_t p[4];
      silu_fast<T, IN_PLACE>(g, u, p);
      widen8<T>(make_uint4(p[0], p[1], p[2], p[3]), v);
      if constexpr (!std::is_same<T, __half>::value) {
        uint32_t top = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) top = Packed<T>::max_abs(top, p[i]);
        const float2 ends = Packed<T>::widen(top);
        exact = top && fmaxf(ends.x, ends.y) < 0x1p-100f;
      }
    }
    if (__builtin_expect(exact, 0)) {
      uint4 product;
      silu8<T, MATH>(g4, u4, v, product);
      if (debug) *reinterpret_cast<uint4*>(debug + int64_t(row) * k + col) = product;
    }
    __syncwarp(mask);
  } else {
    const uint4 x4 = *reinterpret_cast<const uint4*>(src);
    const uint32_t xw[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = to_float<T>(uint16_t(xw[i >> 1] >> ((i & 1) * 16)));
  }

  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
  amax = fmaxf(amax, __shfl_xor_sync(mask, amax, 1));
  amax = fmaxf(amax, __shfl_xor_sync(mask, amax, 2));
  const int e = mx_exponent<FP4>(amax);
  const float inv = mx_inverse_scale(e);
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] *= inv;

  if constexpr (FP4) {
    *static_cast<uint32_t*>(to) = cvt_e2m1x8(v);
  } else {
    uint2 codes;
    codes.x = cvt_e4m3x2(v[0], v[1]) | (cvt_e4m3x2(v[2], v[3]) << 16);
    codes.y = cvt_e4m3x2(v[4], v[5]) | (cvt_e4m3x2(v[6], v[7]) << 16);
    *static_cast<uint2*>(to) = codes;
  }

  // Gather the four K32 exponents of this K128 block into one scale word.
  const int base = lane & 16;
  const uint32_t byte = uint32_t(e + 127);
  const uint32_t word = __shfl_sync(mask, byte, base) | (__shfl_sync(mask, byte, base + 4) << 8) |
                        (__shfl_sync(mask, byte, base + 8) << 16) | (__shfl_sync(mask, byte, base + 12) << 24);
  if (sub == 0) *scale_word = word;
}

// ---- Many rows: weights at load time, prefill activations -----------------------------------------------------------
//
// A warp owns rows r, r+32, r+64, r+96 of a 128-row scale block x 512 columns, sixteen consecutive values per lane and row,
// and has their four 32-byte loads in flight (SwiGLU: those of the next row during a row's arithmetic).  Sixteen values per lane halve the
// instructions per value against eight (one shuffle, one exponent and one scale byte per sixteen, maxima in packed 16-bit
// form): the kernel above is bound by them, 3.8 TB/s on a 272 MB weight matrix.  The four rows share the 16-byte
// entries of the scale atoms, so scales leave as whole entries instead of single words, each a partial write of a
// sector.  With row lists the rows are gathered: a layer's two partitions are packed from the 16-bit matrix in one
// launch, without copies of the partitions in between.
constexpr int kRowsBlocks = 3;   // resident blocks of mx_rows_kernel per SM: 24 warps with 4 KB in flight each
struct QuantPart {
  const int32_t* ids;   // source row of each packed row; null = the same
  uint8_t* codes;
  uint8_t* sf;
  int rows, sources;    // packed rows; rows of the source matrix
};

struct Raw16 { uint32_t w[8]; };   // sixteen 16-bit values

__device__ __forceinline__ Raw16 load16(const uint16_t* p) {
  Raw16 r;
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]), "=r"(r.w[6]), "=r"(r.w[7])
               : "l"(p));
  return r;
}
// Sixteen values of a lane; two lanes make a K32 group, eight a K128 block.  Codes and scales as mx_quant_kernel's (a maximum
// that skips NaNs, exact scaling by a power of two).  Returns the scale word of the block; `codes` null: beyond the row.
template <typename T, bool FP4>
__device__ __forceinline__ uint32_t quantise16(const Raw16& x, uint8_t* codes, int lane) {
  uint32_t top = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) top = Packed<T>::max_abs(top, x.w[i]);
  top = Packed<T>::max_abs(top, __shfl_xor_sync(0xffffffffu, top, 1));
  const float2 ends = Packed<T>::widen(top);
  const int e = mx_exponent<FP4>(fmaxf(fmaxf(0.f, ends.x), ends.y));
  const float inv = mx_inverse_scale(e);
  if (codes) {
    float v[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 pair = Packed<T>::widen(x.w[i]);
      const float2 scaled = mul2(pair, make_float2(inv, inv));
      v[2 * i] = scaled.x;
      v[2 * i + 1] = scaled.y;
    }
    if constexpr (FP4) {
      const float (&low)[8] = *reinterpret_cast<const float (*)[8]>(v), (&high)[8] = *reinterpret_cast<const float (*)[8]>(v + 8);
      *reinterpret_cast<uint2*>(codes) = make_uint2(cvt_e2m1x8(low), cvt_e2m1x8(high));
    } else {
      uint32_t c[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) c[i] = cvt_e4m3x2(v[4 * i], v[4 * i + 1]) | (cvt_e4m3x2(v[4 * i + 2], v[4 * i + 3]) << 16);
      *reinterpret_cast<uint4*>(codes) = make_uint4(c[0], c[1], c[2], c[3]);
    }
  }
  uint32_t word = uint32_t(e + 127) << (8 * ((lane >> 1) & 3));
  word |= __shfl_xor_sync(0xffffffffu, word, 2);
  return word | __shfl_xor_sync(0xffffffffu, word, 4);
}

// Source row of packed row 128 (group / 32) + group % 32 + 32 lane (lanes 0 to 3); -1: none.
__device__ __forceinline__ int find_row(const QuantPart& part, int group, int lane) {
  const int row = (group >> 5) * 128 + (group & 31) + 32 * lane;
  if (lane >= 4 || row >= part.rows) return -1;
  const int s = part.ids ? __ldg(part.ids + row) : row;
  // a list is incomplete, its entries undefined, when ids were repeated or out of range
  return uint32_t(s) < uint32_t(part.sources) ? s : -1;
}
// Columns col .. col + 15 of this lane in row r of the group whose source rows lanes 0 to 3 hold.
__device__ __forceinline__ Raw16 load_row(int sources, int r, const uint16_t* __restrict__ in, int col, int k) {
  const int source = __shfl_sync(0xffffffffu, sources, r);
  Raw16 raw{};
  if (source >= 0 && col < k) raw = load16(in + int64_t(source) * k + col);
  return raw;
}
// Converts a group's four rows; each makes room for the same row of the next item.
template <typename T, bool FP4>
__device__ __forceinline__ void emit_rows(Raw16 (&raw)[4], const QuantPart& part, int group, int col, int k, int lane, int sources, const uint16_t* __restrict__ in, int next_col) {
  const int row0 = (group >> 5) * 128 + (group & 31);
  uint32_t word[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int row = row0 + 32 * r;
    word[r] = 0x7f7f7f7fu;   // padding rows of the last 128-row scale block
    if (row < part.rows) {
      const int64_t at = int64_t(row) * k + col;
      word[r] = quantise16<T, FP4>(raw[r], col < k ? part.codes + (FP4 ? at >> 1 : at) : nullptr, lane);
    }
    raw[r] = load_row(sources, r, in, next_col, k);
  }
  if (col < k && (lane & 7) == 0)
    *reinterpret_cast<uint4*>(part.sf + scale_word_offset(row0, col >> 7, k)) = make_uint4(word[0], word[1], word[2], word[3]);
}

// How row lists say that they are not complete: see partition_rows_kernel.
__device__ __forceinline__ int bad_list_mark(int distinct, int out_of_range) { return -1 - (2 * distinct + out_of_range); }
// {distinct ids, an id was out of range}
__device__ __forceinline__ int2 list_verdict(const int32_t* hi, int n_ids) {
  const int last = n_ids ? __ldcg(hi + n_ids - 1) : 0;
  return last >= 0 ? make_int2(n_ids, 0) : make_int2((-1 - last) >> 1, (-1 - last) & 1);
}

// Packs `low` to MXFP4 and `high` to MXFP8 (either may be empty).  Every warp walks items of one row group x 512 columns.  A row
// that has been converted makes room for the same row of the next item, and the numbers of that item's rows have been under way
// since the item before: a load that has to wait for a row number takes two latencies, and with those of the next item's rows
// asked for together with the rows a layer of 37888 x 3584 took 105.9 us to pack instead of 93.4 (whole call; two sets of four
// rows in registers).  A fourth block per SM gives nothing (94.5), a fifth spills (108).  `verdict`: where to tell the host about
// the lists, or null.
template <typename T>
__global__ void __launch_bounds__(256, kRowsBlocks)
mx_rows_kernel(const uint16_t* __restrict__ in, const QuantPart low, const QuantPart high, int k, int* __restrict__ verdict) {
  pdl_trigger();
  const int lane = threadIdx.x & 31, chunks = (k + 511) >> 9;
  const int low_groups = ((low.rows + 127) & ~127) >> 2, groups = low_groups + (((high.rows + 127) & ~127) >> 2);
  const int stride = gridDim.x * 8, item = blockIdx.x * 8 + (threadIdx.x >> 5);
  int group = item / chunks, col = ((item - group * chunks) << 9) + 16 * lane;
  pdl_wait();   // input and row lists come from the kernels before
  if (verdict && blockIdx.x == 0 && threadIdx.x == 0) *reinterpret_cast<int2*>(verdict) = list_verdict(high.ids, high.rows);
  if (group >= groups) return;
  auto rows_of = [&](int g) { return g < low_groups ? find_row(low, g, lane) : g < groups ? find_row(high, g - low_groups, lane) : -1; };
  Raw16 raw[4];
  int sources = rows_of(group);
#pragma unroll
  for (int r = 0; r < 4; ++r) raw[r] = load_row(sources, r, in, col, k);
  int ahead = item + stride;
  sources = rows_of(ahead / chunks);
  while (group < groups) {
    const int next_group = ahead / chunks, next_col = ((ahead - next_group * chunks) << 9) + 16 * lane;
    ahead += stride;
    const int after = rows_of(ahead / chunks);
    if (group < low_groups) emit_rows<T, true>(raw, low, group, col, k, lane, sources, in, next_col);
    else emit_rows<T, false>(raw, high, group - low_groups, col, k, lane, sources, in, next_col);
    group = next_group;
    col = next_col;
    sources = after;
  }
}

template <typename T, int MATH>
__device__ __forceinline__ void silu16(const Raw16& gate, const Raw16& up, Raw16& product) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    float v[8];
    uint4 p;
    silu8<T, MATH>(make_uint4(gate.w[4 * j], gate.w[4 * j + 1], gate.w[4 * j + 2], gate.w[4 * j + 3]),
                   make_uint4(up.w[4 * j], up.w[4 * j + 1], up.w[4 * j + 2], up.w[4 * j + 3]), v, p);
    product.w[4 * j] = p.x; product.w[4 * j + 1] = p.y; product.w[4 * j + 2] = p.z; product.w[4 * j + 3] = p.w;
  }
}

// SwiGLU + MXFP8 for many rows; bound by instruction issue.  2048 x 18944 bf16 44.8 us (62 % of the memory bandwidth; 46.2 with the
// exact functions at every pair in doubt and four blocks to an SM), 777 rows 19.2 us (21.7), 60 with silu8 throughout at 2048.  The
// bf16 instance spills 32 bytes a thread (80 with four blocks).
template <typename T, int MATH>
__global__ void __launch_bounds__(256, 3)
mx_silu_rows_kernel(const uint16_t* __restrict__ in, uint8_t* __restrict__ out, uint8_t* __restrict__ sf, uint16_t* __restrict__ debug, int rows, int k) {
  pdl_trigger();
  const int lane = threadIdx.x & 31, chunks = (k + 511) >> 9;
  const int item = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int group = item / chunks, col = ((item - group * chunks) << 9) + 16 * lane;
  if (group >= ((rows + 127) & ~127) >> 2) return;
  const int row0 = (group >> 5) * 128 + (group & 31);
  pdl_wait();
  struct Pair { Raw16 gate, up; };
  auto load = [&](Pair& to, int row) {
    to.gate = to.up = Raw16{};
    if (row < rows && col < k) {
      const uint16_t* at = in + int64_t(row) * 2 * k + col;
      to.gate = load16(at);
      to.up = load16(at + k);
    }
  };
  auto convert = [&](const Pair& x, int row) -> uint32_t {   // scale word of the row's K128 block
    if (row >= rows) return 0x7f7f7f7fu;
    Raw16 product;
    if (MATH == 0 && !debug) {
      silu_fast<T>(x.gate.w, x.up.w, product.w);
      if constexpr (!std::is_same<T, __half>::value) {
        uint32_t top = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) top = Packed<T>::max_abs(top, product.w[i]);
        const float2 ends = Packed<T>::widen(top);
        if (__builtin_expect(top && fmaxf(ends.x, ends.y) < 0x1p-100f, 0)) silu16<T, MATH>(x.gate, x.up, product);
      }
    } else {
      silu16<T, MATH>(x.gate, x.up, product);
      if (debug && col < k) {
        uint4* const to = reinterpret_cast<uint4*>(debug + int64_t(row) * k + col);
        to[0] = make_uint4(product.w[0], product.w[1], product.w[2], product.w[3]);
        to[1] = make_uint4(product.w[4], product.w[5], product.w[6], product.w[7]);
      }
    }
    __syncwarp();
    return quantise16<T, false>(product, col < k ? out + int64_t(row) * k + col : nullptr, lane);
  };
  uint32_t word[4] = {};
  Pair a, b;
  load(a, row0);
#pragma unroll 1   // four copies of the body do not fit the instruction cache
  for (int r = 0; r < 4; r += 2) {   // the next row's loads are in flight during a row's arithmetic
    load(b, row0 + 32 * (r + 1));
    word[0] = word[2];
    word[1] = word[3];
    word[2] = convert(a, row0 + 32 * r);
    if (r == 0) load(a, row0 + 64);
    word[3] = convert(b, row0 + 32 * (r + 1));
  }
  if (col < k && (lane & 7) == 0)
    *reinterpret_cast<uint4*>(sf + scale_word_offset(row0, col >> 7, k)) = make_uint4(word[0], word[1], word[2], word[3]);
}

// From this many elements on (SwiGLU: twice as many) the many-rows kernels are faster; below, one load per thread has the shorter chain.
// Inputs in L2, few rows against many, bf16: 1171 x 3584 (4.0 Mi) 3.2 us against 3.6, 1400 x 3584 3.8 and 3.65, 2048 x 3584 5.25 and
// 4.4, 777 x 18944 9.9 and 6.7; SwiGLU 300 x 14336 (4.1 Mi) 6.7 and 9.3, 500 x 14336 10.35 and 10.9, 585 x 14336 (8.0 Mi) 11.9
// and 11.8, 1024 x 8192 11.9 and 12.1, 600 x 18944 15.7 and 13.7, 2048 x 18944 52 and 45; fp16 the same within 5 %.  In layer calls
// around 8 Mi elements the many-rows SwiGLU is 3 % better on average.  gate_up's 37888 x 3584 weights to MXFP4: 107 us against 54.
constexpr int64_t kManyRowsElements = 4 << 20;

// Where the few-rows SwiGLU takes doubtful pairs in place (fp16).  It runs beside the GEMM of gate_up, whose pairs of CTAs (from 33 tokens
// on) leave 4096 registers in three of an SM's four parts: two blocks of 32 registers a thread, one of 40, which is what collecting the
// pairs needs.  Where gate_up fills the chip (144 row tiles) and the blocks find room in twos, or nearly so, one in ones is a wave more:
// gate_up and SwiGLU + down of 4096 x 14336 at 37 tokens (259 blocks) 28.5 us in place, 29.4 collected; of 4096 x 11008 at 40 25.1 and
// 25.6, at 56 (301 blocks) 26.1 and 26.5; of 3584 x 9344 at 64 22.3 and 23.2.  Elsewhere collecting is 1 to 2 % better (8192
// channels at 64 tokens 22.3 and 21.9; 14336 at 44, 308 blocks, 30.0 and 29.7; 18944 at 33, 305 blocks, 30.7 and 30.4).
static bool in_place(int rows, int k) { return rows > 32 && 2 * k >= 144 * 128 && int64_t(rows) * k <= 302 * 2048; }

static unsigned row_blocks(int64_t groups, int k) { return unsigned((groups * ((k + 511) / 512) + 7) / 8); }

template <typename T>
static cudaError_t launch_rows(const void* in, const QuantPart& low, const QuantPart& high, int k, cudaStream_t s, int* verdict = nullptr) {
  const int64_t groups = (int64_t((low.rows + 127) & ~127) + ((high.rows + 127) & ~127)) / 4;
  return launch_kernel(mx_rows_kernel<T>, dim3(std::min(row_blocks(groups, k), unsigned(148 * kRowsBlocks))), dim3(256), 0, s, static_cast<const uint16_t*>(in), low, high, k, verdict);
}

// The row lists of a layer from the ids of its MXFP8 channels: one block, a bitmap of the rows in shared memory, a scan of its
// words, and a warp per word that writes 32 rows at once.  The lists are only complete when ids are distinct and in range.
// Otherwise fewer than n_ids rows are set, the last entry of `hi` is left over, and it says so (list_verdict): the verdict
// belongs to the lists, wherever the packing that reads it is enqueued.
constexpr int kPartitionThreads = 1024;
__global__ void __launch_bounds__(kPartitionThreads)
partition_rows_kernel(const int64_t* __restrict__ ids, int n_ids, int rows, int32_t* __restrict__ lo, int32_t* __restrict__ hi) {
  extern __shared__ uint32_t bitmap[];   // words of the bitmap, then the MXFP8 rows before each word
  __shared__ int warp_sum[32];
  pdl_trigger();
  const int words = (rows + 31) >> 5, tid = threadIdx.x, lane = tid & 31;
  int* const before = reinterpret_cast<int*>(bitmap + words);
  for (int w = tid; w < words; w += kPartitionThreads) bitmap[w] = 0;
  __syncthreads();
  pdl_wait();
  int bad = 0;
  for (int first = tid; first < n_ids; first += 4 * kPartitionThreads) {   // four loads under way at once
    int64_t id[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) id[j] = first + j * kPartitionThreads < n_ids ? ids[first + j * kPartitionThreads] : 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (first + j * kPartitionThreads >= n_ids) continue;
      if (id[j] < 0 || id[j] >= rows) bad = 1;
      else atomicOr(bitmap + (id[j] >> 5), 1u << (id[j] & 31));
    }
  }
  bad = __syncthreads_or(bad);
  const int per = (words + kPartitionThreads - 1) / kPartitionThreads, begin = min(words, tid * per), end = min(words, begin + per);
  int mine = 0;
  for (int w = begin; w < end; ++w) mine += __popc(bitmap[w]);
  int sum = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int other = __shfl_up_sync(0xffffffffu, sum, d);
    if (lane >= d) sum += other;
  }
  if (lane == 31) warp_sum[tid >> 5] = sum;
  __syncthreads();
  if (tid < 32) {
    int total = warp_sum[tid];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int other = __shfl_up_sync(0xffffffffu, total, d);
      if (tid >= d) total += other;
    }
    warp_sum[tid] = total;
  }
  __syncthreads();
  int running = sum - mine + (tid >= 32 ? warp_sum[(tid >> 5) - 1] : 0);
  for (int w = begin; w < end; ++w) {
    before[w] = running;
    running += __popc(bitmap[w]);
  }
  __syncthreads();
#pragma unroll 4
  for (int w = tid >> 5; w < words; w += kPartitionThreads / 32) {
    const uint32_t bits = bitmap[w];
    const int row = w * 32 + lane, high = before[w] + __popc(bits & ((1u << lane) - 1u));
    if (row >= rows) continue;
    if ((bits >> lane) & 1u) {
      if (high < n_ids) hi[high] = row;
    } else if (row - high < rows - n_ids) {
      lo[row - high] = row;
    }
  }
  if (tid == 0 && warp_sum[31] != n_ids) hi[n_ids - 1] = bad_list_mark(warp_sum[31], bad);
}

template <typename T, bool FP4, bool SILU, int MATH>
static cudaError_t launch_quant(const void* in, void* out, void* sf, void* debug, int rows, int k, cudaStream_t s) {
  if (int64_t(rows) * k >= (SILU ? 2 : 1) * kManyRowsElements && (reinterpret_cast<uintptr_t>(in) & 31) == 0) {   // 32-byte loads
    if constexpr (SILU) {
      const int64_t groups = ((int64_t(rows) + 127) & ~int64_t(127)) / 4;
      return launch_kernel(mx_silu_rows_kernel<T, MATH>, dim3(row_blocks(groups, k)), dim3(256), 0, s, static_cast<const uint16_t*>(in),
                           static_cast<uint8_t*>(out), static_cast<uint8_t*>(sf), static_cast<uint16_t*>(debug), rows, k);
    } else {
      const QuantPart part{nullptr, static_cast<uint8_t*>(out), static_cast<uint8_t*>(sf), rows, rows}, none{};
      return launch_rows<T>(in, FP4 ? part : none, FP4 ? none : part, k, s);
    }
  }
  const int kblocks = k / 128;
  const int64_t pad_rows = ((rows + 127) & ~127) - rows;
  const int64_t threads = int64_t(rows) * kblocks * 16 + pad_rows * kblocks;
  const int64_t blocks = (threads + 255) / 256;
  if constexpr (SILU && MATH == 0 && std::is_same<T, __half>::value)
    if (in_place(rows, k))
      return launch_kernel(mx_quant_kernel<T, FP4, SILU, MATH, true>, dim3(unsigned(blocks)), dim3(256), 0, s,
                           static_cast<const uint16_t*>(in), static_cast<uint8_t*>(out), static_cast<uint8_t*>(sf),
                           static_cast<uint16_t*>(debug), rows, k);
  return launch_kernel(mx_quant_kernel<T, FP4, SILU, MATH>, dim3(unsigned(blocks)), dim3(256), 0, s,
                       static_cast<const uint16_t*>(in), static_cast<uint8_t*>(out), static_cast<uint8_t*>(sf),
                       static_cast<uint16_t*>(debug), rows, k);
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

static void pack_any(const void* in, void* out, void* sf, int rows, int k, int fp4, void* stream, bool bf16) {
  // Argument rule of integrations/vllm/native/runtime.cu:121.
  if (rows <= 0 || k <= 0 || k % 128 || !in || !out || !sf) throw std::runtime_error("Invalid MX pack arguments");
  if (!aligned16(in) || !aligned16(out) || !aligned16(sf))
    throw std::runtime_error("MX pack pointers must be 16-byte aligned");
  auto s = static_cast<cudaStream_t>(stream);
  cudaError_t e;
  if (bf16) e = fp4 ? launch_quant<__nv_bfloat16, true, false, 0>(in, out, sf, nullptr, rows, k, s)
                    : launch_quant<__nv_bfloat16, false, false, 0>(in, out, sf, nullptr, rows, k, s);
  else      e = fp4 ? launch_quant<__half, true, false, 0>(in, out, sf, nullptr, rows, k, s)
                    : launch_quant<__half, false, false, 0>(in, out, sf, nullptr, rows, k, s);
  check(e, "MX pack launch");
}

void pack_activations(const void* x, void* codes, void* scales, int tokens, int k, int dtype, cudaStream_t stream) {
  pack_any(x, codes, scales, tokens, k, 0, stream, dtype == HG_DTYPE_BF16);
}

static int silu_any(const void* in, void* q, void* sf, void* debug, int rows, int k, void* stream, int math, bool bf16) {
  // Argument rule and return convention of integrations/vllm/native/producer.cu:46-54.
  if (!in || !q || !sf || rows <= 0 || k <= 0 || k % 128 || math < 0 || math > 2) return int(cudaErrorInvalidValue);
  if (!aligned16(in) || !aligned16(q) || !aligned16(sf) || (debug && !aligned16(debug))) return int(cudaErrorMisalignedAddress);
  auto s = static_cast<cudaStream_t>(stream);
#define HG_SILU(T)                                                                     \
  (math == 0 ? launch_quant<T, false, true, 0>(in, q, sf, debug, rows, k, s)           \
   : math == 1 ? launch_quant<T, false, true, 1>(in, q, sf, debug, rows, k, s)         \
               : launch_quant<T, false, true, 2>(in, q, sf, debug, rows, k, s))
  return int(bf16 ? HG_SILU(__nv_bfloat16) : HG_SILU(__half));
#undef HG_SILU
}

static void split_rows(const int64_t* ids, int n_ids, int rows, int32_t* lo, int32_t* hi, cudaStream_t s) {
  if (rows <= 0 || n_ids < 0 || n_ids > rows || (n_ids && (!ids || !hi)) || (n_ids < rows && !lo)) throw std::runtime_error("Invalid split-rows arguments");
  const size_t shared = size_t((rows + 31) / 32) * 8;
  if (shared > 47 * 1024) throw std::runtime_error("Too many rows for one split");
  check(launch_kernel(partition_rows_kernel, dim3(1), dim3(kPartitionThreads), shared, s, ids, n_ids, rows, lo, hi), "partition launch");
}

static void split_pack(const void* weight, int n_ids, int rows, int k, const int32_t* lo, const int32_t* hi, void* w4, void* sf4, void* w8,
                       void* sf8, int verdict[2], int dtype, cudaStream_t s) {
  if (rows <= 0 || k <= 0 || k % 128 || n_ids < 0 || n_ids > rows || !weight || !verdict) throw std::runtime_error("Invalid split-pack arguments");
  if (dtype != HG_DTYPE_F16 && dtype != HG_DTYPE_BF16) throw std::runtime_error("Unknown weight dtype");
  if (reinterpret_cast<uintptr_t>(weight) & 31) throw std::runtime_error("Split-pack weights must be 32-byte aligned");
  if (!aligned16(w4) || !aligned16(sf4) || !aligned16(w8) || !aligned16(sf8)) throw std::runtime_error("MX pack pointers must be 16-byte aligned");
  const QuantPart low{lo, static_cast<uint8_t*>(w4), static_cast<uint8_t*>(sf4), rows - n_ids, rows}, high{hi, static_cast<uint8_t*>(w8), static_cast<uint8_t*>(sf8), n_ids, rows};
  HostResult buffers(s);
  int* const result = static_cast<int*>(buffers.host);   // written over the bus: no copy afterwards
  check(dtype == HG_DTYPE_BF16 ? launch_rows<__nv_bfloat16>(weight, low, high, k, s, result) : launch_rows<__half>(weight, low, high, k, s, result), "split-pack launch");
  buffers.wait("split-pack");
  verdict[0] = result[0];
  verdict[1] = result[1];
}

void silu_pack_activations(const void* x, void* codes, void* scales, int tokens, int k, int dtype, int math, cudaStream_t stream) {
  check(cudaError_t(silu_any(x, codes, scales, nullptr, tokens, k, stream, math, dtype == HG_DTYPE_BF16)), "SwiGLU producer");
}

}  // namespace hg

extern "C" {

const char* hg_last_error(void) { return hg::last_error().c_str(); }

int64_t hg_scale_size(int rows, int k) { return hg::scale_size(rows, k); }

// `mode` selected among kernels in the reference; every mode wrote the same
// bytes, so here all modes run the one kernel.
int hg_pack(const void* in, void* out, void* sf, int rows, int k, int fp4, void* stream) {
  HG_TRY hg::pack_any(in, out, sf, rows, k, fp4, stream, false); HG_CATCH
}
int hg_pack_mode(const void* in, void* out, void* sf, int rows, int k, int fp4, void* stream, int mode) {
  (void)mode;
  HG_TRY hg::pack_any(in, out, sf, rows, k, fp4, stream, false); HG_CATCH
}
int hg_pack_bf16(const void* in, void* out, void* sf, int rows, int k, int fp4, void* stream) {
  HG_TRY hg::pack_any(in, out, sf, rows, k, fp4, stream, true); HG_CATCH
}
int hg_pack_mode_bf16(const void* in, void* out, void* sf, int rows, int k, int fp4, void* stream, int mode) {
  (void)mode;
  HG_TRY hg::pack_any(in, out, sf, rows, k, fp4, stream, true); HG_CATCH
}

int hg_split_rows(const int64_t* ids, int n_ids, int rows, int32_t* lo, int32_t* hi, void* stream) {
  HG_TRY hg::split_rows(ids, n_ids, rows, lo, hi, static_cast<cudaStream_t>(stream)); HG_CATCH
}
int hg_split_pack(const void* weight, int n_ids, int rows, int k, const int32_t* lo, const int32_t* hi, void* w4, void* sf4, void* w8,
                  void* sf8, int* verdict, int dtype, void* stream) {
  HG_TRY hg::split_pack(weight, n_ids, rows, k, lo, hi, w4, sf4, w8, sf8, verdict, dtype, static_cast<cudaStream_t>(stream)); HG_CATCH
}

int hg_silu_pack(const void* in, void* q, void* sf, void* debug, int rows, int k, void* stream, int math) {
  return hg::silu_any(in, q, sf, debug, rows, k, stream, math, false);
}
int hg_silu_pack_bf16(const void* in, void* q, void* sf, void* debug, int rows, int k, void* stream, int math) {
  return hg::silu_any(in, q, sf, debug, rows, k, stream, math, true);
}

}  // extern "C"
