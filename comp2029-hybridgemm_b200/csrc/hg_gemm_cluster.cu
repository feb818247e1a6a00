// Hybrid MXFP4xMXFP8 + MXFP8xMXFP8 GEMM on clusters of CTAs (sm_100a): what HG_SCHEDULE_AUTO runs.
//
//   out[t, ids[r]] = sum_g 2^(sw[r,g]+sx[t,g]-254) * sum_{k in g} W[r,k] * X[t,k]
//
// Differences from the single-CTA kernel of hg_gemm_tc.cu, which serves the explicit tile schedules:
// * Split K inside a cluster.  A tile's K range is cut over the CTAs (or CTA pairs) of one cluster; each pushes its
//   fp32 partials to the shared memory of the CTAs that own the columns, and the owners add them in K order.
//   No workspace, no ticket, no second launch: the chain store -> ticket -> load through global memory that ended
//   a cut tile cost 3.5 us, the exchange between neighbours about one.
// * Weights by TMA.  MXFP4 rows through the tensor map type 16U4_ALIGN16B, which unpacks sixteen codes into the first half of
//   each swizzled 16-byte chunk, the 8-bit container the f8f6f4 kinds read: one instruction brings a K256 slice of a tile, no
//   thread touches the weights and nothing passes through L1.  Alone it streams at 6.3 TB/s (61 MB, 148 SMs).  8-byte
//   cp.async from loader warps needs a line of L1 for every line in flight, and beside 228 KB of shared memory only 28 KB
//   of L1 are left: the same loop was 3 us slower on gate_up with the larger carve-out.
// * Row tiles of 128, 64 or 32 rows, always inside one 128-row scale atom.  The ring holds only the rows a tile loads; the MMA
//   still reads 128, from the address at which the atom's first row would lie, and the accumulator lanes of rows
//   that were not loaded are never read.
//
// Roles per CTA: warp 0 weights and their scales (TMA), warp 1 MMA issue (idle in the second CTA of a pair, whose copies
// complete on the first CTA's barriers: reporting every stage with a remote arrive cost 750 cycles each), then epilogue warps
// (four; in pairs eight, two per TMEM quarter on alternate groups of sixteen columns), then one warp for the activations and
// their scales (TMA) or, FUSED, up to eight warps that quantise the activations.
// One warp per scheduler runs most of these roles alone, so a dependent instruction costs about five cycles and nothing
// hides it: loops here carry no divisions, addresses are independent of each other, and descriptors are sums.
// Every mbarrier wait is bounded; on expiry the CTA records a code, drains and leaves.
#include <algorithm>
#include <array>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <numeric>
#include <vector>

#include "hg_gemm_cluster.cuh"

namespace hg {

namespace {

constexpr int kClusterQuantThreads = 256;   // activation quantisers at most: sixteen per token and K256 step, and no warp without a token
constexpr int kQuantAhead = 4;              // steps whose activations a quantiser has in registers or on the way
__host__ __device__ constexpr int epilogue_sides(int pair) { return pair == 2 ? 2 : 1; }
__host__ __device__ constexpr int first_act_warp(int pair) { return 2 + 4 * epilogue_sides(pair); }
__host__ __device__ constexpr int cluster_threads(int pair, bool fused) { return first_act_warp(pair) * 32 + (fused ? kClusterQuantThreads : 32); }
constexpr int kClusterMaxStages = 12;
constexpr int kMaxSmem = 232448;
constexpr uint32_t kScaleStride = 16;                           // TMEM columns per scale set: weights 4, activations up to 12

struct ClusterParams {
  int rows[2], cut_log[2], tiles[2];   // a 128-row atom (PAIR: two) is cut into 2^cut_log tiles
  int slot_rows, least_rows;           // height of the taller and of the shorter tiles
  const uint8_t* sfa[2];
  const int32_t* ids[2];
  const uint8_t* sfb;
  OutTargets out;
  int outputs, tokens, k, kblocks;
  int n_tile, n_tail, token_tiles, stages, split, split_log, share_log, clusters;
  int async_push;      // partials travel by st.async
  int ring_exchange;   // partials are exchanged in the ring, which is idle by then (a cluster that splits K has one unit)
  int acc_shift, overlap;
  uint64_t by_token_tiles, by_tiles;   // see fast_div
  uint32_t tmem_cols;
  const uint16_t* x;
  int x_bf16;
  int* status;
  // Of the WIDE instance alone (see ClusterPlan), and behind the others' fields: in front of async_push they shifted what every
  // instance reads, and each launch took 0.03 to 0.05 us longer (GEMM alone, 4096 x 4096 at 37 tokens 5.90 -> 5.94, 6144 x 4096 at 37
  // 6.67 -> 6.71, 2270 x 896 at 775 6.54 -> 6.59).
  int n_step, sf_atoms, turned;
#ifdef HG_TRACE
  unsigned long long* trace;
#endif
};

// Partial tiles are exchanged in groups of four columns, [group][row][4] fp32; every slice owns a power of two of them.
__host__ __device__ inline int share_log_of(int n_tile, int split) {
  int log = 0;
  while ((split << log) * 4 < n_tile) ++log;
  return log;
}

// A pipeline stage covers two K128 blocks (K256): two weight tiles of slot_rows x 128 B in the 8-bit container, two
// activation tiles, two scale atoms of the weights and two per 128 tokens of the activations.
struct ClusterSmem {
  uint32_t b, sfa, sfb, a, red, bars, end;  // byte offsets from the 1024-aligned base; activations start at 0
  uint32_t a_tile, b_tile;                  // bytes of one K128 block
  uint32_t sfb_stage;                       // bytes of the activation scales of a stage: two atoms for every 128 tokens a tile touches
};
__host__ __device__ inline ClusterSmem cluster_smem(int stages, int n_tile, int sf_atoms, int pair, int split, int slot_rows, int least_rows, int ring_exchange) {
  ClusterSmem s;
  s.a_tile = uint32_t(slot_rows) * 128u;
  s.b_tile = uint32_t(n_tile / pair) * 128u;
  s.sfb_stage = uint32_t(sf_atoms) * 1024u;
  s.b = 0;
  s.sfa = uint32_t(stages) * 2u * s.b_tile;
  s.sfb = s.sfa + uint32_t(stages) * 1024u;
  s.a = s.sfb + uint32_t(stages) * s.sfb_stage;
  // An MMA reads the 128 rows of the whole atom: up to 128 - least_rows before the ring, up to 128 - slot_rows behind it.
  const uint32_t before = uint32_t(128 - least_rows) * 128u, behind = uint32_t(128 - slot_rows) * 128u;
  if (s.a < before) s.a = before;
  s.a = (s.a + 1023u) & ~1023u;
  s.red = s.a + uint32_t(stages) * 2u * s.a_tile;
  const uint32_t exchange = split > 1 ? uint32_t(split << share_log_of(n_tile, split)) * 2048u : 0u;
  s.bars = s.red + exchange;
  if (ring_exchange) {
    s.bars = s.a + exchange > s.red ? s.a + exchange : s.red;
    s.red = s.a;
  }
  s.end = s.bars + uint32_t((2 * 12 + 8) * 8 + 32);
  const uint32_t read_end = s.a + uint32_t(stages) * 2u * s.a_tile + behind;
  if (s.end < read_end) s.end = read_end;
  return s;
}
static_assert(kClusterMaxStages == 12, "the barrier block of cluster_smem holds twelve stages");

template <int PAIR> __device__ __forceinline__ void cg_alloc(uint32_t slot, uint32_t cols) {
  if constexpr (PAIR == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  } else {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
}
template <int PAIR> __device__ __forceinline__ void cg_dealloc(uint32_t addr, uint32_t cols) {
  if constexpr (PAIR == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
  else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
// Arrives on the barrier at this offset in every CTA of the tile when all MMAs issued so far have retired.
template <int PAIR> __device__ __forceinline__ void cg_commit(uint32_t bar, uint16_t cta_mask) {
  if constexpr (PAIR == 1) tc_commit(bar);
  else
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"(cta_mask) : "memory");
}
// The same, in every CTA of the mask whatever the tile.
template <int PAIR> __device__ __forceinline__ void cg_commit_to(uint32_t bar, uint16_t cta_mask) {
  if constexpr (PAIR == 1)
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"(cta_mask) : "memory");
  else cg_commit<PAIR>(bar, cta_mask);
}
template <int PAIR> __device__ __forceinline__ void cg_cp_scales(uint32_t tmem, uint64_t desc) {
  if constexpr (PAIR == 1) tc_cp_scales(tmem, desc);
  else asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(tmem), "l"(desc) : "memory");
}
template <int PAIR>
__device__ __forceinline__ void cg_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate, uint32_t sfa, uint32_t sfb) {
  if constexpr (PAIR == 1) tc_mma(d, a, b, idesc, accumulate, sfa, sfb);
  else
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n"
        "}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb) : "memory");
}

// Shared-memory descriptors by words: the high one holds the stride of eight rows, version 1 and the swizzle.
constexpr uint32_t kDescTile = (1024u >> 4) | (1u << 14) | (kSwizzle128B << 29), kDescScales = (128u >> 4) | (1u << 14);
__device__ __forceinline__ uint64_t desc_of(uint32_t low, uint32_t high) { return uint64_t(low) | (uint64_t(high) << 32); }

// Copies into this CTA's shared memory; in a pair `bar` is a cluster address and may lie in either CTA.
template <int PAIR>
__device__ __forceinline__ void cg_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  if constexpr (PAIR == 1) tma_load_3d(dst, map, bar, x, y, z);
  else
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
// Two consecutive 512-byte scale atoms, `row` counted in atoms from the start of the buffer.
__device__ __forceinline__ void load_scales_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int row) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(0), "r"(row) : "memory");
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// The same where nothing in memory is handed over, and the release would wait for the thread's stores.
__device__ __forceinline__ void arrive_remote_relaxed(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void store_remote(uint32_t cluster_addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
// 16 bytes to another CTA's shared memory; their arrival counts on a barrier there, so no fence and no second message.
__device__ __forceinline__ void store_async(uint32_t cluster_addr, uint32_t cluster_bar, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%2, %3, %4, %5}, [%1];"
               ::"r"(cluster_addr), "r"(cluster_bar), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// n / d with inverse = ceil(2^40 / d), exact while n d < 2^40; the host passes 0 where that or the product does not fit.
__host__ __device__ __forceinline__ int fast_div(int64_t n, int d, uint64_t inverse) {
  return inverse ? int((uint64_t(n) * inverse) >> 40) : int(n / d);
}

// One work unit: a row tile and a token tile, token tiles innermost.  Decode runs its MXFP8 tiles first: their stores
// scatter over the whole output row, and all but the last epilogue of a CTA run under the next main loop.  With several
// token tiles they are spread evenly among the MXFP4 tiles, so that the two partitions of a channel range (both sorted)
// are stored at about the same time and meet in L2: an MXFP8 tile writes one or two channels of nearly every sector.
// Where the number of clusters and that of the token tiles have a common factor, a cluster with several units would meet some of the
// token tiles only, and some clusters all the short ones (777 tokens in steps of 256: eight whole tiles beside four whole and four
// short ones).  There a row tile starts with the token tile that its round over the clusters has come to (`turned`).
struct Unit {
  int part, atom, first, last, token0, n;   // rows first .. last - 1 of the 128-row atom (PAIR: of atoms 2 atom and 2 atom + 1)
};
// A cluster's units: u = cluster, cluster + clusters, ...; `turn` counts them modulo the token tiles.
__host__ __device__ __forceinline__ void next_unit(const ClusterParams& p, int& u, int& turn) {
  u += p.clusters;
  if (++turn == p.token_tiles) turn = 0;
}
template <bool WIDE>
__host__ __device__ __forceinline__ Unit unit_at(const ClusterParams& p, int u, int cluster, int turn) {
  Unit w;
  int tile;
  if (p.token_tiles == 1) {
    w.part = u < p.tiles[1];
    tile = w.part ? u : u - p.tiles[1];
    w.token0 = 0;
    w.n = p.n_tail;
  } else {
    const int t = fast_div(u, p.token_tiles, p.by_token_tiles), total = p.tiles[0] + p.tiles[1];
    int tt = u - t * p.token_tiles;
    if (WIDE && p.turned) {   // the row tile's first unit is of this round over the clusters, or of the one before
      tt += turn - (tt > cluster);
      if (tt < 0) tt += p.token_tiles;
      if (tt >= p.token_tiles) tt -= p.token_tiles;
    }
    const int high_before = fast_div(int64_t(t) * p.tiles[1], total, p.by_tiles);
    const int high_after = fast_div(int64_t(t + 1) * p.tiles[1], total, p.by_tiles);
    w.part = high_after > high_before;
    tile = w.part ? high_before : t - high_before;
    const int step = WIDE ? p.n_step : p.n_tile;
    w.token0 = tt * step;
    w.n = tt == p.token_tiles - 1 ? p.n_tail : step;
  }
  const int log = p.cut_log[w.part], height = kTileRows >> log;
  w.atom = tile >> log;
  w.first = (tile & ((1 << log) - 1)) * height;
  w.last = w.first + height;
  return w;
}

// First K256 step of a slice of K (of the slice behind the last one: the end).
__host__ __device__ __forceinline__ int first_step(const ClusterParams& p, int slice) {
  return (((p.kblocks + 1) >> 1) * slice) >> p.split_log;
}

// WIDE: token tiles that start in the middle of a scale atom, a last tile wider than the others, units in turn (see ClusterPlan).  An
// instance by itself: behind a quantiser, where its code is new to the instruction caches, a launch of it takes 0.3 us more (1536 x
// 1536 at 887 tokens, quantiser included, 8.5 us against 8.8; behind another launch of its own both take 6.5).
template <typename T, int PAIR, bool FUSED, bool WIDE>
__global__ void __launch_bounds__(cluster_threads(PAIR, FUSED), 1)
cluster_gemm_kernel(const __grid_constant__ ClusterParams p, const __grid_constant__ ClusterMaps maps) {
  if (threadIdx.x == 0) HG_STAMP(0);
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const ClusterSmem lay = cluster_smem(p.stages, p.n_tile, WIDE ? p.sf_atoms : (p.n_tile + 127) / 128, PAIR, p.split, p.slot_rows, p.least_rows, p.ring_exchange);
  const uint32_t bars = base + lay.bars;
  auto full_bar = [&](int s) { return bars + uint32_t(s) * 8u; };
  auto empty_bar = [&](int s) { return bars + uint32_t(kClusterMaxStages + s) * 8u; };
  auto acc_full_bar = [&](int s) { return bars + uint32_t(2 * kClusterMaxStages + s) * 8u; };
  auto acc_empty_bar = [&](int s) { return bars + uint32_t(2 * kClusterMaxStages + 2 + s) * 8u; };
  const uint32_t red_full = bars + uint32_t(2 * kClusterMaxStages + 4) * 8u;    // every slice's partials of this share are here
  const uint32_t red_empty = bars + uint32_t(2 * kClusterMaxStages + 5) * 8u;   // every slice's ring is idle
  const uint32_t drain_bar = bars + uint32_t(2 * kClusterMaxStages + 6) * 8u;
  volatile int* words = reinterpret_cast<volatile int*>(base_ptr + lay.bars + (2 * kClusterMaxStages + 8) * 8);
  volatile int* abort_flag = words + 1;

  constexpr int kSides = epilogue_sides(PAIR), kActWarp = first_act_warp(PAIR);
  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int cluster_ctas = PAIR * p.split;
  const int rank = cluster_ctas == 1 ? 0 : int(cluster_rank());
  const int cluster = cluster_ctas == 1 ? int(blockIdx.x) : int(blockIdx.x) / cluster_ctas;
  const int half = PAIR == 2 ? rank & 1 : 0;
  const int slice = PAIR == 2 ? rank >> 1 : rank;

  if (threadIdx.x == 0) {
    if (p.tiles[0]) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.low)) : "memory");
    if (p.tiles[1]) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.high)) : "memory");
    if (!FUSED) {
      if (PAIR == 2) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.act_scales)) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.act)) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.tail)) : "memory");
    }
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full_bar(s), 1 + (FUSED ? (blockDim.x >> 5) - kActWarp : 1));   // weights; activations or the quantiser warps
      mbar_init(empty_bar(s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(acc_full_bar(s), 1);
      mbar_init(acc_empty_bar(s), 4 * kSides * PAIR);
    }
    mbar_init(red_full, p.async_push ? 1u : uint32_t(4 * kSides * p.split));   // one thread, with the bytes to come; or every warp
    mbar_init(red_empty, uint32_t(p.split));
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) cg_alloc<PAIR>(smem_u32(const_cast<int*>(words)), p.tmem_cols);
  tc_fence_before();
  __syncwarp();
  if (cluster_ctas > 1) cluster_sync();   // barriers of every CTA are initialised before anyone arrives remotely
  else __syncthreads();
  tc_fence_after();
  pdl_trigger();
  const uint32_t tmem_base = uint32_t(*words);
  if (threadIdx.x == 0) HG_STAMP(1);

  const uint32_t sf_cols = tmem_base + p.tmem_cols - 2u * kScaleStride;
  const int units = (p.tiles[0] + p.tiles[1]) * p.token_tiles;
  const int step_begin = first_step(p, slice), step_end = first_step(p, slice + 1);   // K256 steps of this slice
  int error = 0;

  if (warp == 0) {
    // ------------------------------------------------------------------ weights and their scales (TMA)
    // They were complete before the first launch (hg_run), so this stream does not wait for the kernel in front.  The warp
    // walks the loop together and an elected lane issues: behind a `lane == 0` branch every copy took 80 cycles to issue.
    const uint32_t smem0 = __shfl_sync(0xffffffffu, base, 0);
    const uint32_t bars0 = PAIR == 1 ? smem0 + lay.bars : __shfl_sync(0xffffffffu, map_to_rank(bars, uint32_t(rank & ~1)), 0);
    int stage = 0;
    uint32_t phase = 1;
    for (int u = cluster, turn = 0; u < units && !error; next_unit(p, u, turn)) {
      const Unit w = unit_at<WIDE>(p, u, cluster, turn);
      const int atom = w.atom * PAIR + half;
      const uint8_t* sfa_src = p.sfa[w.part] + int64_t(atom) * p.kblocks * 512;
      const int row = atom * kTileRows + w.first;
      const uint32_t weight_bytes = uint32_t(w.last - w.first) * (w.part ? 256u : 128u);
      for (int step = step_begin; step < step_end; ++step) {
        const int kb = 2 * step, nkb = min(2, p.kblocks - kb);
        if (!warp_wait(empty_bar(stage), phase, abort_flag)) { error = kErrLoader; break; }
        if (elect_one()) {
          const uint32_t bar = bars0 + uint32_t(stage) * 8u, dst = smem0 + lay.a + uint32_t(2 * stage) * lay.a_tile;
          const uint32_t scales = smem0 + lay.sfa + uint32_t(stage) * 1024u;
          // Rows and blocks beyond the matrix arrive as zeros.  In a pair the first CTA expects both CTAs' bytes.
          if (PAIR == 1) mbar_expect_tx(bar, weight_bytes + uint32_t(nkb) * 512u);
          else if (half == 0) mbar_expect_tx(full_bar(stage), 2u * (weight_bytes + 1024u));
          if (w.part) cg_load_3d<PAIR>(dst, &maps.high, bar, 0, row, kb);
          else cg_load_3d<PAIR>(dst, &maps.low, bar, 0, row, kb);
          if (PAIR == 1) bulk_load(scales, sfa_src + int64_t(kb) * 512, uint32_t(nkb) * 512u, bar);
          else load_scales_pair(scales, w.part ? &maps.high_scales : &maps.low_scales, bar, atom * p.kblocks + kb);
        }
        __syncwarp();
        if (++stage == p.stages) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (!FUSED && warp == kActWarp) {
    // ------------------------------------------------------------------ activations and their scales (TMA)
    // One copy brings both K128 blocks (the map's third dimension counts them).
    if (!FUSED) {
      // They are the previous kernel's output; the weight stream is not and already runs.  Everything up to the first copy is
      // done before the wait.
      bool waiting = true;
      const uint32_t smem0 = __shfl_sync(0xffffffffu, base, 0);
      const uint32_t bars0 = PAIR == 1 ? smem0 + lay.bars : __shfl_sync(0xffffffffu, map_to_rank(bars, uint32_t(rank & ~1)), 0);
      const int atoms = (p.tokens + 127) >> 7;
      int stage = 0;
      uint32_t phase = 1;
      for (int u = cluster, turn = 0; u < units && !error; next_unit(p, u, turn)) {
        const Unit w = unit_at<WIDE>(p, u, cluster, turn);
        const int first_atom = w.token0 >> 7, n_atoms = min(((WIDE ? w.token0 & 127 : 0) + w.n + 127) >> 7, atoms - first_atom);
        const int row = w.token0 + half * (w.n / PAIR);
        const bool whole = w.n == (WIDE ? p.n_step : p.n_tile);
        const uint8_t* sfb_src = p.sfb + int64_t(first_atom) * p.kblocks * 512;
        for (int step = step_begin; step < step_end; ++step) {
          const int kb = 2 * step, nkb = min(2, p.kblocks - kb);
          if (!warp_wait(empty_bar(stage), phase, abort_flag)) { error = kErrProducer; break; }
          if (waiting) {
            pdl_wait();
            waiting = false;
            if (lane == 0) HG_STAMP(2);
          }
          if (elect_one()) {
            const uint32_t bar = bars0 + uint32_t(stage) * 8u, dst = smem0 + lay.b + uint32_t(2 * stage) * lay.b_tile;
            if (PAIR == 1) mbar_expect_tx(bar, uint32_t(w.n) * 256u + uint32_t(n_atoms * nkb) * 512u);   // a block beyond K arrives as zeros
            else if (half == 0) mbar_expect_tx(full_bar(stage), 2u * (uint32_t(w.n / 2) * 256u + uint32_t(n_atoms) * 1024u));
            // a last token tile of another width has a box of its own: its second block follows the first directly
            if (whole) cg_load_3d<PAIR>(dst, &maps.act, bar, 0, row, kb);
            else cg_load_3d<PAIR>(dst, &maps.tail, bar, 0, row, kb);
            for (int a = 0; a < n_atoms; ++a) {
              const uint32_t scales = smem0 + lay.sfb + uint32_t(stage) * lay.sfb_stage + uint32_t(a) * 1024u;
              if (PAIR == 1) bulk_load(scales, sfb_src + (int64_t(a) * p.kblocks + kb) * 512, uint32_t(nkb) * 512u, bar);
              else load_scales_pair(scales, &maps.act_scales, bar, (first_atom + a) * p.kblocks + kb);
            }
          }
          __syncwarp();
          if (++stage == p.stages) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (FUSED && warp >= kActWarp) {
    // ------------------------------------------------------------------ activation quantisers
    // Two neighbouring threads own one K32 group of one token in each K256 step, with the arithmetic of mx_quant_kernel: codes and
    // scales are the bytes hg_pack would have produced.  What bounds this is latency, of the loads above all, so a thread has
    // the next kQuantAhead steps' values on the way.  With 128 threads of 32 values each and one step ahead a block of
    // Qwen2.5-7B took longer in captured calls than with a quantiser in front from two tokens on; now it does not up to sixteen
    // (8 tokens 40.7 us with separate quantisers, 40.4 with qkv and o_proj quantised here, 39.1 with gate_up too).  A launch has two
    // tokens to a warp and no more warps than that: seven idle ones made a block at one token take 38.8 us instead of 37.1, at four
    // 38.9 instead of 38.0.
    if constexpr (FUSED) {
      const int tq = threadIdx.x - kActWarp * 32;
      const int token = tq >> 4, blk = (tq >> 3) & 1, g = (tq >> 1) & 3, part = tq & 1;
      const int steps = cluster < units ? step_end - step_begin : 0;
      const int mine = token < p.tokens ? min(steps, ((p.kblocks - blk + 1) >> 1) - step_begin) : 0;   // steps that have this block
      const char* const x_at = reinterpret_cast<const char*>(p.x + int64_t(token) * p.k + int64_t(step_begin) * 256 + (tq & 15) * 16);
      const uint32_t codes_at = base + lay.b + uint32_t(blk) * lay.b_tile + uint32_t(token) * 128u + ((uint32_t(2 * g + part) ^ uint32_t(token & 7)) << 4);
      const uint32_t scale_at = base + lay.sfb + uint32_t(blk) * 512u + uint32_t(token) * 16u + uint32_t(g);
      struct Values { uint4 low, high; } ahead[kQuantAhead];
      auto load_x = [&](int step, Values& to) {
        to.low = to.high = make_uint4(0u, 0u, 0u, 0u);
        if (step < mine) {
          const uint4* const src = reinterpret_cast<const uint4*>(x_at + step * 512);
          to.low = src[0];
          to.high = src[1];
        }
      };
      auto quantise = [&](const Values& x, uint32_t (&codes)[4], auto type) {   // returns the scale byte
        using X = decltype(type);
        const uint32_t word[8] = {x.low.x, x.low.y, x.low.z, x.low.w, x.high.x, x.high.y, x.high.z, x.high.w};
        uint32_t top = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) top = Packed<X>::max_abs(top, word[i]);
        top = Packed<X>::max_abs(top, __shfl_xor_sync(0xffffffffu, top, 1));
        const float2 ends = Packed<X>::widen(top);
        const int e = mx_exponent<false>(fmaxf(fmaxf(0.f, ends.x), ends.y));
        const float inv = mx_inverse_scale(e);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 a = Packed<X>::widen(word[2 * i]), b = Packed<X>::widen(word[2 * i + 1]);
          codes[i] = cvt_e4m3x2(a.x * inv, a.y * inv) | (cvt_e4m3x2(b.x * inv, b.y * inv) << 16);
        }
        return uint32_t(e + 127);
      };
      // An input that no kernel has just written comes into L2 during the wait.
      for (int i = 0; i < mine; ++i) asm volatile("prefetch.global.L2 [%0];" ::"l"(x_at + i * 512) : "memory");
      int stage = 0;
      uint32_t phase = 1;
      pdl_wait();   // x is the previous kernel's output
      for (int u = cluster; u < units && !error; u += p.clusters) {
#pragma unroll
        for (int i = 0; i < kQuantAhead; ++i) load_x(i, ahead[i]);
        for (int first = 0; first < steps && !error; first += kQuantAhead) {
#pragma unroll
          for (int i = 0; i < kQuantAhead; ++i) {
            const int step = first + i;
            if (step >= steps || error) break;
            uint32_t codes[4];
            const uint32_t scale = p.x_bf16 ? quantise(ahead[i], codes, __nv_bfloat16()) : quantise(ahead[i], codes, __half());
            load_x(step + kQuantAhead, ahead[i]);
            if (!warp_wait(empty_bar(stage), phase, abort_flag)) { error = kErrLoader; break; }
            if (step < mine) {   // columns of tokens that are not there are never stored
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(codes_at + uint32_t(2 * stage) * lay.b_tile),
                           "r"(codes[0]), "r"(codes[1]), "r"(codes[2]), "r"(codes[3]) : "memory");
              if (part == 0) asm volatile("st.shared.u8 [%0], %1;" ::"r"(scale_at + uint32_t(stage) * lay.sfb_stage), "r"(scale) : "memory");
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(full_bar(stage));
            if (++stage == p.stages) { stage = 0; phase ^= 1u; }
          }
        }
      }
    }
  } else if (warp == 1) {
    if (half == 0) {
      // ---------------------------------------------------------------- MMA issue
      const uint32_t smem0 = __shfl_sync(0xffffffffu, base, 0), tmem0 = __shfl_sync(0xffffffffu, tmem_base, 0);
      const uint32_t sf0 = __shfl_sync(0xffffffffu, sf_cols, 0);
      const uint16_t pair_mask = uint16_t(3u << (rank & ~1));
      // low words of the shared-memory descriptors of stage 0; a stage is a constant number of 16-byte units further on
      const uint32_t a_desc = (smem0 + lay.a) >> 4, a_stage = lay.a_tile >> 3, b_desc = smem0 >> 4, b_stage = lay.b_tile >> 3;
      const uint32_t sfa_desc = (smem0 + lay.sfa) >> 4, sfb_desc = (smem0 + lay.sfb) >> 4, sfb_stage = lay.sfb_stage >> 4;
      // Waits until the accumulator of the n-th unit is free.  Overlapping accumulators: one becomes free when the epilogue of the
      // OTHER one has drained the shared columns, so accumulator 1 waits for an arrival on its first use as well.
      auto acc_free = [&](int n) {
        const uint32_t parity = (uint32_t(n >> 1) & 1u) ^ (p.overlap && (n & 1) ? 0u : 1u);
        return PAIR == 2 ? warp_wait_cluster(acc_empty_bar(n & 1), parity, abort_flag) : warp_wait(acc_empty_bar(n & 1), parity, abort_flag);
      };
      int stage = 0, it = 0, issued = 0;
      uint32_t phase = 0;
      for (int u = cluster, turn = 0; u < units && !error; next_unit(p, u, turn), ++it) {
        const Unit w = unit_at<WIDE>(p, u, cluster, turn);
        const int acc = it & 1;
        if (!acc_free(it)) { error = kErrMmaAcc; break; }
        tc_fence_after();
        const uint32_t tmem_d = tmem0 + uint32_t(acc * p.acc_shift);
        const uint32_t a_block = uint32_t(w.last - w.first) * 8u;
        const uint32_t b_block = uint32_t(w.n / PAIR) * 8u;   // descriptor units (16 bytes) between the stage's activation tiles
        const uint32_t idesc = (w.part ? 0u : 5u << 7) | (uint32_t(w.n >> 3) << 17) | (1u << 23) | (uint32_t(PAIR * kTileRows >> 4) << 24);
        // After an odd multiple of 64 tokens a tile starts in the middle of a scale atom.
        const uint32_t sfb_col = 4u + (uint32_t(w.token0 & 127) >> 5), sf_end = (uint32_t(w.token0) & 127u) + uint32_t(w.n);
        const bool two_atoms = WIDE ? sf_end > 128 : w.n > 128;
        uint32_t accumulate = 0;
        int step = step_begin;
        for (; step < step_end; ++step) {
          const int nkb = min(2, p.kblocks - 2 * step);
          if (!warp_wait(full_bar(stage), phase, abort_flag)) { error = kErrMmaFull; break; }
          // the quantisers write codes and scales through the generic proxy; the tensor core reads through the async proxy
          if (FUSED) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          tc_fence_after();
#ifdef HG_TRACE
          if (lane == 0 && it == 0 && step == step_begin) HG_STAMP(3);
#endif
          if (elect_one()) {
            const uint32_t a_lo = a_desc + uint32_t(stage) * a_stage - uint32_t(w.first) * 8u, b_lo = b_desc + uint32_t(stage) * b_stage;
            const uint32_t sfa_lo = sfa_desc + uint32_t(stage) * 64u, sfb_lo = sfb_desc + uint32_t(stage) * sfb_stage;
#pragma unroll
            for (uint32_t i = 0; i < 2; ++i) {
              if (i == 1 && nkb == 1) break;
              const uint32_t sf = sf0 + i * kScaleStride;
              cg_cp_scales<PAIR>(sf, desc_of(sfa_lo + i * 32u, kDescScales));
              cg_cp_scales<PAIR>(sf + 4, desc_of(sfb_lo + i * 32u, kDescScales));
              if (two_atoms) {
                cg_cp_scales<PAIR>(sf + 8, desc_of(sfb_lo + i * 32u + 64u, kDescScales));
                if (WIDE && sf_end > 256) cg_cp_scales<PAIR>(sf + 12, desc_of(sfb_lo + i * 32u + 128u, kDescScales));
              }
#pragma unroll
              for (uint32_t j = 0; j < 4; ++j)
                cg_mma<PAIR>(tmem_d, desc_of(a_lo + i * a_block + 2 * j, kDescTile), desc_of(b_lo + i * b_block + 2 * j, kDescTile),
                             idesc | (j << 29) | (j << 4), i + j > 0 ? 1u : accumulate, sf, sf + sfb_col);
            }
            cg_commit<PAIR>(empty_bar(stage), pair_mask);
          }
          __syncwarp();
          accumulate = 1;
          if (++stage == p.stages) { stage = 0; phase ^= 1u; }
        }
        if (error) break;
        issued += min(2 * step, p.kblocks) - 2 * step_begin;   // as far as the loop came
        if (p.ring_exchange && elect_one()) cg_commit_to<PAIR>(red_empty, uint16_t((1u << cluster_ctas) - 1u));
        __syncwarp();
        if (elect_one()) cg_commit<PAIR>(acc_full_bar(acc), pair_mask);
        __syncwarp();
#ifdef HG_TRACE
        if (lane == 0 && it < 4) HG_STAMP(4 + it);
#endif
      }
      // A pair's MMA works on a tile of each CTA.  (Added inside the loop, and after the drain, a block at 16 tokens took 0.6 % longer.)
      if (lane == 0 && issued) atomicAdd(p.status + 1, issued * PAIR);
      // Every MMA of this CTA (pair) retires before TMEM is released.
      if (elect_one()) cg_commit<PAIR>(drain_bar, pair_mask);
      __syncwarp();
      if (!warp_wait(drain_bar, 0, abort_flag) && !error) error = kErrDrain;
      // The other CTA's epilogues arrive here also for units that do not follow: this CTA stays until they have.
      if (PAIR == 2)
        for (int n = it; p.split == 1 && n <= it + (p.overlap ? 0 : 1) && !error; ++n)
          if (!acc_free(n)) error = kErrDrain;
    } else if (PAIR == 2) {
      // ---------------------------------------------------------------- second CTA of a pair: wait for the last MMA
      if (!warp_wait(drain_bar, 0, abort_flag) && !error) error = kErrDrain;
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int quarter = warp & 3, side = (warp - 2) >> 2;   // TMEM lanes this warp may read; which of the two warps of the quarter
    const int row_in_tile = quarter * 32 + lane;
    const uint32_t lane_addr = uint32_t(quarter * 32) << 16;
    int it = 0, stored = 0;
    pdl_wait();   // nothing is written to global memory before every earlier kernel has finished
    char* const out = out_base(p.out);
    const bool out_f32 = p.out.f32 != 0;
    const int row_bytes = p.outputs * (out_f32 ? 4 : 2);
    const uint32_t leader = uint32_t(rank & ~(PAIR - 1));
    for (int u = cluster, turn = 0; u < units; next_unit(p, u, turn), ++it) {
      const Unit w = unit_at<WIDE>(p, u, cluster, turn);
      const int acc = it & 1;
      const int row = (w.atom * PAIR + half) * kTileRows + row_in_tile;
      const bool active = quarter * 32 >= w.first && quarter * 32 < w.last;   // this quarter's rows belong to the tile
      const bool row_ok = active && row < p.rows[w.part];
      const int channel = row_ok ? p.ids[w.part][row] : 0;   // fetched while the main loop runs
      const int valid = min(w.n, p.tokens - w.token0);
      char* const out_row = out + int64_t(channel) * (out_f32 ? 4 : 2) + int64_t(w.token0) * row_bytes;
      if (!warp_wait(acc_full_bar(acc), uint32_t(it >> 1) & 1u, abort_flag)) { error = kErrEpilogue; break; }
      tc_fence_after();
      if (threadIdx.x == 64 && it < 3) HG_STAMP(8 + 2 * it);
      const uint32_t taddr = tmem_base + lane_addr + uint32_t(acc * p.acc_shift);
      auto release = [&](int which) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (PAIR == 1) mbar_arrive(acc_empty_bar(which));
          else arrive_remote_relaxed(map_to_rank(acc_empty_bar(which), leader));
        }
      };
      // N columns of this thread's row from column c on.
      auto store = [&](int c, const auto& v) {
        constexpr int N = sizeof(v) / sizeof(float);
        char* at = out_row + int64_t(row_bytes) * c;
        const int left = valid - c;
        if (!row_ok) return;
        if (!out_f32 && left >= N) {
#pragma unroll
          for (int i = 0; i < N; ++i) *reinterpret_cast<uint16_t*>(at + int64_t(row_bytes) * i) = from_float<T>(v[i]);
        } else if (!out_f32) {
#pragma unroll
          for (int i = 0; i < N; ++i)
            if (i < left) *reinterpret_cast<uint16_t*>(at + int64_t(row_bytes) * i) = from_float<T>(v[i]);
        } else {
#pragma unroll
          for (int i = 0; i < N; ++i)
            if (i < left) *reinterpret_cast<float*>(at + int64_t(row_bytes) * i) = v[i];
        }
      };

      if (p.split > 1) {
        // Every slice owns 2^share_log groups of four columns.  A partial goes straight to the shared memory of the slice
        // that owns its group (lanes write 512 contiguous bytes), one hop; the owner adds the pieces in K order.
        // In the ring: every slice's last commit tells all the others that its MMAs, and with them its ring, are done.
        if (p.ring_exchange && !warp_wait_cluster(red_empty, 0, abort_flag)) { error = kErrEpilogue; break; }
        const uint32_t share = 1u << p.share_log;
        const uint32_t my_piece = base + lay.red + (uint32_t(slice) << (p.share_log + 11)) + uint32_t(row_in_tile) * 16u;
        const int groups = (valid + 3) >> 2;
        const int g_begin = slice << p.share_log, g_end = min(groups, (slice + 1) << p.share_log);
        // st.async saves a round trip (the release of the stores before an arrival; 0.5 us), but counts every 16 bytes on the
        // barrier one after the other: beyond 32 columns plain stores and one arrival per warp are faster (o_proj at 128
        // tokens, K in two: 8.5 us against 10.4).
        if (p.async_push && threadIdx.x == 64) mbar_expect_tx(red_full, uint32_t(max(0, g_end - g_begin) * p.split * (w.last - w.first)) * 16u);
        for (int g0 = 4 * side; g0 < groups && active; g0 += 4 * kSides) {
          uint32_t r[16];
          tc_load16(taddr + uint32_t(g0) * 4u, r);
          tc_wait_ld();
#pragma unroll
          for (uint32_t i = 0; i < 4; ++i) {
            const uint32_t g = uint32_t(g0) + i;
            const uint32_t owner = (g >> p.share_log) * PAIR + uint32_t(half);
            const uint32_t to = map_to_rank(my_piece + ((g & (share - 1u)) << 11), owner);
            if (!p.async_push) store_remote(to, tc_loaded(r[4 * i]), tc_loaded(r[4 * i + 1]), tc_loaded(r[4 * i + 2]), tc_loaded(r[4 * i + 3]));
            else if (int(g) < groups)
              store_async(to, map_to_rank(red_full, owner), tc_loaded(r[4 * i]), tc_loaded(r[4 * i + 1]), tc_loaded(r[4 * i + 2]), tc_loaded(r[4 * i + 3]));
          }
        }
        // A cluster that splits K has one unit, and nobody waits for the accumulator.  Single CTAs hand it back all the same: without
        // that layer calls of 23 shapes take 0.3 % longer on average (1214 x 896 at 46 tokens 4.46 -> 4.54 us, 4608 x 3584 at 16 5.87 ->
        // 5.96) and the GEMM alone the same; the cause is not known.
        if constexpr (PAIR == 1) release(acc);
        else __syncwarp();   // an arrival releases what the whole warp stored
        if (!p.async_push && lane < p.split) arrive_remote(map_to_rank(red_full, uint32_t(lane * PAIR + half)));
        if (!warp_wait_cluster(red_full, 0, abort_flag)) { error = kErrEpilogue; break; }
        const uint32_t pieces = base + lay.red + uint32_t(row_in_tile) * 16u;
        for (int g = g_begin + side; g < g_end && active; g += kSides) {
          const uint32_t from = pieces + (uint32_t(g - g_begin) << 11);
          float v[8][4];
#pragma unroll
          for (int s = 0; s < 8; ++s)
            if (s < p.split)
              asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[s][0]), "=f"(v[s][1]), "=f"(v[s][2]), "=f"(v[s][3])
                           : "r"(from + (uint32_t(s) << (p.share_log + 11))) : "memory");
#pragma unroll
          for (int s = 1; s < 8; ++s)
            if (s < p.split) {
#pragma unroll
              for (int i = 0; i < 4; ++i) v[0][i] += v[s][i];
            }
          store(4 * g, v[0]);
        }
      } else {
        // This warp's groups of sixteen columns, the TMEM read of the next one in flight while the current one is stored.
        // The columns two accumulators share are drained first and handed to the next main loop.
        const int chunks = active ? (w.n + 15) >> 4 : 0;
        const int begin = p.overlap && acc == 0 && 14 + side < chunks ? 14 + side : side;   // column 224 of accumulator 0 is column 0 of accumulator 1
        bool hand_over = p.overlap;
        if (hand_over && acc == 0 && begin != 14 + side) { release(1); hand_over = false; }
        uint32_t a[16];
        int c = begin;
        if (c < chunks) tc_load16(taddr + uint32_t(c) * 16u, a);
        while (c < chunks) {
          tc_wait_ld();
          float r[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) r[i] = __uint_as_float(tc_loaded(a[i]));
          if (hand_over) { release(acc ^ 1); hand_over = false; }
          // 14 + side comes first where it is shared, then side, side + 2, ...
          int next = begin > side && c == begin ? side : c + kSides;
          if (begin > side && next == begin) next = chunks;
          if (next < chunks) tc_load16(taddr + uint32_t(next) * 16u, a);
          store(16 * c, r);
          c = next;
        }
        if (hand_over) release(acc ^ 1);
        if (!p.overlap) release(acc);
      }
      if (threadIdx.x == 64 && it < 3) HG_STAMP(9 + 2 * it);
      ++stored;
    }
    // One warp speaks for the CTA's: an accumulator is only free for the next unit once all of them have arrived.  (Counted over all
    // warps in shared memory, a block took 1 % longer at 16 tokens, 2 % at 37.)
    if (threadIdx.x == 64 && stored) atomicAdd(p.status + 2, stored);
  }

  auto settle = [] {   // time for everything in flight to land
    const long long start = clock64();
    while (clock64() - start < 400000ll) __nanosleep(1000);
  };
  if (error) {
    *abort_flag = 1;
    atomicCAS(p.status, 0, error * 1000000 + int(blockIdx.x));
    settle();   // copies and MMAs, before shared memory and TMEM are released
  }
  tc_fence_before();
  __syncwarp();
  // No CTA leaves while another may still write its shared memory or arrive on its barriers.  All that was sent has been waited for
  // where it arrives, so the barrier needs no release, which would wait for the stores to global memory; the end of the grid does.
  // Not so where a wait ran out: what this CTA sent is covered by its release, and what the others still sent to it, whose
  // arrival says nothing about their stores, gets time to land once they have all arrived.
  if (cluster_ctas > 1) {
    if (error) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    else asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (error) settle();
  } else {
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    cg_dealloc<PAIR>(tmem_base, p.tmem_cols);
  }
}

}  // namespace

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------

static int tuning(const char* name, int value) {
  const char* text = std::getenv(name);
  return text ? std::atoi(text) : value;
}

// Estimated microseconds of a launch, up to what all plans of a shape share.  A K256 step of a CTA takes the longest of: the
// tensor core with its operand reads from shared memory; a turn of the ring (from commit to the next full stage); what L2
// delivers, over all SMs and to one.  An SM stores 1.4 sectors per cycle: 128 rows of an MXFP4 tile touch 13 sectors per token,
// 128 rows of an MXFP8 tile 128, so an MXFP8 tile of 256 tokens is stored for 13 us.  Finer MXFP8 tiles spread that over more
// CTAs (qkv of Qwen2.5-7B: 24.8 -> 17.5 us at 777 tokens, 46.7 -> 37.5 us at 2048).  Stores run under the next main loop.  The
// launch takes the busiest cluster's time, plus a little per CTA and the exchange of partials; prefill also no less than its
// weights' time from HBM.  (In decode the busiest cluster's L2 reads hold the weights already; a bound there decided none of 24000
// shapes.)
//
// The constants are weights of a fit to the order of measured launches, every plan a shape can have, for shapes drawn from 640 to
// 38000 channels and K 512 to 18944; a rate among them need not be one that a unit of the chip has.  Prefill: layer calls
// (quantiser and GEMM), 7236 shapes of 129 to 4096 tokens, up to 25 plans of each, 70 % of the shapes fitted to and the rest checked: the
// plan preferred is 0.7 % slower than the best one of the shape on average (0.4 % up to 256 tokens, 0.7 % up to 512, 1.2 % from 1025
// on), and 1.0 % of the shapes are more than 5 % slower than with steps of 128 and 256 tokens and the constants for those (1.3 %
// faster on average).  Constants fitted to the GEMM alone, in graphs so short that a replay's steps of 2 us blurred small layers, and
// then edited for one layer preferred plans 1.0 % slower than the best (1024 x 4096 at 174 tokens in two parts of K 8.9 us, in four 8.3);
// 2.8 % of the shapes lost more than 5 %.  Up to 128 tokens: layer calls
// (quantiser and GEMM) back to back, 2400 shapes, of which every fourth or so was fitted to and the rest checked: 0.9 % slower than the
// best up to 64 tokens (1.9 % with constants fitted to the GEMM alone) and 1.1 % from 65 on (1.5 %; 10 % when two tiles of 64
// tokens were no choice).  Up to twelve layers took turns there, so weights of less than about 10 MB stayed in L2.  Checked since on
// 905 other layers of up to 12000 channels with all their weights cold: 1.8 % and 2.3 % (the same layers with weights in L2 1.6 %
// and 1.9 %).  Behind a kernel that has just written the activations and does not release its dependents early (an elementwise
// kernel of torch was measured) small layers at few tokens want fewer CTAs than back to back: 2009 x 640 at 14 tokens takes 5.98
// us with 34 CTAs, that kernel included, and took 5.82 with 19 (back to back 3.77 and 4.28).  Over 110 layers such calls took
// 5.4 % less than with the constants and kernels before.
struct PlanFit {
  double mma_floor, mma;                             // cycles of a single CTA's narrow MMA with its operand reads; factor on the time of every MMA
  double turn, l2, l2_wide, to_one;                  // us per turn of the ring; bytes per ns from L2 to all SMs, tiles of 129 tokens and more, to one
  double unit, split_unit, split_token;              // after a unit's main loop, whole or one of several parts of K; per token
  double store, store_token, low_row, high_row;      // stores: start; per token; cycles per token and row
  double hops, exchange, part, part_token;           // exchange: per doubling of the cluster, constant, per part, per part and token
  double cta, pair, cut, finer, hbm;                 // per CTA of the grid, paired CTAs, cut of all tiles, further cut of MXFP8 tiles; bytes per ns (0: no bound)
};
constexpr PlanFit kDecodeFit{234.0, 1, 1.313, 12213, 12213, 189.6, 0.09482, 0.5133, 0.0314, 1.07, 0.01755, 0.02057, 0.9327, -0.657, 0.1007, 0.0143, 0.005931,
                             0.008127, 0.5955, -0.0378, 0.268, 0};
constexpr PlanFit kWideDecodeFit{236.7, 1, 1.328, 12840, 12840, 250.0, 0.2656, 0.7058, 0.02462, 0.3386, 0.01767, 0.01224, 0.9089, -0.538, 0.1856, 0.06477, 0.003302,
                                 0.01379, 0.5441, -0.02387, 0.2337, 0};
constexpr PlanFit kPrefillFit{234, 1.357, 1.571, 26230, 10420, 119.2, 0.5252, 0.5565, 0.02775, 0.3909, 0.01591, 0.01591, 0.7769, -0.6515, -0.6216, 0.03302,
                              0.006075, 0.007576, 2.55, 0.0711, 0.09681, 5156};

// `reject`: a plan that costs this much or more may be given any cost from there on.
static double plan_cost(const ClusterPlan& plan, int units, int kblocks, double weight_kilobytes, double reject) {
  const int columns = (plan.token_tiles - 1) * plan.n_step + plan.n_tail;
  const PlanFit& fit = columns <= 64 ? kDecodeFit : columns <= 128 ? kWideDecodeFit : kPrefillFit;
  const double steps = double((kblocks + 1) / 2) / plan.split;
  const int cluster_ctas = plan.pair * plan.split, ctas = plan.clusters * cluster_ctas;
  auto main_loop = [&](int n, bool high) {
    const double b = double(n) / plan.pair;
    const double mma = 2 * (plan.pair == 2 ? std::max(2.0 * n, 200.0 + b) : std::max(171.0, fit.mma_floor + 1.3 * b)) / 1900 * fit.mma;
    auto bytes = [&](int part) { return 1000 * (double(kTileRows >> plan.cut_log[part]) * (part ? 0.25 : 0.125) + b * 0.25 + 2); };
    const double average = (bytes(0) * plan.tiles[0] + bytes(1) * plan.tiles[1]) / (double(plan.tiles[0]) + plan.tiles[1]);
    const double step = std::max({mma, fit.turn / plan.stages, average * ctas / (1000 * (n > 128 ? fit.l2_wide : fit.l2)), bytes(high) / (1000 * fit.to_one)});
    return steps * step + (plan.split > 1 ? fit.split_unit + fit.split_token * n : fit.unit);
  };
  auto stores = [&](int n, bool high) {
    const double rows = double(kTileRows >> plan.cut_log[high]);
    return fit.store + std::max(fit.store_token * n, n * rows * (high ? fit.high_row : fit.low_row) / 1900) / plan.split;
  };
  const double main_of[2][2] = {{main_loop(plan.n_step, false), main_loop(plan.n_tail, false)},
                                {plan.tiles[1] ? main_loop(plan.n_step, true) : 0, plan.tiles[1] ? main_loop(plan.n_tail, true) : 0}};
  const double store_of[2][2] = {{stores(plan.n_step, false), stores(plan.n_tail, false)}, {stores(plan.n_step, true), stores(plan.n_tail, true)}};
  double exchange = 0;
  if (plan.split > 1)
    exchange = fit.hops * std::log2(double(cluster_ctas)) + fit.exchange + (fit.part + fit.part_token * plan.n_tile) * plan.split;
  const double least = fit.hbm ? weight_kilobytes / fit.hbm + store_of[0][1] : 0;
  auto total = [&](double busiest) {
    return fit.cta * ctas + (plan.pair == 2 ? fit.pair : 0) + fit.cut * plan.cut_log[0] + fit.finer * (plan.cut_log[1] - plan.cut_log[0]) +
           std::max(busiest, least) + exchange;
  };
  // Cluster 0 has the most units, and no plan is done before an average cluster's main loops and the last one's stores are, or before
  // an average cluster's stores and the main loop of the first ones are.  (The margin is far above the rounding of the sums below.)
  const int most = (units + plan.clusters - 1) / plan.clusters;
  double main_least = 1e30, main_all = 0, store_least = 1e30, store_all = 0;
  for (int part = 0; part < 2; ++part)
    if (plan.tiles[part]) {
      main_least = std::min({main_least, main_of[part][0], main_of[part][1]});
      store_least = std::min({store_least, store_of[part][0], store_of[part][1]});
      main_all += plan.tiles[part] * ((plan.token_tiles - 1) * main_of[part][0] + main_of[part][1]);
      store_all += plan.tiles[part] * ((plan.token_tiles - 1) * store_of[part][0] + store_of[part][1]);
    }
  const double soonest = std::max(std::max(most * main_least, main_all / plan.clusters) + store_least, main_least + store_all / plan.clusters);
  if (const double bound = total(soonest * (1 - 1e-9)); bound >= reject) return bound;

  // End of a cluster's main loops and of its stores.  Two accumulators: a main loop starts once the stores before the last ones are done.
  struct Ends { double main = 0, stores = 0; };
  auto add = [&](Ends& ends, bool high, bool tail) {
    ends.main = std::max(ends.main + main_of[high][tail], ends.stores);
    ends.stores = ends.main + store_of[high][tail];
  };
  double busiest = 0;
  if (plan.token_tiles == 1) {
    // MXFP8 tiles come first, so clusters differ only in how many units of each kind they have: the first ones may have one more.
    for (const int cluster : {0, plan.tiles[1] % plan.clusters, units % plan.clusters}) {
      Ends ends;
      for (int u = cluster; u < units; u += plan.clusters) add(ends, u < plan.tiles[1], true);
      busiest = std::max(busiest, ends.stores);
    }
  } else {
    std::vector<Ends> ends(size_t(plan.clusters));
    const int tiles = plan.tiles[0] + plan.tiles[1];
    const double enough = (reject - total(0) + least) * (1 + 1e-9);   // a cluster that is busy for so long decides against the plan
    int cluster = 0, round = 0;   // of the next unit; see unit_at
    int spread = 0;               // how far the running share of MXFP8 tiles is beyond the last whole one
    for (int t = 0; t < tiles; ++t) {
      spread += plan.tiles[1];
      const bool high = spread >= tiles;
      if (high) spread -= tiles;
      const int last = plan.token_tiles - 1 - (plan.turned ? round % plan.token_tiles : 0);
      for (int tt = 0; tt < plan.token_tiles; ++tt) {
        Ends& e = ends[size_t(cluster)];
        add(e, high, tt == last);
        busiest = std::max(busiest, e.stores);
        if (++cluster == plan.clusters) { cluster = 0; ++round; }
      }
      if (busiest >= enough) return total(busiest);
    }
  }
  return total(busiest);
}

// Ring, TMEM and shared-memory figures that follow from the other choices.  False when the ring would be too shallow.
static bool finish_plan(ClusterPlan& plan, int most_stages) {
  const int n_cols = (plan.n_tile + 31) & ~31;
  plan.overlap = plan.n_tile > 224 ? 1 : 0;
  plan.acc_shift = plan.overlap ? 224 : n_cols;
  const int cols = plan.acc_shift + n_cols + int(2 * kScaleStride);
  plan.tmem_cols = 64;
  while (plan.tmem_cols < cols) plan.tmem_cols *= 2;
  plan.slot_rows = kTileRows >> std::min(plan.cut_log[0], plan.cut_log[1]);
  plan.least_rows = kTileRows >> std::max(plan.cut_log[0], plan.cut_log[1]);
  for (plan.stages = most_stages; plan.stages >= 2; --plan.stages) {
    plan.smem_bytes = 1024 + int(cluster_smem(plan.stages, plan.n_tile, plan.sf_atoms, plan.pair, plan.split, plan.slot_rows, plan.least_rows, plan.ring_exchange).end);
    if (plan.smem_bytes <= kMaxSmem) return true;
  }
  return false;
}

// Token tiles of a prompt: `count` of them, `step` tokens each, the last one holding what is left (`tail`, in MMA columns).
struct TokenTiles { int step, count, tail, sf_atoms; };

// Steps of 128, 256 and 192 tokens, and those of 128 and 192 with a short last tile joined to the one before it, so that the tiles of a
// ragged prompt fit the clusters: 37888 x 3584 at 160 tokens in one tile 31.5 -> 25.0 us, at 300 in 192 + 108 48.9 -> 45.0, 3584 x
// 18944 at 777 in 3 x 192 + 201 54.4 -> 49.4, 4608 x 3584 at 2048 by steps of 192 36.1 -> 31.8.  hg_plan tells its callers the
// widest tile, of which a prompt has ceil(tokens / widest): joined tails that would need a tile more are left out (beyond 1376 tokens
// all of them).  Each split is listed once: a search walks it in up to 15 ways, and every new length of a prompt pays for one search per
// layer.
static int token_tiles_of(int tokens, TokenTiles (&ways)[5]) {
  int n = 0;
  for (const int way : {128, 256, 192, -128, -192}) {
    TokenTiles t;
    t.step = std::abs(way);
    t.count = way < 0 ? tokens / t.step : (tokens + t.step - 1) / t.step;
    if (t.count < 1) continue;
    t.tail = (tokens - (t.count - 1) * t.step + 31) / 32 * 32;
    if (t.tail > 256) continue;
    if (t.count == 1) t.step = t.tail;
    const int widest = std::max(t.step, t.tail);
    if ((tokens + widest - 1) / widest != t.count) continue;
    // Atoms that the last tile and the first ones touch; a second one may start in the middle of its first.
    const int last_start = (t.count - 1) * t.step % 128, odd_start = t.count > 2 ? t.step % 128 : 0;
    t.sf_atoms = std::max(last_start + t.tail + 127, t.count > 1 ? odd_start + t.step + 127 : 0) / 128;
    bool listed = false;
    for (int i = 0; i < n; ++i) listed |= ways[i].step == t.step && ways[i].count == t.count;
    if (!listed) ways[n++] = t;
  }
  return n;
}

ClusterPlan make_cluster_plan(int lo, int hi, int tokens, int k, const int max_clusters[4]) {
  const int kblocks = k / kTileK, steps = (kblocks + 1) / 2;
  const int atoms[2] = {(lo + kTileRows - 1) / kTileRows, (hi + kTileRows - 1) / kTileRows};
  ClusterPlan best;
  best.cost = 1e30;
  const int force_split = tuning("HYGEMM_CL_SPLIT", 0), force_pair = tuning("HYGEMM_CL_PAIR", 0), force_n = tuning("HYGEMM_CL_N", 0);
  const int force_cut = tuning("HYGEMM_CL_CUT", -1), force_cut_high = tuning("HYGEMM_CL_CUT_HIGH", -1);
  TokenTiles ways[5];
  const int n_ways = tokens <= 128 ? 2 : token_tiles_of(tokens, ways);
  const int most_stages = std::min(kClusterMaxStages, tuning("HYGEMM_CL_STAGES", kClusterMaxStages));
  for (int pair = 1; pair <= 2; ++pair)
    for (int log = pair - 1; log < 4; ++log)
      for (int cut = 0; cut < 3; ++cut)
        for (int more = 0; more < 3; ++more)
          for (int way = 0; way < n_ways; ++way) {
              ClusterPlan plan;
              plan.pair = pair;
              plan.split = (1 << log) / pair;
              plan.cut_log[0] = cut;
              plan.cut_log[1] = cut + more;
              if (plan.split > steps || cut + more > 2 || max_clusters[log] < 1) continue;
              if (tokens <= 128) {
                // From 65 tokens on also two tiles of 64: twice the CTAs with half the accumulators each, for a second read of the
                // weights from L2.  Layers with few row tiles gain (128 tokens: 4608 x 3584 8.8 -> 7.7 us, 4096 x 1024 5.8 -> 4.2, 7003 x 2432
                // at 77 tokens 7.3 -> 6.7), wide and long ones do not (37888 x 3584 23.7 -> 27.0, 3584 x 18944 16.1 -> 17.1).
                if ((way && tokens <= 64) || (!way && tokens > 64 && pair == 1) || (tokens <= 32 && pair == 2)) continue;   // (fused quantisation: single CTAs)
                plan.token_tiles = way ? 2 : 1;
                plan.n_tail = (tokens - 64 * way + 16 * pair - 1) / (16 * pair) * (16 * pair);
                plan.n_step = way ? 64 : plan.n_tail;
                plan.n_tile = std::max(plan.n_step, plan.n_tail);
                plan.sf_atoms = 1;
              } else {
                if (pair == 1 || cut) continue;
                const TokenTiles& t = ways[way];
                plan.token_tiles = t.count;
                plan.n_step = t.step;
                plan.n_tail = t.tail;
                plan.n_tile = std::max(t.step, t.tail);
                plan.sf_atoms = t.sf_atoms;
                if (plan.n_tile > 224 && plan.split > 1) continue;
              }
              if ((force_split && plan.split != force_split) || (force_pair && pair != force_pair) || (force_n && plan.n_tile != force_n) ||
                  (force_cut >= 0 && cut != force_cut) || (force_cut_high >= 0 && cut + more != force_cut_high))
                continue;
              for (int i = 0; i < 2; ++i) plan.tiles[i] = ((atoms[i] + pair - 1) / pair) << plan.cut_log[i];
              const int64_t units = int64_t(plan.tiles[0] + plan.tiles[1]) * plan.token_tiles;
              plan.clusters = int(std::min<int64_t>(max_clusters[log], units));
              // With several units to a cluster every exchange would stall the next main loop (gate_up at 16 tokens, K in
              // two: 19.8 us against 15.4).
              if (plan.split > 1 && units > plan.clusters) continue;
              plan.turned = tokens > 128 && 4 * plan.n_tail <= 3 * plan.n_step && units > plan.clusters && plan.clusters >= plan.token_tiles &&
                            std::gcd(plan.clusters, plan.token_tiles) > 1;
              // Worth its extra hop (about 0.4 us) where the exchange buffer would take a stage from the ring (down_proj at 128
              // tokens 17.1 -> 16.0 us).
              plan.ring_exchange = plan.split > 1 && plan.n_tile > 32;
              if (!finish_plan(plan, most_stages)) continue;
              plan.wide = plan.turned || (tokens > 128 && plan.token_tiles > 1 && (plan.n_step % 128 || plan.n_tail > plan.n_step));
              // Of the same fit; what its colder code costs is in there.
              const double margin = plan.wide ? 1.01 : 1, start = plan.wide ? -0.073 : 0;
              plan.cost = margin * plan_cost(plan, int(units), kblocks, (lo * 0.53125 + hi * 1.03125) * k * 1e-3, (best.cost - start) / margin) + start;
              if (plan.cost < best.cost) best = plan;
            }
  if (best.cost >= 1e30) throw std::runtime_error("No cluster schedule for this shape");
  return best;
}

template <typename T, int PAIR, bool FUSED, bool WIDE = false>
static void set_limits() {
  check(cudaFuncSetAttribute(cluster_gemm_kernel<T, PAIR, FUSED, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem), "cudaFuncSetAttribute");
}

void configure_cluster_kernels() {
  set_limits<__nv_bfloat16, 1, false>(); set_limits<__nv_bfloat16, 1, true>(); set_limits<__nv_bfloat16, 2, false>(); set_limits<__nv_bfloat16, 2, false, true>();
  set_limits<__half, 1, false>(); set_limits<__half, 1, true>(); set_limits<__half, 2, false>(); set_limits<__half, 2, false, true>();
}

void cluster_kernel_attributes(const ClusterPlan& plan, int dtype, int* registers, int* local_bytes, int* stage_bytes) {
  cudaFuncAttributes attr{};
  const bool bf16 = dtype == HG_DTYPE_BF16;
  auto get = [&](auto wide_kernel, auto pair_kernel, auto kernel) {
    check(cudaFuncGetAttributes(&attr, plan.wide ? wide_kernel : plan.pair == 2 ? pair_kernel : kernel), "cudaFuncGetAttributes");
  };
  if (bf16) get(cluster_gemm_kernel<__nv_bfloat16, 2, false, true>, cluster_gemm_kernel<__nv_bfloat16, 2, false, false>, cluster_gemm_kernel<__nv_bfloat16, 1, false, false>);
  else get(cluster_gemm_kernel<__half, 2, false, true>, cluster_gemm_kernel<__half, 2, false, false>, cluster_gemm_kernel<__half, 1, false, false>);
  *registers = attr.numRegs;
  *local_bytes = int(attr.localSizeBytes);
  const ClusterSmem lay = cluster_smem(plan.stages, plan.n_tile, plan.sf_atoms, plan.pair, plan.split, plan.slot_rows, plan.least_rows, plan.ring_exchange);
  *stage_bytes = int(2 * lay.b_tile + 1024 + lay.sfb_stage);
}

const int* cluster_capacity() {
  static int capacity[64][4];
  static std::once_flag once[64];
  int device = 0;
  check(cudaGetDevice(&device), "cudaGetDevice");
  if (device < 0 || device >= 64) throw std::runtime_error("Device ordinals 0..63 are supported");
  std::call_once(once[device], [&] {
    configure_cluster_kernels();
    int sms = 0;
    check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "SM count");
    capacity[device][0] = sms;
    for (int log = 1; log < 4; ++log) {
      cudaLaunchConfig_t config{};
      config.gridDim = dim3(unsigned(sms >> log << log));
      config.blockDim = dim3(cluster_threads(2, false));
      config.dynamicSmemBytes = kMaxSmem;
      cudaLaunchAttribute attribute[1];
      attribute[0].id = cudaLaunchAttributeClusterDimension;
      attribute[0].val.clusterDim = {1u << log, 1u, 1u};
      config.attrs = attribute;
      config.numAttrs = 1;
      int clusters = 0;
      check(cudaOccupancyMaxActiveClusters(&clusters, cluster_gemm_kernel<__nv_bfloat16, 2, false, false>, &config), "cluster occupancy");
      capacity[device][log] = std::min(clusters, sms >> log);
    }
  });
  return capacity[device];
}

// Clusters of 1, 2, 4 and 8 CTAs on a device with `sms` SMs: what the current device holds if it has as many, else as many
// as fit if no SM were out of reach of a cluster.
static std::array<int, 4> capacity_for(int sms) {
  int devices = 0, device = 0, count = 0;
  if (cudaGetDeviceCount(&devices) == cudaSuccess && devices > 0 && cudaGetDevice(&device) == cudaSuccess &&
      cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) == cudaSuccess && count == sms) {
    const int* held = cluster_capacity();
    return {held[0], held[1], held[2], held[3]};
  }
  cudaGetLastError();   // no GPU: not this call's error
  return {sms, sms >> 1, sms >> 2, sms >> 3};
}

ClusterPlan make_cluster_plan_for(int lo, int hi, int tokens, int k, int sms) {
  return make_cluster_plan(lo, hi, tokens, k, capacity_for(sms).data());
}

template <typename T, int PAIR, bool FUSED, bool WIDE = false>
static cudaError_t launch(const ClusterPlan& plan, const ClusterParams& p, const ClusterMaps& maps, cudaStream_t stream, bool pdl) {
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(unsigned(plan.clusters * plan.pair * plan.split));
  config.blockDim = dim3(FUSED ? first_act_warp(PAIR) * 32 + (p.tokens + 1) / 2 * 32 : cluster_threads(PAIR, false));
  config.dynamicSmemBytes = size_t(plan.smem_bytes);
  config.stream = stream;
  cudaLaunchAttribute attribute[2];
  int count = 0;
  if (plan.pair * plan.split > 1) {
    attribute[count].id = cudaLaunchAttributeClusterDimension;
    attribute[count++].val.clusterDim = {unsigned(plan.pair * plan.split), 1u, 1u};
  }
  if (pdl && pdl_enabled()) {
    attribute[count].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[count++].val.programmaticStreamSerializationAllowed = 1;
  }
  config.attrs = attribute;
  config.numAttrs = unsigned(count);
  return cudaLaunchKernelEx(&config, cluster_gemm_kernel<T, PAIR, FUSED, WIDE>, p, maps);
}

// What follows from the plan and the shape alone.
static ClusterParams shape_params(const ClusterPlan& plan, int rows_low, int rows_high, int tokens, int k) {
  ClusterParams p{};
  const int rows[2] = {rows_low, rows_high};
  for (int i = 0; i < 2; ++i) { p.rows[i] = rows[i]; p.cut_log[i] = plan.cut_log[i]; p.tiles[i] = plan.tiles[i]; }
  p.slot_rows = plan.slot_rows; p.least_rows = plan.least_rows;
  p.tokens = tokens; p.k = k; p.kblocks = k / kTileK;
  p.n_step = plan.n_step; p.sf_atoms = plan.sf_atoms; p.turned = plan.turned;
  p.n_tile = plan.n_tile; p.n_tail = plan.n_tail; p.token_tiles = plan.token_tiles; p.stages = plan.stages;
  p.async_push = plan.n_tile <= 32;
  p.ring_exchange = plan.ring_exchange; p.split = plan.split; p.clusters = plan.clusters;
  while ((1 << p.split_log) < plan.split) ++p.split_log;
  p.share_log = share_log_of(plan.n_tile, plan.split);
  const uint64_t tiles = uint64_t(plan.tiles[0]) + uint64_t(plan.tiles[1]), most = uint64_t(1) << 40;
  auto inverse = [&](uint64_t n_max, uint64_t d) {
    const uint64_t inv = (most + d - 1) / d;
    return n_max < most / d && n_max < (uint64_t(1) << 63) / inv ? inv : uint64_t(0);
  };
  p.by_token_tiles = inverse(tiles * plan.token_tiles, uint64_t(plan.token_tiles));
  p.by_tiles = inverse((tiles + 1) * uint64_t(plan.tiles[1]), tiles);
  p.acc_shift = plan.acc_shift; p.overlap = plan.overlap;
  p.tmem_cols = uint32_t(plan.tmem_cols);
  return p;
}

std::vector<ClusterPart> cluster_parts(const ClusterPlan& plan, int rows_low, int rows_high, int tokens, int k) {
  const ClusterParams p = shape_params(plan, rows_low, rows_high, tokens, k);
  const int units = (p.tiles[0] + p.tiles[1]) * p.token_tiles, cluster_ctas = plan.pair * plan.split;
  std::vector<ClusterPart> parts;
  parts.reserve(size_t(units) * cluster_ctas);
  for (int cluster = 0; cluster < plan.clusters; ++cluster)
    for (int rank = 0; rank < cluster_ctas; ++rank)
      for (int u = cluster, turn = 0; u < units; next_unit(p, u, turn)) {
        const Unit w = plan.wide ? unit_at<true>(p, u, cluster, turn) : unit_at<false>(p, u, cluster, turn);
        const int half = rank % plan.pair, slice = rank / plan.pair, atom = w.atom * plan.pair + half, log = p.cut_log[w.part];
        ClusterPart part;
        part.cta = cluster * cluster_ctas + rank;
        part.tile = (w.part ? plan.pair * p.tiles[0] : 0) + (atom << log) + (w.first >> (7 - log));
        part.token_tile = w.token0 / p.n_step;
        part.kb_begin = 2 * first_step(p, slice);
        part.kb_end = std::min(2 * first_step(p, slice + 1), p.kblocks);
        part.slice = slice;
        part.first_row = atom * kTileRows + w.first;
        part.rows = std::max(0, std::min(kTileRows >> log, p.rows[w.part] - part.first_row));
        parts.push_back(part);
      }
  return parts;
}

void launch_cluster(const ClusterPlan& plan, const ClusterCall& call, const ClusterMaps& maps, cudaStream_t stream, bool pdl) {
  const hg_problem &l = *call.low, &h = *call.high, &any = l.rows ? l : h;
  ClusterParams p = shape_params(plan, l.rows, h.rows, any.tokens, any.k);
  const hg_problem* parts[2] = {&l, &h};
  for (int i = 0; i < 2; ++i) {
    p.sfa[i] = static_cast<const uint8_t*>(parts[i]->weight_scales);
    p.ids[i] = static_cast<const int32_t*>(parts[i]->ids);
  }
  p.sfb = static_cast<const uint8_t*>(any.activation_scales);
  p.out = call.out;
  p.outputs = any.outputs;
  p.x = static_cast<const uint16_t*>(call.x);
  p.x_bf16 = call.x_dtype == HG_DTYPE_BF16;
  p.status = call.status;
#ifdef HG_TRACE
  p.trace = call.trace;
#endif
  const bool bf16 = call.dtype == HG_DTYPE_BF16;
  cudaError_t e;
  if (call.x) e = bf16 ? launch<__nv_bfloat16, 1, true>(plan, p, maps, stream, pdl) : launch<__half, 1, true>(plan, p, maps, stream, pdl);
  else if (plan.pair == 1) e = bf16 ? launch<__nv_bfloat16, 1, false>(plan, p, maps, stream, pdl) : launch<__half, 1, false>(plan, p, maps, stream, pdl);
  else if (plan.wide) e = bf16 ? launch<__nv_bfloat16, 2, false, true>(plan, p, maps, stream, pdl) : launch<__half, 2, false, true>(plan, p, maps, stream, pdl);
  else e = bf16 ? launch<__nv_bfloat16, 2, false>(plan, p, maps, stream, pdl) : launch<__half, 2, false>(plan, p, maps, stream, pdl);
  check(e, "hybrid GEMM launch");
}

}  // namespace hg
