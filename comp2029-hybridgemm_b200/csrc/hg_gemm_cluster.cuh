// Host-side interface of the cluster GEMM (see hg_gemm_cluster.cu).
#pragma once
#include <cuda.h>

#include "hg_tcgen05.cuh"

namespace hg {

struct ClusterPlan {
  int pair = 1;            // CTAs that share one MMA tile: 1, or 2 (cta_group::2)
  int split = 1;           // slices of K per tile, one CTA (pair) of the cluster each
  int clusters = 0;        // persistent clusters of pair * split CTAs
  int n_tile = 0;          // tokens per tile
  int n_tail = 0;          // MMA columns of the last token tile
  int token_tiles = 0;
  int tile_rows[2] = {0, 0};   // weight rows per CTA tile of each partition, at most 128
  int tiles[2] = {0, 0};       // tiles (pair * tile_rows rows) of each partition
  int stages = 0;          // K256 stages of the ring
  int acc_shift = 0;       // TMEM columns between the two accumulators
  int overlap = 0;         // the accumulators share 32 columns (256-token tiles)
  int tmem_cols = 0;
  int smem_bytes = 0;
  double cost = 0;         // estimated cycles
};

// Plan for one shape; `max_clusters[i]` is the number of clusters of 2^i CTAs the device holds at once.
ClusterPlan make_cluster_plan(int rows_low, int rows_high, int tokens, int k, const int max_clusters[4]);

// What the device holds of clusters of 1, 2, 4 and 8 CTAs (one CTA per SM); queried once per device.
const int* cluster_capacity();

struct ClusterCall {
  const hg_problem* low;
  const hg_problem* high;
  const void* x;          // 16-bit activations to quantise in the kernel (at most 16 tokens), or null
  int x_dtype;
  OutTargets out;
  int dtype;              // output type
  int audit_tokens;       // tokens per tile of the schedule whose units the audit counters count
  int* status;
  unsigned long long* trace;
};
// `map_act`, `map_tail`: activation maps of boxes n_tile / pair and n_tail / pair rows (unused when `x` is set).
void launch_cluster(const ClusterPlan& plan, const ClusterCall& call, const CUtensorMap& map_act, const CUtensorMap& map_tail,
                    cudaStream_t stream, bool pdl);
void configure_cluster_kernels();

}  // namespace hg
