// Host-side interface of the cluster GEMM (see hg_gemm_cluster.cu).
#pragma once
#include <cuda.h>

#include "hg_tcgen05.cuh"

namespace hg {

struct ClusterPlan {
  int pair = 1;            // CTAs that share one MMA tile: 1, or 2 (cta_group::2)
  int split = 1;           // slices of K per tile, one CTA (pair) of the cluster each
  int clusters = 0;        // persistent clusters of pair * split CTAs
  int wide = 0;            // token tiles that only the kernel's WIDE instance takes
  int n_tile = 0;          // MMA columns of the widest token tile
  int n_step = 0;          // tokens of every token tile but the last
  int n_tail = 0;          // MMA columns of the last token tile; may be more than n_step
  int sf_atoms = 0;        // 128-token scale atoms that a token tile touches at most
  int turned = 0;          // rows of units start with another token tile each round over the clusters
  int token_tiles = 0;
  int cut_log[2] = {0, 0};     // each partition's 128-row atoms (pairs of atoms) are cut into 2^cut_log tiles
  int tiles[2] = {0, 0};       // tiles of each partition
  int slot_rows = 0, least_rows = 0;   // the taller and the shorter tile height; a ring slot holds the taller
  int ring_exchange = 0;       // partials are exchanged in the ring, idle by then
  int stages = 0;          // K256 stages of the ring
  int acc_shift = 0;       // TMEM columns between the two accumulators
  int overlap = 0;         // the accumulators share 32 columns (256-token tiles)
  int tmem_cols = 0;
  int smem_bytes = 0;
  double cost = 0;         // estimated microseconds
};

// Plan for one shape; `max_clusters[i]` is the number of clusters of 2^i CTAs the device holds at once.
ClusterPlan make_cluster_plan(int rows_low, int rows_high, int tokens, int k, const int max_clusters[4]);

// The same for a device with `sms` SMs; asks the current device if it has as many.
ClusterPlan make_cluster_plan_for(int rows_low, int rows_high, int tokens, int k, int sms);

// What one CTA does for one unit, CTA by CTA and in the order of its units.  The kernel's counters add kb_end - kb_begin and
// one per part.  Tiles are numbered through the partitions; `rows` is what is left of the tile's height at the end of one
// (0 in the second CTA of a pair whose atom is not there).
struct ClusterPart { int cta, tile, token_tile, kb_begin, kb_end, slice, first_row, rows; };
std::vector<ClusterPart> cluster_parts(const ClusterPlan& plan, int rows_low, int rows_high, int tokens, int k);

// What the device holds of clusters of 1, 2, 4 and 8 CTAs (one CTA per SM); queried once per device.
const int* cluster_capacity();

struct ClusterCall {
  const hg_problem* low;
  const hg_problem* high;
  const void* x;          // 16-bit activations to quantise in the kernel (at most 16 tokens), or null
  int x_dtype;
  OutTargets out;
  int dtype;              // output type
  int* status;
  unsigned long long* trace;
};
// Boxes: weights 128 >> cut_log rows x 2 K128 blocks; activations n_step / pair and, for the last token tile, n_tail / pair rows;
// scales (pairs only) 2 atoms.  Maps a launch does not use (an absent partition; activations quantised in the kernel) may
// be zeros.
struct ClusterMaps { CUtensorMap low, high, act, tail, low_scales, high_scales, act_scales; };
void launch_cluster(const ClusterPlan& plan, const ClusterCall& call, const ClusterMaps& maps, cudaStream_t stream, bool pdl);
void configure_cluster_kernels();
// Registers and local memory of the instance a plan launches on prepacked activations; bytes of activations and of all
// scales that a CTA brings in per K256 stage.
void cluster_kernel_attributes(const ClusterPlan& plan, int dtype, int* registers, int* local_bytes, int* stage_bytes);

}  // namespace hg
