// Kernel argument block of the persistent walker (walker.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "geom.cuh"
#include "n2w.h"

namespace n2w {

constexpr int kOutStats = 0;    // per-point FP64 accumulators
constexpr int kOutSamples = 1;  // per-sample value / steps / flags (reference layout)
constexpr int kOutPrefix = 2;   // per-sample prefix records for the cache levels

constexpr int kWalkerMaxThreads = 256;
// Resident 256-thread blocks the register budget must allow (64 registers per
// thread): the traversal hides L1/L2 latency with warps, so occupancy matters.
constexpr int kWalkerMinBlocks = 4;
constexpr int kDefaultWalkerThreads = 128;
// Walks of one point that a lane takes from the queue at a time.  One: a launch
// ends when its slowest lane has finished its last chunk, and a chunk of k walks
// is a serial chain of k walks.  Chunk 8 / 4 / 2 / 1: 4.02 / 2.39 / 1.50 / 1.02 ms
// for 37 points x 64 walks, 21.9 / 19.5 / 18.3 / 17.7 ms for 20,011 x 101, 19.9 /
// 16.5 / 14.3 / 13.4 ms for a two-level estimate of 8,192 points; 366.4 / 364.7 /
// 364.6 / 365.0 ms for 40,000 x 1,024, where the tail no longer shows: the queue
// pops and per-point flushes of single walks cost nothing that can be measured.
constexpr int kDefaultChunk = 1;
// Waiting lanes that make a warp leave the traversal for the walk update: more
// lanes share the update, fewer traverse meanwhile.  8 / 12 / 14 / 16 / 20:
// 47.8 / 46.3 / 46.2 / 46.2 / 47.2 ms (Poisson slice, 5.1 M walks), 39.2 / 37.9 /
// 37.5 / 37.4 / 37.4 ms (batched instances); 16 samples per ball, 8 / 12 / 16 / 20:
// 16.5 / 15.7 / 15.3 / 15.5 ms.
constexpr int kDefaultRegen = 16;
// Source samples per ball from which a warp shares them (warp_ball_source).
constexpr int kManySamples = 4;

// One instance of a batched launch: its geometry inside the merged scene, its
// problem, its points and accumulators, and its slice of the global chunk queue.
struct alignas(16) BatchInst {
  const n2w_vec3* points;       // this instance's points
  const n2w_problem* problem;   // device copy of its problem
  double* sum;                  // per-point accumulators (local point index)
  double* sum_sq;
  uint32_t* count;
  uint64_t* steps;
  uint32_t* forced;
  int64_t point_base;           // first global point index (first-query cache)
  int64_t point_count;
  int64_t chunk_base;           // first global chunk of this instance
  int64_t chunks_per_point;
  dev::SeedGrid grid;           // cells already rebased into the merged scene
  float box_lo[3], box_hi[3];   // domain box (walks never leave it)
  int32_t walks_per_point;
  int32_t root;                 // root node of this instance's mesh in the scene
  uint32_t k0, k1;              // Philox key of the instance
  int32_t has_source, source_center, source_samples, pad;
  int64_t wid_base;             // added to every walk id (a point range of a larger request)
};

struct WalkArgs {
  const float4* nodes;  // FrameNode4 array
  const float4* boxes;  // Node4 array of the same tree, for first queries (batched launches: nullptr)
  const float4* tris;   // TriEdges array
  dev::SeedGrid grid;
  float box_lo[3], box_hi[3];  // domain box: the mesh box grown by 20 % (walks never leave it)
  const n2w_vec3* points;
  // Per-point first query (closest point + d2, id + slot): every walk of a
  // point starts with the same query, computed once by a pre-pass.
  const float4* first_cpd;
  const int2* first_ids;
  int64_t total_chunks;
  int64_t chunks_per_point;
  int walks_per_point;
  int chunk;
  int regen;  // waiting lanes that trigger the walk-update phase
  int lanes;  // lanes of a warp that take walks
  int max_steps;
  int depth_m;
  float eps;
  float step_scale;
  uint32_t k0, k1;
  int has_source;
  int source_center;
  int source_samples;  // points averaged per ball (>= 1)
  int first_boxes;     // first queries search `boxes` (n2w_bvh::use_boxes)
  int small_tree;      // nodes and triangles stay in L1 (fits_l1)
  int own_regen;       // regen is the caller's
  int warp_points;     // first queries of up to this many points run one to a warp (warp_query_limit)
  int64_t deadline_ns;
  n2w_problem problem;
  // kOutStats
  double* sum;
  double* sum_sq;
  uint32_t* count;
  uint64_t* steps;
  uint32_t* forced;
  // kOutSamples / kOutPrefix
  float* s_value;
  int* s_steps;
  int* s_forced;
  int* s_overflow;
  float* p_inputs;
  float* p_boundary;
  float* p_cont;
  uint8_t* p_needs;
  float in_min[3];
  float in_ext[3];
  // scratch
  unsigned long long* queue;
  n2w_walk_counters* counters;
  // batched launches: instance table sorted by chunk_base / point_base
  const BatchInst* insts;
  int n_insts;
};

dev::SeedGrid seed_grid_of(const n2w_bvh& b);
void validate_problem(const n2w_problem& p);
void validate_walk_options(const n2w_walk_options& o);

// Batched launches (walker.cu): per-point first queries of every instance, and
// the persistent walker over the concatenated chunk queue of all instances.
// reg_variant 0: 64 registers / 4 blocks per SM; 1: 80 registers / 3 blocks.
void launch_first_query_batch(const WalkArgs& a, int64_t total_points, float4* cpd, int2* ids, cudaStream_t s);
void launch_walker_batch(const WalkArgs& a, int block, int blocks_per_sm, int reg_variant, cudaStream_t s);
int walker_batch_occupancy(int block, int reg_variant);

}  // namespace n2w
