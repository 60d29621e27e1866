// Host-side internals shared by the library's translation units.
#pragma once

#include <cuda_runtime.h>

#include <array>
#include <cstdint>
#include <stdexcept>
#include <string>
#include <vector>

#include "layout.h"
#include "n2w.h"

struct n2w_mesh {
  std::vector<std::array<float, 3>> vertices;
  std::vector<std::array<uint32_t, 3>> triangles;
  std::string name;
};

struct n2w_bvh {
  n2w::Node4* d_nodes = nullptr;         // axis-aligned boxes: ray parity, counted queries, the copied-out layout
  n2w::FrameNode4* d_frames = nullptr;  // the same tree with boxes in per-node frames: walks, most trees' queries
  n2w::TriRec* d_tris = nullptr;        // leaf-ordered triangles: ray parity, the copied-out layout
  n2w::TriEdges* d_edges = nullptr;     // the same triangles for the closest-point test
  int4* d_seed = nullptr;  // seed grid: nearest triangle's leaf slot and start subtrees per lattice node (geom.cuh)
  float seed_lo[3] = {0, 0, 0};
  float seed_h = 0.0f;
  int seed_n = 0;
  float seed_far = 0.0f;   // SeedGrid::far
  bool use_boxes = false;  // queries search d_nodes, not d_frames (choose_nodes)
  n2w_bvh_stats stats{};
  int device = 0;
};

namespace n2w {

class Error : public std::runtime_error {
 public:
  Error(int code, const std::string& msg) : std::runtime_error(msg), code_(code) {}
  int code() const { return code_; }

 private:
  int code_;
};

void set_last_error(const std::string& msg);

#define N2W_CUDA(expr)                                                                         \
  do {                                                                                         \
    cudaError_t err__ = (expr);                                                                \
    if (err__ != cudaSuccess) {                                                                \
      throw ::n2w::Error(N2W_ECUDA, std::string("CUDA error at ") + __FILE__ + ":" +          \
                                        std::to_string(__LINE__) + ": " +                      \
                                        cudaGetErrorString(err__));                            \
    }                                                                                          \
  } while (false)

#define N2W_REQUIRE(cond, msg)                        \
  do {                                                \
    if (!(cond)) throw ::n2w::Error(N2W_EINVAL, msg); \
  } while (false)

// Runs f, converting exceptions into status codes + last-error text.
template <typename F>
int guarded(F&& f) {
  try {
    f();
    return N2W_OK;
  } catch (const Error& e) {
    set_last_error(e.what());
    return e.code();
  } catch (const std::bad_alloc&) {
    set_last_error("host allocation failed");
    return N2W_ENOMEM;
  } catch (const std::exception& e) {
    set_last_error(e.what());
    return N2W_EINTERNAL;
  }
}

// ---- host BVH build (bvh_build.cpp) ----
struct TriRange {
  int32_t first, last;  // leaf-order triangles [first, last)
};
struct HostBvh {
  std::vector<Node4> nodes;
  std::vector<TriRange> ranges;  // triangles below each node
  std::vector<TriRec> tris;
  int64_t binary_nodes = 0;
  int64_t leaves = 0;
  int max_depth = 0;
  double sah_cost = 0.0;
};
HostBvh build_bvh4(const n2w_mesh& mesh, int leaf_size, const std::string& method);
n2w_bvh_stats host_stats(const HostBvh& h, int leaf_size, double ms);

// Launches of up to this many queries (or first queries of walks) give each a warp: with
// a lane per query a launch lasts as long as its slowest serial search, whatever its size,
// but a warp per query takes longer for queries that are short.  Lane / warp per query over
// the frames of 81,920 triangles: 8,000 uniform 128 / 32 us, 16,000 124 / 61, 32,768
// 140 / 99; near the surface 33 / 23, 35 / 39, 38 / 70.  Boxes, whose search wants an order
// that a warp's batches do not have, near an axis-aligned cube: 8,000 20 / 21, 16,000
// 21 / 32.  12 triangles: 8,000 around them 14 / 25.
// First queries over frames keep to warps for longer: their lanes have no budget to hand a
// long search off by (24,000 in a bumpy sphere of 65,024 triangles: 236 / 120 us).
inline int warp_query_limit(int64_t triangles, bool boxes, bool first_queries) {
  return triangles <= 32 ? 4096 : (boxes ? 8192 : (first_queries ? 32768 : 16384));
}

// ---- device query launch (closest_point.cu) ----
void launch_closest_point(const n2w_bvh& bvh, const n2w_vec3* d_points, const uint8_t* d_active,
                          int n, float* d_d2, n2w_vec3* d_cp, int* d_id, int* d_overflow,
                          int* d_nodes, int* d_tris, int block_size, cudaStream_t stream);

// Fills b.d_edges and b.d_frames from the uploaded nodes and triangles.
void build_edges(n2w_bvh& b, int64_t triangles);
void build_frames(n2w_bvh& b, const HostBvh& h);

// Fills the start subtrees of the seed grid's cells, whose slots are set.
void build_cell_entries(n2w_bvh& b);
// Host copy of the seed grid's n slots.
void copy_cell_slots(const n2w_bvh& b, int64_t n, int* out);

void build_seed_grid(n2w_bvh& b, const n2w_mesh& mesh, int n);

// Whether a tree's frame nodes and triangles are few enough that most of a launch's loads
// hit in L1 (256 KB per SM, shared with the lanes' lists) if they allocate there.
// 1,000,003 uniform queries with / without: 80 triangles 376 / 793 us, 1,280 (125 KB)
// 545 / 730, 3,000 in a soup (320 KB) 294 / 404, 5,120 (500 KB) 705 / 759, 20,480 in a
// smooth mesh 950 / 909; 12 triangles 69 / 193.  20,000 x 256 walks 11.8 / 22.9, 17.5 / 20.2,
// 39.4 / 57.6, 23.7 / 22.8 ms on the first four (3,968 triangles, 340 KB: 21.5 / 21.0).
constexpr int64_t kL1Bytes = 288 << 10;
inline bool fits_l1(int64_t nodes, int64_t triangles) {
  return nodes * static_cast<int64_t>(sizeof(FrameNode4)) + triangles * static_cast<int64_t>(sizeof(TriEdges)) <= kL1Bytes;
}

void launch_inside(const n2w_bvh& bvh, const n2w_vec3* d_points, int n, uint8_t* d_inside, int* d_overflow,
                   int block_size, cudaStream_t stream);

int sm_count_current();

// ---- device utilities (util.cu) ----
void launch_oracle_cache(const n2w_problem& pb, const float* d_inputs, int64_t n, const float* in_min,
                         const float* in_ext, float* d_out, cudaStream_t s);
void launch_count_samples(const uint8_t* needs, const int* forced, const int* overflow, int64_t n,
                          unsigned long long* d_counts, cudaStream_t s);
void launch_exact(const n2w_problem& pb, const n2w_vec3* d_points, int64_t n, float* d_out, cudaStream_t s);

// ---- stream-ordered scratch (util.cu) ----
// Allocations come from a memory pool the library owns on each device, which
// keeps up to kScratchRetainBytes cached across synchronisations, so repeated
// calls reuse mapped memory instead of remapping it (the device's default
// pool, left untouched, releases everything at each synchronisation).
constexpr uint64_t kScratchRetainBytes = uint64_t{2} << 30;
void* scratch_alloc(size_t bytes, cudaStream_t s);
void scratch_free(void* p, cudaStream_t s);

}  // namespace n2w
