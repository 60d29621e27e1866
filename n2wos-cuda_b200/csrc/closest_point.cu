// Device-pointer closest-point queries over the 4-wide BVH (reference
// CudaBvh::query_device, src/cuda/bvh_query.cu:228-261, and the masked cuBQL
// variant, src/cuda/cubql_bvh.cu:187-214).  Each query is seeded with the
// triangle stored at the nearest seed-grid node (a real candidate, so the
// exact answer is unchanged), started at that cell's subtrees and finished by
// the search over the frame nodes of geom.cuh, or over the axis-aligned ones
// where those are the better (choose_nodes, far_limit), or by a whole warp
// (warp_search.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>

#include "geom.cuh"
#include "internal.hpp"
#include "philox.cuh"
#include "warp_search.cuh"

namespace n2w {

dev::SeedGrid seed_grid_of(const n2w_bvh& b) {
  dev::SeedGrid g;
  g.cells = b.d_seed;
  g.lo_x = b.seed_lo[0];
  g.lo_y = b.seed_lo[1];
  g.lo_z = b.seed_lo[2];
  g.inv_h = b.seed_h > 0.0f ? 1.0f / b.seed_h : 0.0f;
  g.n = b.seed_n;
  g.far = b.seed_far;
  return g;
}

dev::QueryNodes query_nodes_of(const n2w_bvh& b) {
  return dev::QueryNodes{reinterpret_cast<const float4*>(b.d_frames), reinterpret_cast<const float4*>(b.d_nodes),
                         b.use_boxes};
}

namespace {

// Persistent state machine, one lane per query.  Every iteration each busy
// lane advances its query by one step (a triangle and two nodes; the
// counting variant by one unit of dev::trav_step_boxes), and a lane whose query
// is complete writes it and takes the next query in the same iteration.  Each
// block owns the contiguous range [b n / B, (b + 1) n / B) of the queries and
// its lanes take them from a shared-memory counter as they finish, so a lane
// that drew slow queries does not hold up queries that idle lanes of its
// block could run (with a fixed grid-stride sequence, launches of ~1-2
// queries per lane last as long as their unluckiest lane's pair).  Lanes
// therefore never wait for another lane's whole traversal (one-query-per-thread
// loops leave ~3.6 of 32 lanes active on incoherent queries).
constexpr int kQueryBlock = 256;
// Traversal units (node expansions + triangle tests) a lane spends on one
// query before handing it to the warp-cooperative finisher, when the launch
// holds about one query per resident lane; the few queries far from the
// surface in every direction (near the centre of a closed mesh) need
// thousands against a mean of ~40, and one of them per lane would set the
// launch's length.  With more queries per lane the lanes' totals even out and
// the budget grows in proportion, so a full GPU hands off only the extreme
// queries.  Budget 64 / 80 / 96 / 112 / 128: 409 / 370 / 357 / 357 / 362 us
// (262,144 uniform queries), 179 / 181 / 183 / 187 / 190 us (300,000 near the
// surface), 170 / 153 / 158 / 151 / 151 us (40,000); 4,194,304: the same.
constexpr uint32_t kQueryBudget = 112;
constexpr uint32_t kBoxBudget = 384;  // the same over the boxes, whose long queries have more nodes to visit
constexpr int kFinishWarps = 32;    // warps per SM that a finisher launch aims at (24 are resident: 78 registers)
constexpr int kHandOff = 2;         // overflow-slot mark of a handed-off query
constexpr int kHandOffFar = 3;      // the same for a far one (far_limit), handed off as soon as it is seeded
// Between warp_query_limit and kShortQueries a lane keeps only the queries whose seed lies
// within kShortCells of the grid's cells and hands the others off at once: 24,000 uniform
// 106 us (all lanes 133, all warps 76), near the surface 39 (36, 54).  Small trees
// (fits_l1) do without: their searches are short everywhere.
constexpr int kShortQueries = 32768;
constexpr float kShortCells = 1.0f;
// Resident blocks per SM the traversal is compiled for: 4 (56-62 registers, no
// spills).  3 / 4 / 5: 420 / 372 / 404 us (262,144 uniform queries), 426 / 423 / 503
// us (1,000,003 masked, near the surface), 4.38 / 4.22 / 4.37 ms (4,194,304).
constexpr int kQueryBlocks = 4;

// What a launch of lanes searches.
enum { kFrames, kBoxes, kCounted };  // frame nodes; boxes; boxes with every visit from the root counted

// One lane's query in flight; step() returns false once it is complete.
template <int kMode, bool kL1>
struct Search {
  dev::TravState t;
  int2 stack[kTraversalStack];
  __device__ __forceinline__ void start(int4) { t = dev::TravState{0, 0, 0, 0}; }
  __device__ __forceinline__ bool step(const float4* __restrict__ nodes, const float4* __restrict__ tris, dev::V3 p,
                                       dev::ClosestHit& hit, uint32_t& c_nodes, uint32_t& c_tris, bool& overflow) {
    // Two units per pass.
    return dev::trav_step_boxes<kL1>(nodes, tris, p, hit, t, stack, c_nodes, c_tris, overflow) &&
           (kMode == kCounted || dev::trav_step_boxes<kL1>(nodes, tris, p, hit, t, stack, c_nodes, c_tris, overflow));
  }
};
template <bool kL1>
struct Search<kFrames, kL1> {
  dev::FrameTrav t;
  dev::FrameStack stack;
  __device__ __forceinline__ void start(int4 cell) { t.start(cell, stack); }
  __device__ __forceinline__ bool step(const float4* __restrict__ frames, const float4* __restrict__ tris, dev::V3 p,
                                       dev::ClosestHit& hit, uint32_t& c_nodes, uint32_t& c_tris, bool& overflow) {
    // Two nodes per triangle: uniform queries expand 26 nodes and test 13
    // triangles (one node: 372 against 357 us for 262,144 queries, equal for
    // 1,000,003 near the surface and 4,194,304).
    dev::trav_triangle<false, kL1>(tris, p, hit, t, stack, c_tris);
    dev::trav_node<kL1, true>(frames, p, hit, t, stack, c_nodes, overflow);
    dev::trav_node<kL1, true>(frames, p, hit, t, stack, c_nodes, overflow);
    return !t.done();
  }
};

template <bool kMasked, int kMode, bool kL1>
__global__ void __launch_bounds__(kQueryBlock, kQueryBlocks) closest_point_kernel(
    const float4* __restrict__ nodes, const float4* __restrict__ tris, const dev::SeedGrid grid,
    const n2w_vec3* __restrict__ points, const uint8_t* __restrict__ active, int n,
    float* __restrict__ out_d2, n2w_vec3* __restrict__ out_cp, int* __restrict__ out_id,
    int* __restrict__ out_overflow, int* __restrict__ out_nodes, int* __restrict__ out_tris, uint32_t budget,
    float keep_d2) {
  // next unclaimed query of this block's range (unsigned: after the range
  // runs out each lane claims once more, up to b_end + blockDim.x <= 2^31 + 1023)
  constexpr bool kCount = kMode == kCounted;
  __shared__ unsigned s_next;
  const unsigned b_end = static_cast<unsigned>((static_cast<int64_t>(blockIdx.x) + 1) * n / gridDim.x);
  if (threadIdx.x == 0) s_next = static_cast<unsigned>(static_cast<int64_t>(blockIdx.x) * n / gridDim.x);
  __syncthreads();
  int q = 0;
  bool busy = false, drained = false;
  dev::V3 p = dev::v3(0.0f, 0.0f, 0.0f);
  dev::ClosestHit hit;
  hit.d2 = hit.lim = FLT_MAX;
  hit.id = INT32_MAX;
  hit.slot = -1;
  hit.cp = p;
  uint32_t c_nodes = 0, c_tris = 0;
  bool overflow = false;
  Search<kMode, kL1> search;
  // Hands the query to the finisher with its best so far (a bound on the answer) in
  // its own output slots.
  auto hand_off = [&](int mark) {
    out_d2[q] = hit.d2;
    out_cp[q] = n2w_vec3{hit.cp.x, hit.cp.y, hit.cp.z};
    out_id[q] = hit.id == INT32_MAX ? -1 : hit.id;
    out_overflow[q] = mark;
  };
  for (;;) {
    while (!busy && !drained) {
      const unsigned claim = atomicAdd(&s_next, 1u);
      if (claim >= b_end) {
        drained = true;  // stop claiming
        break;
      }
      q = static_cast<int>(claim);
      const n2w_vec3 pt = points[q];
      if (kMasked && active[q] == 0) {
        out_d2[q] = 0.0f;
        out_cp[q] = pt;
        out_id[q] = -1;
        out_overflow[q] = 0;
        if (kCount) {
          out_nodes[q] = 0;
          out_tris[q] = 0;
        }
        continue;
      }
      p = dev::v3(pt.x, pt.y, pt.z);
      hit.d2 = hit.lim = FLT_MAX;
      hit.id = INT32_MAX;
      hit.slot = -1;
      hit.cp = dev::v3(0.0f, 0.0f, 0.0f);
      c_nodes = c_tris = 0;
      overflow = false;
      int4 cell = make_int4(0, 0, kEmptyChild, kEmptyChild);  // the root
      if (grid.cells) {
        bool far = false;
        cell = kMode == kFrames ? dev::seed_cell_any(grid, p, 0, far) : dev::seed_cell(grid, p, 0);
        dev::test_slot<kL1>(tris, cell.x, p, hit);
        ++c_tris;
        if (kMode == kFrames && (far || hit.d2 > keep_d2)) {
          hand_off(far ? kHandOffFar : kHandOff);
          continue;
        }
      }
      search.start(cell);
      busy = true;
    }
    if (!__any_sync(0xffffffffu, busy)) break;
    if (busy) {
      if (!kCount && budget && c_nodes + c_tris > budget) {
        hand_off(kHandOff);  // over budget
        busy = false;
      } else if (!search.step(nodes, tris, p, hit, c_nodes, c_tris, overflow)) {
        out_d2[q] = hit.d2;
        out_cp[q] = n2w_vec3{hit.cp.x, hit.cp.y, hit.cp.z};
        out_id[q] = hit.id == INT32_MAX ? -1 : hit.id;
        out_overflow[q] = overflow ? 1 : 0;
        if (kCount) {
          out_nodes[q] = static_cast<int>(c_nodes);
          out_tris[q] = static_cast<int>(c_tris);
        }
        busy = false;
      }
    }
  }
}

// Finisher for the queries that ran over the per-lane budget or are far away (marked in
// their overflow slot): one warp per group of up to 32 consecutive queries takes its
// marked queries one at a time and searches again (warp_search.cuh) with the
// lane's best so far as the bound.  Blocks whose groups hold no marked query
// exit at once, so the block scheduler balances the work.  (A lane per far query
// instead: 81,920 triangles, 100,003 queries 500 extents away 727 -> 1,335 us, two close
// sheets of 45,000 triangles 4 -> 50 ms.)
__global__ void __launch_bounds__(32 * dev::kWarpsPerBlock) closest_point_finish_kernel(
    const dev::QueryNodes nodes, const float4* __restrict__ tris, const dev::SeedGrid grid,
    const n2w_vec3* __restrict__ points, int n, int group, float* __restrict__ out_d2,
    n2w_vec3* __restrict__ out_cp, int* __restrict__ out_id, int* __restrict__ out_overflow) {
  extern __shared__ int2 s_work[];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  int2* work = s_work + warp * dev::kWarpList;
  const int64_t q0 = (static_cast<int64_t>(blockIdx.x) * dev::kWarpsPerBlock + warp) * group;
  if (q0 >= n) return;
  const int64_t mine = q0 + lane;
  const int mark = lane < group && mine < n ? out_overflow[mine] : 0;
  unsigned pending = __ballot_sync(0xffffffffu, mark >= kHandOff);
  const unsigned far = __ballot_sync(0xffffffffu, mark == kHandOffFar);
  while (pending) {
    const int i = __ffs(pending) - 1, q = static_cast<int>(q0) + i;
    pending &= pending - 1;
    const n2w_vec3 pt = points[q], c0 = out_cp[q];
    const dev::V3 p = dev::v3(pt.x, pt.y, pt.z);
    const int id0 = out_id[q];
    dev::WarpBest b;
    b.key = b.mine = dev::hit_key(out_d2[q], id0 < 0 ? INT32_MAX : id0);
    b.cp = dev::v3(c0.x, c0.y, c0.z);
    b.slot = -1;
    int4 start = make_int4(0, 0, kEmptyChild, kEmptyChild);  // the root
    bool at_far;
    if (grid.cells) start = dev::seed_cell_any(grid, p, 0, at_far);
    dev::warp_search<false>(nodes, tris, p, start, (far >> i) & 1u, b, work);
    if (b.winner()) {
      const int id = static_cast<int>(b.key & 0xffffffffu);
      out_d2[q] = dev::key_d2(b.key);
      out_id[q] = id == INT32_MAX ? -1 : id;
      out_cp[q] = n2w_vec3{b.cp.x, b.cp.y, b.cp.z};
      out_overflow[q] = b.dropped;
    }
    __syncwarp();
  }
}

// Small launches: one warp per query (warp_search.cuh).  The smallest are as short as the
// code they fetch and run without the search over boxes: 1,000 / 40 queries of 5,120
// triangles, waited for, 16.9 / 14.9 -> 15.9 / 14.3 us.  (1,000 queries 50,000 extents from
// 81,920 triangles then take 1.1 ms instead of 0.04; 5,000 extents 0.2.)
constexpr int kFramesOnlyQueries = 2048;

template <bool kMasked, bool kFramesOnly>
__global__ void __launch_bounds__(32 * dev::kWarpsPerBlock) closest_point_warp_kernel(
    const dev::QueryNodes nodes, const float4* __restrict__ tris, const dev::SeedGrid grid,
    const n2w_vec3* __restrict__ points, const uint8_t* __restrict__ active, int n, float* __restrict__ out_d2,
    n2w_vec3* __restrict__ out_cp, int* __restrict__ out_id, int* __restrict__ out_overflow) {
  extern __shared__ int2 s_work[];
  const int warp = threadIdx.x >> 5;
  const int q = static_cast<int>(blockIdx.x) * dev::kWarpsPerBlock + warp;
  if (q >= n) return;
  const n2w_vec3 pt = points[q];
  if (kMasked && active[q] == 0) {
    if ((threadIdx.x & 31) == 0) {
      out_d2[q] = 0.0f;
      out_cp[q] = pt;
      out_id[q] = -1;
      out_overflow[q] = 0;
    }
    return;
  }
  const dev::WarpBest b = dev::warp_query<kFramesOnly>(nodes, tris, grid, dev::v3(pt.x, pt.y, pt.z), 0,
                                                       dev::v3(0.0f, 0.0f, 0.0f), s_work + warp * dev::kWarpList);
  if (b.winner()) {
    const int id = static_cast<int>(b.key & 0xffffffffu);
    out_d2[q] = dev::key_d2(b.key);
    out_cp[q] = n2w_vec3{b.cp.x, b.cp.y, b.cp.z};
    out_id[q] = id == INT32_MAX ? -1 : id;
    out_overflow[q] = b.dropped;
  }
}

// Builds the seed grid: an exact query at every lattice node, in two passes.  The
// first runs cold queries (ordered, over the axis-aligned nodes) at every
// kSeedStride-th node of each axis; the second seeds every other node with the
// triangle of the nearest of those.  129^3 nodes of the 81,920-triangle icosphere:
// 16.2 -> 4.1 ms against cold queries at all nodes.
constexpr int kSeedStride = 8;
static_assert(kSeedGridCells % kSeedStride == 0, "the coarse lattice spans the lattice");

// Lattice position lo + h * i, rounded per operation (no FMA) so a host
// float32 evaluation of the same expression gives the same point.
__device__ __forceinline__ dev::V3 lattice_point(float lox, float loy, float loz, float h, int ix, int iy, int iz) {
  return dev::v3(__fadd_rn(lox, __fmul_rn(h, static_cast<float>(ix))),
                 __fadd_rn(loy, __fmul_rn(h, static_cast<float>(iy))),
                 __fadd_rn(loz, __fmul_rn(h, static_cast<float>(iz))));
}

// kCold: node i of the (n / kSeedStride + 1)^3 coarse lattice into coarse[i]; else
// node i of all into cells[i], from the coarse ones.
template <bool kCold>
__global__ void __launch_bounds__(256) seed_grid_kernel(const dev::QueryNodes nodes,
                                                        const float4* __restrict__ tris, float lox, float loy,
                                                        float loz, float h, int n, int4* coarse, int4* cells,
                                                        int* overflow) {
  const int per_axis = kCold ? n / kSeedStride + 1 : n + 1;
  const int64_t total = static_cast<int64_t>(per_axis) * per_axis * per_axis;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int scale = kCold ? kSeedStride : 1;
  const int ix = scale * static_cast<int>(i % per_axis), iy = scale * static_cast<int>((i / per_axis) % per_axis),
            iz = scale * static_cast<int>(i / (static_cast<int64_t>(per_axis) * per_axis));
  const dev::V3 p = lattice_point(lox, loy, loz, h, ix, iy, iz);
  dev::ClosestHit hit;
  hit.d2 = hit.lim = FLT_MAX;
  hit.id = INT32_MAX;
  hit.slot = 0;
  hit.cp = p;
  dev::TraversalStats st{0, 0, 0};
  if constexpr (kCold) {
    dev::traverse(nodes.boxes, tris, p, hit, st);
    coarse[i] = make_int4(hit.slot, 0, kEmptyChild, kEmptyChild);
  } else {
    // the coarse lattice is a seed grid itself, each node its nearest point's seed
    const dev::SeedGrid g{coarse, lox, loy, loz, 1.0f / (h * kSeedStride), n / kSeedStride, INFINITY};
    if (ix % kSeedStride == 0 && iy % kSeedStride == 0 && iz % kSeedStride == 0) {
      const int m = n / kSeedStride + 1;
      hit.slot = coarse[(static_cast<int64_t>(iz / kSeedStride) * m + iy / kSeedStride) * m + ix / kSeedStride].x;
    } else {
      dev::traverse_query(nodes, tris, g, p, hit, st, 0);
    }
    cells[i] = make_int4(hit.slot, 0, kEmptyChild, kEmptyChild);  // from the root until build_cell_entries
  }
  if (st.overflow) atomicOr(overflow, 1);
}

// ---- frames or boxes -----------------------------------------------------------
// The work (nodes and triangles) of sample queries over both kinds of node, for
// choose_nodes: kind 0 in the mesh's box, 1 near the surface, 2 around it outside the
// lattice.  One lane per sample; a search ends after kSampleUnits.
constexpr int kSamples = 2048;  // of each kind
constexpr uint32_t kSampleUnits = 1024;

__global__ void __launch_bounds__(64) sample_work_kernel(const dev::QueryNodes nodes, const float4* __restrict__ tris,
                                                         int n_tris, const dev::SeedGrid grid,
                                                         unsigned long long* __restrict__ work) {
  const int i = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x), kind = i / kSamples;
  const U4 r = philox4x32_10(U4{static_cast<uint32_t>(i), 0u, 0u, 0u}, 0x5bd1e995u, 0x2545f491u);
  const float ux = 2.0f * u01(r.x) - 1.0f, uy = 2.0f * u01(r.y) - 1.0f, uz = 2.0f * u01(r.z) - 1.0f;
  const float half = 0.5f * static_cast<float>(grid.n) / grid.inv_h;  // of the lattice; the mesh's box: 5/7 of it
  float scale = half * (5.0f / 7.0f);
  dev::V3 c = dev::v3(grid.lo_x + half, grid.lo_y + half, grid.lo_z + half);
  if (kind == 1) {
    const float4* t = tris + 4 * static_cast<size_t>(static_cast<uint32_t>(r.w % static_cast<uint32_t>(n_tris)));
    const float4 a = __ldg(t), e = __ldg(t + 1), f = __ldg(t + 2);
    c = dev::v3(a.x + (e.x + e.w) / 3.0f, a.y + (e.y + f.x) / 3.0f, a.z + (e.z + f.y) / 3.0f);
    scale = half * (1.0f / 64.0f);
  } else if (kind == 2) {
    scale = 2.0f * half / fmaxf(fmaxf(fabsf(ux), fabsf(uy)), fmaxf(fabsf(uz), 1.0e-3f));
  }
  const dev::V3 p = dev::v3(c.x + scale * ux, c.y + scale * uy, c.z + scale * uz);
  dev::ClosestHit seed;
  seed.d2 = seed.lim = FLT_MAX;
  seed.id = INT32_MAX;
  seed.slot = -1;
  seed.cp = p;
  bool far;
  const int4 cell = dev::seed_cell_any(grid, p, 0, far);
  dev::test_slot(tris, cell.x, p, seed);
  uint32_t units[2] = {0, 0};
  bool overflow = false;
  {
    dev::ClosestHit hit = seed;
    Search<kFrames, true> s;
    uint32_t c_nodes = 0, c_tris = 0;
    s.start(cell);
    while (!s.t.done() && c_nodes + c_tris < kSampleUnits) {
      s.step(nodes.frames, tris, p, hit, c_nodes, c_tris, overflow);
    }
    units[0] = min(c_nodes + c_tris, kSampleUnits);
  }
  {
    dev::ClosestHit hit = seed;
    Search<kBoxes, true> s;
    uint32_t c_nodes = 0, c_tris = 0;
    s.start(cell);
    while (c_nodes + c_tris < kSampleUnits && s.step(nodes.boxes, tris, p, hit, c_nodes, c_tris, overflow)) {
    }
    units[1] = min(c_nodes + c_tris, kSampleUnits);
  }
  for (int k = 0; k < 2; ++k) {
    const uint32_t sum = __reduce_add_sync(0xffffffffu, units[k]);
    if ((threadIdx.x & 31) == 0) atomicAdd(&work[2 * kind + k], static_cast<unsigned long long>(sum));
  }
}

// Inside/outside by ray parity along +x with the reference's deterministic
// offset (src/cuda/cubql_bvh.cu:446-455).
__global__ void __launch_bounds__(1024) inside_kernel(const float4* __restrict__ nodes,
                                                      const float4* __restrict__ tris,
                                                      const n2w_vec3* __restrict__ points, int n,
                                                      uint8_t* __restrict__ inside, int* __restrict__ overflow) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const n2w_vec3 p = points[q];
  int ov = 0;
  const int hits = dev::ray_x_crossings(nodes, tris, dev::v3(p.x, p.y + 1.928371e-6f, p.z + 3.141593e-6f), ov);
  inside[q] = (hits & 1) ? 1 : 0;
  if (ov) atomicOr(overflow, 1);
}

}  // namespace

void launch_inside(const n2w_bvh& bvh, const n2w_vec3* d_points, int n, uint8_t* d_inside, int* d_overflow,
                   int block_size, cudaStream_t stream) {
  const int grid = (n + block_size - 1) / block_size;
  inside_kernel<<<grid, block_size, 0, stream>>>(reinterpret_cast<const float4*>(bvh.d_nodes),
                                                 reinterpret_cast<const float4*>(bvh.d_tris), d_points, n,
                                                 d_inside, d_overflow);
  N2W_CUDA(cudaGetLastError());
}

void launch_closest_point(const n2w_bvh& bvh, const n2w_vec3* d_points, const uint8_t* d_active,
                          int n, float* d_d2, n2w_vec3* d_cp, int* d_id, int* d_overflow,
                          int* d_nodes, int* d_tris, int block_size, cudaStream_t stream) {
  // block_size (the reference's launch knob, validated to [1, 1024]) is a hint:
  // the kernel runs 256-thread blocks, each over its own range of the queries,
  // with the grid sized to the resident capacity of the GPU.
  (void)block_size;
  const dev::QueryNodes nodes = query_nodes_of(bvh);
  const float4* tris = reinterpret_cast<const float4*>(bvh.d_edges);
  const dev::SeedGrid sg = seed_grid_of(bvh);
  const bool small_tree = fits_l1(bvh.stats.nodes, bvh.stats.triangles);
  const bool only_short = n <= kShortQueries && !small_tree && !nodes.use_boxes;
  const float keep = only_short ? kShortCells * bvh.seed_h : 1.0e19f;
  auto launch = [&](auto kern, const float4* searched, const uint8_t* act, uint32_t lane_budget, int* dn, int* dt) {
    int occ = 0;
    N2W_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kQueryBlock, 0));
    const int64_t blocks_needed = (static_cast<int64_t>(n) + kQueryBlock - 1) / kQueryBlock;
    const int64_t resident = static_cast<int64_t>(sm_count_current()) * std::max(occ, 1);
    const int grid = static_cast<int>(std::max<int64_t>(1, std::min(blocks_needed, resident)));
    const int64_t lanes = resident * kQueryBlock;
    const int64_t per_lane = (static_cast<int64_t>(n) + 2 * lanes - 1) / (2 * lanes);  // ceil(n / (2 lanes))
    const uint32_t budget = static_cast<uint32_t>(std::min<int64_t>(lane_budget * std::max<int64_t>(per_lane, 1),
                                                                    1 << 30));
    kern<<<grid, kQueryBlock, 0, stream>>>(searched, tris, sg, d_points, act, n, d_d2, d_cp, d_id, d_overflow, dn, dt,
                                           budget, keep * keep);
  };
  if (d_nodes) {
    // the counting variant runs every query to completion in one lane, so its
    // counts are the single-lane traversal's (the algorithmic work)
    launch(closest_point_kernel<false, kCounted, true>, nodes.boxes, d_active, 0, d_nodes, d_tris);
    N2W_CUDA(cudaGetLastError());
    return;
  }
  if (n <= warp_query_limit(bvh.stats.triangles, nodes.use_boxes, false)) {
    const unsigned blocks = static_cast<unsigned>((n + dev::kWarpsPerBlock - 1) / dev::kWarpsPerBlock);
    const bool frames_only = n <= kFramesOnlyQueries && !nodes.use_boxes;
    auto kern = d_active ? (frames_only ? closest_point_warp_kernel<true, true> : closest_point_warp_kernel<true, false>)
                         : (frames_only ? closest_point_warp_kernel<false, true> : closest_point_warp_kernel<false, false>);
    kern<<<blocks, 32 * dev::kWarpsPerBlock, dev::kWarpSearchBytes, stream>>>(nodes, tris, sg, d_points, d_active, n,
                                                                             d_d2, d_cp, d_id, d_overflow);
    N2W_CUDA(cudaGetLastError());
    return;
  }
  if (nodes.use_boxes) {
    // few nodes are visited, and often the same: their lines are kept
    auto kern = d_active ? closest_point_kernel<true, kBoxes, true> : closest_point_kernel<false, kBoxes, true>;
    launch(kern, nodes.boxes, d_active, kBoxBudget, nullptr, nullptr);
  } else if (small_tree) {
    auto kern = d_active ? closest_point_kernel<true, kFrames, true> : closest_point_kernel<false, kFrames, true>;
    launch(kern, nodes.frames, d_active, kQueryBudget, nullptr, nullptr);
  } else {
    auto kern = d_active ? closest_point_kernel<true, kFrames, false> : closest_point_kernel<false, kFrames, false>;
    launch(kern, nodes.frames, d_active, kQueryBudget, nullptr, nullptr);
  }
  N2W_CUDA(cudaGetLastError());
  // A warp's queries are searched one after the other.  Where most are handed off there
  // are few to a warp (4 a warp at most: 24,000 uniform 127 -> 106 us against 6), else as
  // few as the resident warps allow: launching more costs more than it gives (65,000 near
  // the surface 43.6 -> 46.8 us).
  const int64_t warps = static_cast<int64_t>(sm_count_current()) * kFinishWarps * (only_short ? 4 : 1);
  const int group = static_cast<int>(std::min<int64_t>((n + warps - 1) / warps, 32));
  const int64_t groups = (static_cast<int64_t>(n) + group - 1) / group;
  const unsigned blocks = static_cast<unsigned>((groups + dev::kWarpsPerBlock - 1) / dev::kWarpsPerBlock);
  closest_point_finish_kernel<<<blocks, 32 * dev::kWarpsPerBlock, dev::kWarpSearchBytes, stream>>>(
      nodes, tris, sg, d_points, n, group, d_d2, d_cp, d_id, d_overflow);
  N2W_CUDA(cudaGetLastError());
}

int sm_count_current() {
  int dev = 0, sms = 0;
  N2W_CUDA(cudaGetDevice(&dev));
  N2W_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  return sms;
}

// Chooses the nodes that queries of this tree search, with samples seeded by `grid`.  The frames' planes are whole
// bytes of a node's extent and their limit carries a margin, which pays where patches
// are oblique or curved; boxes around axis-aligned sides or bundles of needles are as
// thin and need neither.  The choice is the kind of node that the sample queries did
// less work over, in the geometric mean of their kinds: boxes / frames for 1 unit of
// uniform, near and outside queries 0.98 / 1.2 / 0.4 on an axis-aligned cube of 120,000
// triangles (300,000 uniform queries 157 us over frames, 125 over boxes), 4.0 / 2.2 /
// 4.6 on a torus of 80,000.
void choose_nodes(n2w_bvh& b, int triangles, const dev::SeedGrid& grid) {
  unsigned long long* d = nullptr;
  N2W_CUDA(cudaMalloc(&d, 6 * sizeof(unsigned long long)));
  unsigned long long w[6] = {};
  cudaError_t e = cudaMemset(d, 0, sizeof(w));
  if (e == cudaSuccess) {
    sample_work_kernel<<<3 * kSamples / 64, 64>>>(query_nodes_of(b), reinterpret_cast<const float4*>(b.d_edges),
                                                  triangles, grid, d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(w, d, sizeof(w), cudaMemcpyDeviceToHost);
  cudaFree(d);
  N2W_CUDA(e);
  double frames = 1.0, boxes = 1.0;
  for (int k = 0; k < 3; ++k) {
    frames *= static_cast<double>(w[2 * k] + 1);
    boxes *= static_cast<double>(w[2 * k + 1] + 1);
  }
  b.use_boxes = boxes < frames;
}

// SeedGrid::far.  The margin of the frame nodes' limit (prune_limit) grows with the
// query's distance d from the mesh c, 2^-20 |p|_1 + 2^-18 d <= 5.3e-6 d + 2^-20 |c|_1.
// Where it reaches a quarter of the triangles' edge it covers patches of them, and the
// axis-aligned boxes, which need none, leave far fewer to test: 81,920 triangles, work of
// a query over frames / boxes 158 / 244 at 500 extents, 1,764 / 249 at 5,000.
float far_limit(const n2w_bvh& b, double edge) {
  const double half = 0.5 * b.seed_n * static_cast<double>(b.seed_h);
  double centre = 0.0;
  for (int a = 0; a < 3; ++a) centre += std::fabs(b.seed_lo[a] + half);
  const double far = (0.25 * edge - centre * 0x1p-20) / (5.3e-6 * half);
  return static_cast<float>(far > 0.0 ? far : 0.0);  // (not a number: 0)
}

// Mean of the longer of two edges of each triangle.
double mean_edge(const n2w_mesh& mesh) {
  double edge = 0.0;
  for (const auto& t : mesh.triangles) {
    double l2[2] = {0.0, 0.0};
    for (int a = 0; a < 3; ++a) {
      const double x = mesh.vertices[t[0]][a];
      l2[0] += (mesh.vertices[t[1]][a] - x) * (mesh.vertices[t[1]][a] - x);
      l2[1] += (mesh.vertices[t[2]][a] - x) * (mesh.vertices[t[2]][a] - x);
    }
    edge += std::sqrt(std::max(l2[0], l2[1]));
  }
  return edge / static_cast<double>(mesh.triangles.size());
}

// Seed grid over the mesh box grown by 20 % of its largest extent on every side.
void build_seed_grid(n2w_bvh& b, const n2w_mesh& mesh, int n) {
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (const auto& v : mesh.vertices) {
    for (int a = 0; a < 3; ++a) {
      lo[a] = std::min(lo[a], v[a]);
      hi[a] = std::max(hi[a], v[a]);
    }
  }
  const float ext = std::max(std::max(hi[0] - lo[0], hi[1] - lo[1]), hi[2] - lo[2]);
  const float pad = 0.2f * ext + 1e-6f;
  const float h = (ext + 2.0f * pad) / static_cast<float>(n);
  for (int a = 0; a < 3; ++a) b.seed_lo[a] = 0.5f * (lo[a] + hi[a]) - 0.5f * (ext + 2.0f * pad);
  b.seed_h = h;
  b.seed_n = n;
  const int64_t total = static_cast<int64_t>(n + 1) * (n + 1) * (n + 1);
  N2W_CUDA(cudaMalloc(&b.d_seed, total * sizeof(int4)));
  const int64_t per_axis = n / kSeedStride + 1, cold = per_axis * per_axis * per_axis;
  char* tmp = nullptr;  // the coarse lattice, then the overflow flag
  N2W_CUDA(cudaMalloc(&tmp, cold * sizeof(int4) + sizeof(int)));
  int4* coarse = reinterpret_cast<int4*>(tmp);
  int* d_ov = reinterpret_cast<int*>(coarse + cold);
  int ov = 0;
  try {
    N2W_CUDA(cudaMemset(d_ov, 0, sizeof(int)));
    const int block = 256, cold_block = 64;  // cold queries are few and long: spread over the SMs
    const float4* tris = reinterpret_cast<const float4*>(b.d_edges);
    seed_grid_kernel<true><<<static_cast<unsigned>((cold + cold_block - 1) / cold_block), cold_block>>>(
        query_nodes_of(b), tris, b.seed_lo[0], b.seed_lo[1], b.seed_lo[2], h, n, coarse, b.d_seed, d_ov);
    N2W_CUDA(cudaGetLastError());
    choose_nodes(b, static_cast<int>(mesh.triangles.size()),
                 dev::SeedGrid{coarse, b.seed_lo[0], b.seed_lo[1], b.seed_lo[2], 1.0f / (h * kSeedStride),
                               n / kSeedStride, INFINITY});
    const double edge = mean_edge(mesh);
    b.seed_far = far_limit(b, edge);
    seed_grid_kernel<false><<<static_cast<unsigned>((total + block - 1) / block), block>>>(
        query_nodes_of(b), tris, b.seed_lo[0], b.seed_lo[1], b.seed_lo[2], h, n, coarse, b.d_seed, d_ov);
    N2W_CUDA(cudaGetLastError());
    // The cells' subtrees stand on computed distances being distances.  A triangle test
    // multiplies four lengths: where that overflows or loses its digits a search starts at
    // the root, as the cells say already.
    if (edge > 1.0e-8 && static_cast<double>(h) * n < 1.0e9) build_cell_entries(b);
    N2W_CUDA(cudaMemcpy(&ov, d_ov, sizeof(int), cudaMemcpyDeviceToHost));
  } catch (...) {
    cudaFree(tmp);
    throw;
  }
  cudaFree(tmp);
  if (ov) throw Error(N2W_EINTERNAL, "traversal stack overflow while building the seed grid");
}

}  // namespace n2w

using namespace n2w;

namespace {

void check_query_args(const n2w_bvh* bvh, const void* pts, int n, const void* d2, const void* cp,
                      const void* id, const void* ov, int block_size) {
  N2W_REQUIRE(bvh && bvh->d_nodes && bvh->d_tris, "query_device called on empty BVH");
  N2W_REQUIRE(n >= 0, "query_device query_count must be non-negative");
  if (n == 0) return;
  N2W_REQUIRE(pts && d2 && cp && id && ov, "query_device received a null device pointer");
  N2W_REQUIRE(block_size >= 1 && block_size <= 1024, "CUDA block size must be in [1, 1024]");
}

void release(n2w_bvh* b) {
  if (b->d_nodes) cudaFree(b->d_nodes);
  if (b->d_frames) cudaFree(b->d_frames);
  if (b->d_tris) cudaFree(b->d_tris);
  if (b->d_edges) cudaFree(b->d_edges);
  if (b->d_seed) cudaFree(b->d_seed);
  delete b;
}

}  // namespace

extern "C" {

int n2w_bvh_create(const n2w_mesh* mesh, int leaf_size, const char* build_method, n2w_bvh** out) {
  return guarded([&] {
    N2W_REQUIRE(mesh && out, "n2w_bvh_create: null argument");
    const auto t0 = std::chrono::steady_clock::now();
    HostBvh h = build_bvh4(*mesh, leaf_size, build_method ? build_method : "sah");
    auto* b = new n2w_bvh();
    try {
      N2W_CUDA(cudaGetDevice(&b->device));
      N2W_CUDA(cudaMalloc(&b->d_nodes, h.nodes.size() * sizeof(Node4)));
      N2W_CUDA(cudaMalloc(&b->d_tris, h.tris.size() * sizeof(TriRec)));
      N2W_CUDA(cudaMemcpy(b->d_nodes, h.nodes.data(), h.nodes.size() * sizeof(Node4), cudaMemcpyHostToDevice));
      N2W_CUDA(cudaMemcpy(b->d_tris, h.tris.data(), h.tris.size() * sizeof(TriRec), cudaMemcpyHostToDevice));
      build_edges(*b, static_cast<int64_t>(h.tris.size()));
      build_frames(*b, h);
      build_seed_grid(*b, *mesh, kSeedGridCells);
      N2W_CUDA(cudaDeviceSynchronize());
    } catch (...) {
      release(b);
      throw;
    }
    const auto t1 = std::chrono::steady_clock::now();
    b->stats = host_stats(h, leaf_size, std::chrono::duration<double, std::milli>(t1 - t0).count());
    b->stats.device_bytes += static_cast<int64_t>(h.nodes.size() * sizeof(FrameNode4) + h.tris.size() * sizeof(TriEdges));
    b->stats.device_bytes += static_cast<int64_t>(kSeedGridCells + 1) * (kSeedGridCells + 1) * (kSeedGridCells + 1) *
                              static_cast<int64_t>(sizeof(int4));
    *out = b;
  });
}

int n2w_bvh_stats_get(const n2w_bvh* bvh, n2w_bvh_stats* out) {
  return guarded([&] {
    N2W_REQUIRE(bvh && out, "null argument");
    *out = bvh->stats;
  });
}

void n2w_bvh_destroy(n2w_bvh* bvh) {
  if (bvh) release(bvh);
}

int n2w_bvh_query_device(const n2w_bvh* bvh, const n2w_vec3* d_points, int query_count,
                         float* d_distance2, n2w_vec3* d_closest, int* d_triangle_id,
                         int* d_overflow, int block_size, n2w_stream_t stream) {
  return guarded([&] {
    check_query_args(bvh, d_points, query_count, d_distance2, d_closest, d_triangle_id, d_overflow, block_size);
    if (query_count == 0) return;
    launch_closest_point(*bvh, d_points, nullptr, query_count, d_distance2, d_closest, d_triangle_id,
                         d_overflow, nullptr, nullptr, block_size, stream);
  });
}

int n2w_bvh_query_device_masked(const n2w_bvh* bvh, const n2w_vec3* d_points,
                                const uint8_t* d_active, int query_count, float* d_distance2,
                                n2w_vec3* d_closest, int* d_triangle_id, int* d_overflow,
                                int block_size, n2w_stream_t stream) {
  return guarded([&] {
    check_query_args(bvh, d_points, query_count, d_distance2, d_closest, d_triangle_id, d_overflow, block_size);
    if (query_count == 0) return;
    N2W_REQUIRE(d_active, "query_device_masked received a null mask");
    launch_closest_point(*bvh, d_points, d_active, query_count, d_distance2, d_closest, d_triangle_id,
                         d_overflow, nullptr, nullptr, block_size, stream);
  });
}

int n2w_bvh_query_device_counted(const n2w_bvh* bvh, const n2w_vec3* d_points, int query_count,
                                 float* d_distance2, n2w_vec3* d_closest, int* d_triangle_id,
                                 int* d_overflow, int* d_node_visits, int* d_tri_tests,
                                 int block_size, n2w_stream_t stream) {
  return guarded([&] {
    check_query_args(bvh, d_points, query_count, d_distance2, d_closest, d_triangle_id, d_overflow, block_size);
    if (query_count == 0) return;
    N2W_REQUIRE(d_node_visits && d_tri_tests, "counted query needs counter outputs");
    launch_closest_point(*bvh, d_points, nullptr, query_count, d_distance2, d_closest, d_triangle_id,
                         d_overflow, d_node_visits, d_tri_tests, block_size, stream);
  });
}

int n2w_bvh_inside_device(const n2w_bvh* bvh, const n2w_vec3* d_points, int query_count, uint8_t* d_inside,
                          int* d_overflow, int block_size, n2w_stream_t stream) {
  return guarded([&] {
    N2W_REQUIRE(bvh && bvh->d_nodes && bvh->d_tris, "inside_device called on empty BVH");
    N2W_REQUIRE(query_count >= 0, "query_count must be non-negative");
    if (query_count == 0) return;
    N2W_REQUIRE(d_points && d_inside && d_overflow, "inside_device received a null device pointer");
    N2W_REQUIRE(block_size >= 1 && block_size <= 1024, "CUDA block size must be in [1, 1024]");
    launch_inside(*bvh, d_points, query_count, d_inside, d_overflow, block_size, stream);
  });
}

int n2w_bvh_copy_layout(const n2w_bvh* bvh, void* nodes_out, void* tris_out) {
  return guarded([&] {
    N2W_REQUIRE(bvh, "null bvh");
    if (nodes_out) {
      N2W_CUDA(cudaMemcpy(nodes_out, bvh->d_nodes, static_cast<size_t>(bvh->stats.nodes) * sizeof(Node4),
                          cudaMemcpyDeviceToHost));
    }
    if (tris_out) {
      N2W_CUDA(cudaMemcpy(tris_out, bvh->d_tris, static_cast<size_t>(bvh->stats.triangles) * sizeof(TriRec),
                          cudaMemcpyDeviceToHost));
    }
  });
}

int n2w_bvh_seed_grid(const n2w_bvh* bvh, float* lo_out, float* h_out, int* n_out, int* slots_out) {
  return guarded([&] {
    N2W_REQUIRE(bvh && bvh->d_seed, "BVH has no seed grid");
    if (lo_out) std::memcpy(lo_out, bvh->seed_lo, sizeof(bvh->seed_lo));
    if (h_out) *h_out = bvh->seed_h;
    if (n_out) *n_out = bvh->seed_n;
    if (slots_out) {
      const size_t s = static_cast<size_t>(bvh->seed_n) + 1;
      copy_cell_slots(*bvh, static_cast<int64_t>(s * s * s), slots_out);
    }
  });
}

}  // extern "C"
