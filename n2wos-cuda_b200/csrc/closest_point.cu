// Device-pointer closest-point queries over the 4-wide BVH (reference
// CudaBvh::query_device, src/cuda/bvh_query.cu:228-261, and the masked cuBQL
// variant, src/cuda/cubql_bvh.cu:187-214).  Each query is seeded with the
// triangle stored at the nearest seed-grid node (a real candidate, so the
// exact answer is unchanged), started at that cell's subtrees and finished by
// the search over the frame nodes of geom.cuh, or by a whole warp
// (warp_search.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstring>

#include "geom.cuh"
#include "internal.hpp"
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
  return g;
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
constexpr int kHandOff = 2;         // overflow-slot mark of a handed-off query
// Launches of at most this many queries give each query a warp: with a lane per
// query a launch lasts as long as its slowest serial search, whatever its size.
// Lane / warp per query, uniform points, 81,920 triangles: 71 / 11 us (40
// queries), 126 / 12 (1,000), 144 / 26 (4,000), 151 / 74 (16,000), 153 / 141
// (32,000), 374 / 1,076 (262,144).
constexpr int kWarpQueries = 32768;
// Resident blocks per SM the traversal is compiled for: 4 (56-62 registers, no
// spills).  3 / 4 / 5: 420 / 372 / 404 us (262,144 uniform queries), 426 / 423 / 503
// us (1,000,003 masked, near the surface), 4.38 / 4.22 / 4.37 ms (4,194,304).
constexpr int kQueryBlocks = 4;

// One lane's query in flight; step() returns false once it is complete.
template <bool kCount>
struct Search {
  dev::FrameTrav t;
  dev::FrameStack stack;
  __device__ __forceinline__ void start(int4 cell) { t.start(cell, stack); }
  __device__ __forceinline__ bool step(const float4* __restrict__ frames, const float4* __restrict__ tris, dev::V3 p,
                                       dev::ClosestHit& hit, uint32_t& c_nodes, uint32_t& c_tris, bool& overflow) {
    // Two nodes per triangle: uniform queries expand 26 nodes and test 13
    // triangles (one node: 372 against 357 us for 262,144 queries, equal for
    // 1,000,003 near the surface and 4,194,304).
    dev::trav_triangle<false>(tris, p, hit, t, stack, c_tris);
    dev::trav_node<false, true>(frames, p, hit, t, stack, c_nodes, overflow);
    dev::trav_node<false, true>(frames, p, hit, t, stack, c_nodes, overflow);
    return !t.done();
  }
};
template <>
struct Search<true> {
  dev::TravState t;
  int2 stack[kTraversalStack];
  __device__ __forceinline__ void start(int4) { t = dev::TravState{0, 0, 0, 0}; }  // every visit from the root counts
  __device__ __forceinline__ bool step(const float4* __restrict__ nodes, const float4* __restrict__ tris, dev::V3 p,
                                       dev::ClosestHit& hit, uint32_t& c_nodes, uint32_t& c_tris, bool& overflow) {
    return dev::trav_step_boxes(nodes, tris, p, hit, t, stack, c_nodes, c_tris, overflow);
  }
};

template <bool kMasked, bool kCount>
__global__ void __launch_bounds__(kQueryBlock, kQueryBlocks) closest_point_kernel(
    const float4* __restrict__ nodes, const float4* __restrict__ tris, const dev::SeedGrid grid,
    const n2w_vec3* __restrict__ points, const uint8_t* __restrict__ active, int n,
    float* __restrict__ out_d2, n2w_vec3* __restrict__ out_cp, int* __restrict__ out_id,
    int* __restrict__ out_overflow, int* __restrict__ out_nodes, int* __restrict__ out_tris, uint32_t budget) {
  // next unclaimed query of this block's range (unsigned: after the range
  // runs out each lane claims once more, up to b_end + blockDim.x <= 2^31 + 1023)
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
  Search<kCount> search;
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
        cell = kCount ? dev::seed_cell(grid, p, 0) : dev::seed_cell_any(grid, p, 0);
        dev::test_slot(tris, cell.x, p, hit);
        ++c_tris;
      }
      search.start(cell);
      busy = true;
    }
    if (!__any_sync(0xffffffffu, busy)) break;
    if (busy) {
      if (!kCount && budget && c_nodes + c_tris > budget) {
        // Over budget: hand the query to the warp-cooperative finisher with its
        // best so far (a bound on the answer) in its own output slots.
        out_d2[q] = hit.d2;
        out_cp[q] = n2w_vec3{hit.cp.x, hit.cp.y, hit.cp.z};
        out_id[q] = hit.id == INT32_MAX ? -1 : hit.id;
        out_overflow[q] = kHandOff;
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

// Finisher for the queries that ran over the per-lane budget (marked kHandOff in
// their overflow slot): one warp per group of 32 consecutive queries takes its
// marked queries one at a time and searches again (warp_search.cuh) with the
// lane's best so far as the bound.  Blocks whose groups hold no marked query
// exit at once, so the block scheduler balances the work.
__global__ void __launch_bounds__(32 * dev::kWarpsPerBlock) closest_point_finish_kernel(
    const float4* __restrict__ nodes, const float4* __restrict__ tris, const dev::SeedGrid grid,
    const n2w_vec3* __restrict__ points, int n, float* __restrict__ out_d2, n2w_vec3* __restrict__ out_cp,
    int* __restrict__ out_id, int* __restrict__ out_overflow) {
  extern __shared__ int2 s_work[];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  int2* work = s_work + warp * dev::kWarpList;
  const int64_t q0 = (static_cast<int64_t>(blockIdx.x) * dev::kWarpsPerBlock + warp) * 32;
  if (q0 >= n) return;
  const int64_t mine = q0 + lane;
  unsigned pending = __ballot_sync(0xffffffffu, mine < n && out_overflow[mine] == kHandOff);
  while (pending) {
    const int q = static_cast<int>(q0) + __ffs(pending) - 1;
    pending &= pending - 1;
    const n2w_vec3 pt = points[q], c0 = out_cp[q];
    const dev::V3 p = dev::v3(pt.x, pt.y, pt.z);
    const int id0 = out_id[q];
    dev::WarpBest b;
    b.key = b.mine = dev::hit_key(out_d2[q], id0 < 0 ? INT32_MAX : id0);
    b.cp = dev::v3(c0.x, c0.y, c0.z);
    b.slot = -1;
    int4 start = make_int4(0, 0, kEmptyChild, kEmptyChild);  // the root
    if (grid.cells) start = dev::seed_cell_any(grid, p, 0);
    dev::warp_search(nodes, tris, p, start, b, work);
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

// Small launches: one warp per query (warp_search.cuh).
template <bool kMasked>
__global__ void __launch_bounds__(32 * dev::kWarpsPerBlock) closest_point_warp_kernel(
    const float4* __restrict__ nodes, const float4* __restrict__ tris, const dev::SeedGrid grid,
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
  const dev::WarpBest b = dev::warp_query(nodes, tris, grid, dev::v3(pt.x, pt.y, pt.z), 0, dev::v3(0.0f, 0.0f, 0.0f),
                                          s_work + warp * dev::kWarpList);
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
// triangle of the nearest of those and searches the frame nodes.  129^3 nodes of
// the 81,920-triangle icosphere: 16.2 -> 4.1 ms against cold queries at all nodes.
constexpr int kSeedStride = 8;

template <bool kCold>
__global__ void __launch_bounds__(256) seed_grid_kernel(const float4* __restrict__ nodes,
                                                        const float4* __restrict__ tris, float lox, float loy,
                                                        float loz, float h, int n, int4* cells, int* overflow) {
  const int s = n + 1;
  const int per_axis = kCold ? n / kSeedStride + 1 : s;
  const int64_t total = static_cast<int64_t>(per_axis) * per_axis * per_axis;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int scale = kCold ? kSeedStride : 1;
  const int ix = scale * static_cast<int>(i % per_axis), iy = scale * static_cast<int>((i / per_axis) % per_axis),
            iz = scale * static_cast<int>(i / (static_cast<int64_t>(per_axis) * per_axis));
  if (!kCold && ix % kSeedStride == 0 && iy % kSeedStride == 0 && iz % kSeedStride == 0) return;  // first pass
  auto index = [s](int x, int y, int z) { return (static_cast<int64_t>(z) * s + y) * s + x; };
  // Lattice position lo + h * i, rounded per operation (no FMA) so a host
  // float32 evaluation of the same expression gives the same point.
  const dev::V3 p = dev::v3(__fadd_rn(lox, __fmul_rn(h, static_cast<float>(ix))),
                            __fadd_rn(loy, __fmul_rn(h, static_cast<float>(iy))),
                            __fadd_rn(loz, __fmul_rn(h, static_cast<float>(iz))));
  dev::ClosestHit hit;
  hit.d2 = hit.lim = FLT_MAX;
  hit.id = INT32_MAX;
  hit.slot = 0;
  hit.cp = p;
  dev::TraversalStats st{0, 0, 0};
  if constexpr (kCold) {
    dev::traverse(nodes, tris, p, hit, st);
  } else {
    auto nearest = [n](int x) { return min((x + kSeedStride / 2) / kSeedStride * kSeedStride, n / kSeedStride * kSeedStride); };
    dev::test_slot(tris, cells[index(nearest(ix), nearest(iy), nearest(iz))].x, p, hit);
    dev::traverse_frames(nodes, tris, dev::SeedGrid{nullptr, 0.0f, 0.0f, 0.0f, 0.0f, 0}, p, hit, st, 0);
  }
  cells[index(ix, iy, iz)] = make_int4(hit.slot, 0, kEmptyChild, kEmptyChild);  // from the root until build_cell_entries
  if (st.overflow) atomicOr(overflow, 1);
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
  const float4* nodes = d_nodes ? reinterpret_cast<const float4*>(bvh.d_nodes)
                                : reinterpret_cast<const float4*>(bvh.d_frames);
  const float4* tris = reinterpret_cast<const float4*>(bvh.d_edges);
  const dev::SeedGrid sg = seed_grid_of(bvh);
  auto launch = [&](auto kern, const uint8_t* act, int* dn, int* dt) {
    int occ = 0;
    N2W_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kQueryBlock, 0));
    const int64_t blocks_needed = (static_cast<int64_t>(n) + kQueryBlock - 1) / kQueryBlock;
    const int64_t resident = static_cast<int64_t>(sm_count_current()) * std::max(occ, 1);
    const int grid = static_cast<int>(std::max<int64_t>(1, std::min(blocks_needed, resident)));
    const int64_t lanes = resident * kQueryBlock;
    const int64_t per_lane = (static_cast<int64_t>(n) + 2 * lanes - 1) / (2 * lanes);  // ceil(n / (2 lanes))
    const uint32_t budget = static_cast<uint32_t>(std::min<int64_t>(kQueryBudget * std::max<int64_t>(per_lane, 1),
                                                                    1 << 30));
    kern<<<grid, kQueryBlock, 0, stream>>>(nodes, tris, sg, d_points, act, n, d_d2, d_cp, d_id, d_overflow, dn, dt,
                                           dn ? 0u : budget);
  };
  if (d_nodes) {
    // the counting variant runs every query to completion in one lane, so its
    // counts are the single-lane traversal's (the algorithmic work)
    launch(closest_point_kernel<false, true>, d_active, d_nodes, d_tris);
    N2W_CUDA(cudaGetLastError());
    return;
  }
  if (n <= kWarpQueries) {
    const unsigned blocks = static_cast<unsigned>((n + dev::kWarpsPerBlock - 1) / dev::kWarpsPerBlock);
    auto kern = d_active ? closest_point_warp_kernel<true> : closest_point_warp_kernel<false>;
    kern<<<blocks, 32 * dev::kWarpsPerBlock, dev::kWarpSearchBytes, stream>>>(nodes, tris, sg, d_points, d_active, n,
                                                                             d_d2, d_cp, d_id, d_overflow);
    N2W_CUDA(cudaGetLastError());
    return;
  }
  if (d_active) launch(closest_point_kernel<true, false>, d_active, nullptr, nullptr);
  else launch(closest_point_kernel<false, false>, nullptr, nullptr, nullptr);
  N2W_CUDA(cudaGetLastError());
  const int64_t groups = (static_cast<int64_t>(n) + 31) / 32;
  const unsigned blocks = static_cast<unsigned>((groups + dev::kWarpsPerBlock - 1) / dev::kWarpsPerBlock);
  closest_point_finish_kernel<<<blocks, 32 * dev::kWarpsPerBlock, dev::kWarpSearchBytes, stream>>>(
      nodes, tris, sg, d_points, n, d_d2, d_cp, d_id, d_overflow);
  N2W_CUDA(cudaGetLastError());
}

int sm_count_current() {
  int dev = 0, sms = 0;
  N2W_CUDA(cudaGetDevice(&dev));
  N2W_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  return sms;
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
  int* d_ov = nullptr;
  N2W_CUDA(cudaMalloc(&d_ov, sizeof(int)));
  N2W_CUDA(cudaMemset(d_ov, 0, sizeof(int)));
  const int block = 256;
  const float4* tris = reinterpret_cast<const float4*>(b.d_edges);
  const int64_t coarse = n / kSeedStride + 1, cold = coarse * coarse * coarse;
  const int cold_block = 64;  // few and long queries: spread over the SMs
  seed_grid_kernel<true><<<static_cast<unsigned>((cold + cold_block - 1) / cold_block), cold_block>>>(
      reinterpret_cast<const float4*>(b.d_nodes), tris, b.seed_lo[0], b.seed_lo[1], b.seed_lo[2], h, n, b.d_seed, d_ov);
  seed_grid_kernel<false><<<static_cast<unsigned>((total + block - 1) / block), block>>>(
      reinterpret_cast<const float4*>(b.d_frames), tris, b.seed_lo[0], b.seed_lo[1], b.seed_lo[2], h, n, b.d_seed, d_ov);
  N2W_CUDA(cudaGetLastError());
  build_cell_entries(b);
  int ov = 0;
  N2W_CUDA(cudaMemcpy(&ov, d_ov, sizeof(int), cudaMemcpyDeviceToHost));
  cudaFree(d_ov);
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
