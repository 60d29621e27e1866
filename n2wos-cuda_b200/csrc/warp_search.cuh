// One closest-point query by a whole warp over the frame nodes: for queries that
// a lane handed off, and for launches too small to give every lane of the GPU a
// query, where a single lane's search (tens to thousands of dependent loads) is
// the launch's length.
//
// A shared-memory work list of (node or leaf, box distance) entries feeds the 32
// lanes: each iteration every lane takes one entry, expands a node (children
// whose box is within the warp's limit are appended) or tests a leaf's
// triangles, and the warp's best (d2, id) -- a 64-bit key, lowest d2 then lowest
// id -- is the minimum over lanes.  Pruning is conservative, so the answer is
// the exact one a single-lane traversal gives.
#pragma once

#include "geom.cuh"

namespace n2w {
namespace dev {

// Work-list entries per warp (4 KiB).  Entries are taken newest first, so an iteration
// adds at most 96 per tree level; as the list fills, fewer are taken at a time, and the
// last kWarpReserve are left to a depth-first search (3 per level) that fits in them as
// deep as a lane's stack does.  Against 16 KiB, which left 14 warps to an SM: 16,000 /
// 32,768 uniform queries 84.5 -> 60.4 / 152 -> 99.6 us (8 KiB: 63.0 / 105).
constexpr int kWarpList = 512;
constexpr int kWarpReserve = 64;
// Warps per block of the kernels that search by warps.
constexpr int kWarpsPerBlock = 2;
constexpr size_t kWarpSearchBytes = sizeof(int2) * kWarpsPerBlock * kWarpList;

__device__ __forceinline__ unsigned long long hit_key(float d2, int id) {
  return (static_cast<unsigned long long>(__float_as_uint(d2)) << 32) | static_cast<unsigned>(id);
}
__device__ __forceinline__ float key_d2(unsigned long long key) {
  return __uint_as_float(static_cast<unsigned>(key >> 32));
}

struct WarpBest {
  unsigned long long key;   // the warp's best, the same in every lane
  unsigned long long mine;  // this lane's best; cp and slot belong to it
  V3 cp;
  int slot;
  int dropped;           // the work list was full (the answer may be wrong)
  uint32_t nodes, tris;  // this lane's node expansions and triangle tests
  // The lane whose hit is the answer (the lowest, if a seed is).
  __device__ __forceinline__ bool winner() const {
    return (threadIdx.x & 31) == __ffs(__ballot_sync(0xffffffffu, mine == key)) - 1;
  }
};

// Searches the subtrees start.y, start.z, start.w (kEmptyChild when unused) for
// a hit better than b, which holds the seed in every lane.
template <bool kBoxes>
__device__ __forceinline__ void warp_search_over(const float4* __restrict__ nodes, const float4* __restrict__ tris,
                                                 V3 p, int4 start, WarpBest& b, int2* work) {
  const int lane = threadIdx.x & 31;
  b.dropped = 0;
  b.nodes = b.tris = 0;
  if (lane == 0) {
    work[0] = make_int2(start.y, __float_as_int(0.0f));
    work[1] = make_int2(start.z, __float_as_int(0.0f));
    work[2] = make_int2(start.w, __float_as_int(0.0f));
  }
  int sp = 3;  // warp-uniform
  __syncwarp();
  while (sp > 0) {
    const int take = min(min(sp, 32), max((kWarpList - kWarpReserve - sp) >> 2, 1));  // sp + 3 take spares the reserve
    int2 e = make_int2(kEmptyChild, 0);
    if (lane < take) e = work[sp - take + lane];
    __syncwarp();
    sp -= take;
    const float bound = kBoxes ? key_d2(b.key) : prune_limit(key_d2(b.key), p);
    int2 c[4];
    int nc = 0;
    if (e.x != kEmptyChild && __int_as_float(e.y) <= bound) {
      if (e.x >= 0) {
        ++b.nodes;
        float d[4];
        int4 ch;
        if constexpr (kBoxes) {
          ch = box_distances(nodes, e.x, p, d);
        } else {
          const FrameData f = load_frame_node(nodes, e.x);
          frame_distances(f, p, d);
          ch = f.ch;
        }
        const int r[4] = {ch.x, ch.y, ch.z, ch.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          c[k] = make_int2(r[k], __float_as_int(d[k]));
          if (r[k] == kEmptyChild || !(d[k] <= bound)) c[k].x = kEmptyChild;
          nc += c[k].x != kEmptyChild ? 1 : 0;
        }
      } else {
        const int first = leaf_first(e.x), count = leaf_count(e.x);
        for (int i = 0; i < count; ++i) {
          ClosestHit h;
          h.d2 = h.lim = FLT_MAX;
          h.id = INT32_MAX;
          h.slot = 0;
          h.cp = p;
          test_slot(tris, first + i, p, h);
          ++b.tris;
          const unsigned long long k = hit_key(h.d2, h.id);
          if (k < b.mine) {
            b.mine = k;
            b.cp = h.cp;
            b.slot = h.slot;
          }
        }
      }
    }
    unsigned long long wk = b.mine;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) wk = min(wk, __shfl_xor_sync(0xffffffffu, wk, o));
    b.key = min(b.key, wk);
    // append this iteration's children in lane order
    int incl = nc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    int at = sp + incl - nc;
    if (nc > 0) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (c[k].x != kEmptyChild) {
          if (at < kWarpList) work[at] = c[k];
          ++at;
        }
      }
    }
    if (sp + total > kWarpList) b.dropped = 1;
    sp = min(sp + total, kWarpList);
    __syncwarp();
  }
}

template <bool kFramesOnly>
__device__ __forceinline__ void warp_search(const QueryNodes& nodes, const float4* __restrict__ tris, V3 p, int4 start,
                                            bool far, WarpBest& b, int2* work) {
  if (!kFramesOnly && (nodes.use_boxes || far)) warp_search_over<true>(nodes.boxes, tris, p, start, b, work);
  else warp_search_over<false>(nodes.frames, tris, p, start, b, work);
}

// A cold query, seeded and started by the grid if there is one.  kFramesOnly: without the
// search over boxes, for trees over frames, far points included.
template <bool kFramesOnly>
__device__ __forceinline__ WarpBest warp_query(const QueryNodes& nodes, const float4* __restrict__ tris,
                                               const SeedGrid& grid, V3 p, int root, V3 no_hit, int2* work) {
  ClosestHit h;
  h.d2 = h.lim = FLT_MAX;
  h.id = INT32_MAX;
  h.slot = -1;
  h.cp = no_hit;
  int4 cell = make_int4(0, root, kEmptyChild, kEmptyChild);
  bool far = false;
  if (grid.cells) {
    cell = kFramesOnly ? seed_cell_any(grid, p, root, far) : nodes.seed(grid, p, root, far);
    test_slot(tris, cell.x, p, h);
  }
  WarpBest b;
  b.key = b.mine = hit_key(h.d2, h.id);
  b.cp = h.cp;
  b.slot = h.slot;
  warp_search<kFramesOnly>(nodes, tris, p, cell, far, b, work);
  if (grid.cells && (threadIdx.x & 31) == 0) ++b.tris;
  return b;
}

}  // namespace dev
}  // namespace n2w
