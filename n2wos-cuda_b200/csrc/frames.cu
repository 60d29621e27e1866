// Builds the FrameNode4 array (layout.h) and the seed grid's start subtrees on
// the device from the uploaded 4-wide nodes and leaf-ordered triangles.
//
// Each node tries seven frames: the axes, and the mirrors that carry the
// area-weighted mean normal of the triangles below it onto +-x, +-y or +-z.
// It keeps the one whose four child boxes have the least summed area; a box
// around a flat patch is thin along the patch's normal in such a frame.  Along
// walks on the displaced icosphere (81,920 triangles) this cuts a query from
// 26.5 node expansions and 20.5 triangle tests to 18.0 and 7.7; principal axes
// of the patch give the same (18.1 and 7.7) but take 18 operations per node
// and a fourth number, the mirror takes 6 and three.  Measured against the
// axis-aligned nodes: 262,144 uniform queries 1,120 -> 428 us, 20,011 points x
// 101 Laplace walks 56.9 -> 28.4 ms, the results the same bits.
//
// One warp per node: the nodes below ~4,096 triangles hold the work (every
// level reads each triangle once per candidate), and larger patches are curved
// too far for a frame to matter, so they keep the axes and the boxes they have.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "geom.cuh"
#include "internal.hpp"

namespace n2w {
namespace {

constexpr int kFrameBlock = 128;
constexpr int kFrameMaxTris = 4096;
constexpr int kFrameCandidates = 7;
constexpr float kFrameFar = 1.0e30f;

__device__ __forceinline__ float warp_min(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fminf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}
__device__ __forceinline__ float warp_max(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}
__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

__device__ __forceinline__ dev::V3 vertex(const float4* tris, int t, int k) {
  const float4 a = __ldg(tris + static_cast<size_t>(t) * 3 + k);
  return dev::v3(a.x, a.y, a.z);
}

// Bounds of triangles [first, last) in frame v, the same in every lane.
__device__ __forceinline__ void frame_bounds(const float4* tris, int first, int last, dev::V3 v, float* lo, float* hi) {
  for (int a = 0; a < 3; ++a) {
    lo[a] = INFINITY;
    hi[a] = -INFINITY;
  }
  for (int i = 3 * first + static_cast<int>(threadIdx.x & 31); i < 3 * last; i += 32) {
    const dev::V3 q = dev::to_frame(v, vertex(tris, i / 3, i % 3));
    lo[0] = fminf(lo[0], q.x);
    lo[1] = fminf(lo[1], q.y);
    lo[2] = fminf(lo[2], q.z);
    hi[0] = fmaxf(hi[0], q.x);
    hi[1] = fmaxf(hi[1], q.y);
    hi[2] = fmaxf(hi[2], q.z);
  }
  for (int a = 0; a < 3; ++a) {
    lo[a] = warp_min(lo[a]);
    hi[a] = warp_max(hi[a]);
  }
}

// Candidate c >= 1: the mirror that carries the unit vector n onto an axis.
// Undefined (false) where n is that axis already or not a number.
__device__ __forceinline__ bool mirror_onto(dev::V3 n, int c, dev::V3& v) {
  const int axis = (c - 1) % 3;
  const float e = c <= 3 ? 1.0f : -1.0f;
  const dev::V3 w = dev::v3(n.x - (axis == 0 ? e : 0.0f), n.y - (axis == 1 ? e : 0.0f), n.z - (axis == 2 ? e : 0.0f));
  const float l2 = w.x * w.x + w.y * w.y + w.z * w.z;
  if (!(l2 > 1.0e-8f)) return false;
  const float s = sqrtf(2.0f / l2);
  const float sign = w.z < 0.0f ? -s : s;  // v and -v are the same mirror
  v = dev::frame_v(w.x * sign, w.y * sign);
  return true;
}

__global__ void __launch_bounds__(kFrameBlock) frame_nodes_kernel(const Node4* __restrict__ nodes,
                                                                  const TriRange* __restrict__ ranges,
                                                                  const float4* __restrict__ tris, int n,
                                                                  FrameNode4* __restrict__ out) {
  const int node = static_cast<int>((static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (node >= n) return;
  const Node4& nd = nodes[node];
  const TriRange r = ranges[node];
  dev::V3 v = dev::frame_v(0.0f, 0.0f);  // the axes, z mirrored
  float pad = 0.0f;
  int first[4], last[4];
  for (int k = 0; k < 4; ++k) {
    const int c = nd.child[k];
    first[k] = c == kEmptyChild ? 0 : (c >= 0 ? ranges[c].first : leaf_first(c));
    last[k] = c == kEmptyChild ? 0 : (c >= 0 ? ranges[c].last : leaf_first(c) + leaf_count(c));
  }
  float lo[4][3], hi[4][3];
  bool small = r.last - r.first <= kFrameMaxTris;
  if (small) {
    // a frame's arithmetic needs finite coordinates with finite squares
    float far = 0.0f;
    for (int k = 0; k < 4; ++k) {
      if (nd.child[k] == kEmptyChild) continue;
      far = fmaxf(far, fmaxf(fmaxf(fabsf(nd.lo_x[k]), fabsf(nd.hi_x[k])),
                             fmaxf(fmaxf(fabsf(nd.lo_y[k]), fabsf(nd.hi_y[k])), fmaxf(fabsf(nd.lo_z[k]), fabsf(nd.hi_z[k])))));
    }
    small = far < 1.0e18f;
  }
  if (small) {
    float nx = 0.0f, ny = 0.0f, nz = 0.0f, big = 0.0f;
    for (int t = r.first + lane; t < r.last; t += 32) {
      const dev::V3 a = vertex(tris, t, 0), b = vertex(tris, t, 1), c = vertex(tris, t, 2);
      const dev::V3 e = dev::v3(b.x - a.x, b.y - a.y, b.z - a.z), f = dev::v3(c.x - a.x, c.y - a.y, c.z - a.z);
      nx += e.y * f.z - e.z * f.y;
      ny += e.z * f.x - e.x * f.z;
      nz += e.x * f.y - e.y * f.x;
      big = fmaxf(big, fmaxf(fabsf(a.x) + fabsf(a.y) + fabsf(a.z),
                             fmaxf(fabsf(b.x) + fabsf(b.y) + fabsf(b.z), fabsf(c.x) + fabsf(c.y) + fabsf(c.z))));
    }
    nx = warp_sum(nx);
    ny = warp_sum(ny);
    nz = warp_sum(nz);
    pad = warp_max(big);
    const float len = sqrtf(nx * nx + ny * ny + nz * nz);
    const dev::V3 nrm = dev::v3(nx / len, ny / len, nz / len);
    float best = INFINITY;
    for (int c = 0; c < kFrameCandidates; ++c) {
      dev::V3 w = dev::frame_v(0.0f, 0.0f);
      if (c > 0 && (!(len > 0.0f) || !mirror_onto(nrm, c, w))) continue;
      float cost = 0.0f;
      for (int k = 0; k < 4; ++k) {
        if (first[k] >= last[k]) continue;
        frame_bounds(tris, first[k], last[k], w, lo[k], hi[k]);
        const float ex = hi[k][0] - lo[k][0], ey = hi[k][1] - lo[k][1], ez = hi[k][2] - lo[k][2];
        cost += ex * ey + ey * ez + ez * ex;
      }
      if (cost < 0.98f * best) {  // the axes stand unless a frame is clearly better
        best = cost;
        v = w;
      }
    }
    for (int k = 0; k < 4; ++k) {
      if (first[k] < last[k]) frame_bounds(tris, first[k], last[k], v, lo[k], hi[k]);
    }
  } else {
    // the boxes that the node has, z mirrored
    for (int k = 0; k < 4; ++k) {
      lo[k][0] = nd.lo_x[k];
      hi[k][0] = nd.hi_x[k];
      lo[k][1] = nd.lo_y[k];
      hi[k][1] = nd.hi_y[k];
      lo[k][2] = -nd.hi_z[k];
      hi[k][2] = -nd.lo_z[k];
      if (nd.child[k] == kEmptyChild) continue;
      for (int a = 0; a < 3; ++a) pad = fmaxf(pad, 3.0f * fmaxf(fabsf(lo[k][a]), fabsf(hi[k][a])));
    }
  }
  // 2^-19 of the largest |vertex|_1: 8 u of the frame's rounding plus the
  // closest-point arithmetic's few u, twice over (u = 2^-24)
  const float big1 = fminf(pad, kFrameFar);
  pad = pad * 1.9073486328125e-06f + 1e-30f;
  // Planes end at kFrameFar, where a step's multiples are still finite; whatever lies
  // beyond has no finite squared distance to any point that has one to anything.
  for (int k = 0; k < 4; ++k) {
    for (int a = 0; a < 3; ++a) {
      lo[k][a] = fminf(fmaxf(lo[k][a] - pad, -kFrameFar), kFrameFar);
      hi[k][a] = fminf(fmaxf(hi[k][a] + pad, -kFrameFar), kFrameFar);
    }
  }
  FrameNode4 o;
  o.vx = v.x;
  o.vy = v.y;
  o.exps = 0;
  for (int a = 0; a < 3; ++a) {
    float omin = INFINITY, omax = -INFINITY;
    for (int k = 0; k < 4; ++k) {
      if (nd.child[k] == kEmptyChild) continue;
      omin = fminf(omin, lo[k][a]);
      omax = fmaxf(omax, hi[k][a]);
    }
    // The step: a power of two with the children within 253 of them, at least
    // 2^-20 of the coordinates so the origin's rounding is a fraction of it.
    const float want = fmaxf((omax - omin) / 253.0f, fmaxf(big1 * 9.5367431640625e-07f, 1.0e-35f));
    int e = 0;
    frexpf(want, &e);  // want <= 2^e
    e = min(max(e, -120), 120);
    const float step = ldexpf(1.0f, e);
    const float origin = omin - step;
    o.o[a] = origin;
    o.exps |= static_cast<uint32_t>(e + 127) << (8 * a);
    uint32_t wl = 0, wh = 0;
    for (int k = 0; k < 4; ++k) {
      if (nd.child[k] == kEmptyChild) continue;
      // outwards by a quarter of a step, for the origin's and the quotient's rounding
      const float bl = floorf((lo[k][a] - origin) / step - 0.25f);
      const float bh = ceilf((hi[k][a] - origin) / step + 0.25f);
      wl |= static_cast<uint32_t>(fminf(fmaxf(bl, 0.0f), 255.0f)) << (8 * k);
      wh |= static_cast<uint32_t>(fminf(fmaxf(bh, 0.0f), 255.0f)) << (8 * k);
    }
    o.plane[2 * a] = wl;
    o.plane[2 * a + 1] = wh;
  }
  for (int k = 0; k < 4; ++k) o.child[k] = nd.child[k];
  if (lane == 0) out[node] = o;
}

// Start subtrees of one seed-grid cell (geom.cuh SeedGrid).  For a point x of the
// cell, a cube of half-width `half` around the lattice node c, the closest
// triangle is within D = d(c) + |x - c| <= d(c) + sqrt(3) half, so it lies in a
// box only if the box is within D of the cube and within d(c) + 2 sqrt(3) half
// of c, both widened by the rounding of d.  Starting from the root, entries are
// replaced by their children that pass both tests while they fit, so nothing that could
// be closest is left out.
// Three subtrees: 18.0 -> 14.1 expansions per walk query (one: 16.2, two: 15.0;
// more are visited in vain: eight 13.7 and 20 % more triangle tests), and the
// cell stays one 16-byte load.
__global__ void __launch_bounds__(256) cell_entries_kernel(const float4* __restrict__ frames,
                                                           const float4* __restrict__ tris, float lox, float loy,
                                                           float loz, float h, int n, int4* __restrict__ cells) {
  const int s = n + 1;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= static_cast<int64_t>(s) * s * s) return;
  const int ix = static_cast<int>(i % s), iy = static_cast<int>((i / s) % s),
            iz = static_cast<int>(i / (static_cast<int64_t>(s) * s));
  const dev::V3 c = dev::v3(lox + h * static_cast<float>(ix), loy + h * static_cast<float>(iy),
                            loz + h * static_cast<float>(iz));
  dev::ClosestHit hit;
  hit.d2 = hit.lim = FLT_MAX;
  hit.id = INT32_MAX;
  hit.slot = 0;
  hit.cp = c;
  const int slot = cells[i].x;
  dev::test_slot(tris, slot, c, hit);
  // The cube is grown by 0.1 % and the coordinates' rounding: a point is
  // assigned to its lattice node with an error of a few u |coordinate| / h.
  const float scale = fabsf(c.x) + fabsf(c.y) + fabsf(c.z);
  const float half = 0.5005f * h + 4.0e-6f * scale, r = 1.7320509f * half;
  const float d = sqrtf(hit.d2);
  // d(x) is a computed distance.  With edges up to L, height w over the longest and
  // corners within D of x, the test's dot products are off by 5 u L D, its barycentric
  // numerators by 23 u (L D)^2, its denominator (L w)^2 by three times that, so the point by
  // 115 u D^2 / w^2 of L, here and at the lattice node.  Where that is no longer small (a
  // sliver, whose test may even divide by zero) the cell keeps the root.
  const dev::Rec64 t = dev::load_rec<false>(tris, slot);
  const dev::V3 ab = dev::v3(t.r1.x, t.r1.y, t.r1.z), ac = dev::v3(t.r1.w, t.r2.x, t.r2.y),
                bc = dev::vsub(ac, ab);
  const dev::V3 nrm = dev::v3(ab.y * ac.z - ab.z * ac.y, ab.z * ac.x - ab.x * ac.z, ab.x * ac.y - ab.y * ac.x);
  const float edge2 = fmaxf(dev::vdot(ab, ab), fmaxf(dev::vdot(ac, ac), dev::vdot(bc, bc)));
  const float height2 = dev::vdot(nrm, nrm) / edge2, corner = d + 2.0f * r + sqrtf(edge2);
  const float off = 1.52587890625e-05f * corner * corner / height2;  // 2 x 128 u
  if (!(off < 0.25f)) return;
  const float reach = d + r + off * sqrtf(edge2);
  const float lim_c = dev::prune_limit((reach + r) * (reach + r), c);
  const float lim_q = dev::prune_limit(reach * reach, c);
  int e[dev::kCellEntries] = {0, kEmptyChild, kEmptyChild};
  int count = 1;
  if (hit.id != INT32_MAX) {
    for (bool changed = true; changed;) {
      changed = false;
      for (int j = 0; j < count; ++j) {
        if (e[j] < 0) continue;
        const dev::FrameData f = dev::load_frame_node(frames, e[j]);
        const dev::V3 v = f.v, m = dev::to_frame(v, c);
        const float q[3] = {m.x - f.o.x, m.y - f.o.y, m.z - f.o.z};
        // half extents of the cube in the frame
        const float ext[3] = {half * (fabsf(1.0f - v.x * v.x) + fabsf(v.x * v.y) + fabsf(v.x * v.z)),
                              half * (fabsf(v.y * v.x) + fabsf(1.0f - v.y * v.y) + fabsf(v.y * v.z)),
                              half * (fabsf(v.z * v.x) + fabsf(v.z * v.y) + fabsf(1.0f - v.z * v.z))};
        const int kids[4] = {f.ch.x, f.ch.y, f.ch.z, f.ch.w};
        int keep[4], nk = 0;
        for (int k = 0; k < 4; ++k) {
          if (kids[k] == kEmptyChild) continue;
          float dc = 0.0f, dq = 0.0f;
          for (int a = 0; a < 3; ++a) {
            const float l = f.step[a] * static_cast<float>((f.plane[2 * a] >> (8 * k)) & 255u);
            const float u = f.step[a] * static_cast<float>((f.plane[2 * a + 1] >> (8 * k)) & 255u);
            const float gc = q[a] - fminf(fmaxf(q[a], l), u);
            const float gq = q[a] - fminf(fmaxf(q[a], l - ext[a]), u + ext[a]);
            dc += gc * gc;
            dq += gq * gq;
          }
          if (dc <= lim_c && dq <= lim_q) keep[nk++] = kids[k];
        }
        if (nk == 0 || count - 1 + nk > dev::kCellEntries) continue;
        e[j] = keep[0];
        for (int k = 1; k < nk; ++k) e[count++] = keep[k];
        changed = true;
      }
    }
  }
  cells[i] = make_int4(slot, e[0], e[1], e[2]);
}

__global__ void __launch_bounds__(256) edges_kernel(const TriRec* __restrict__ tris, int64_t n,
                                                    TriEdges* __restrict__ out) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const TriRec t = tris[i];
  TriEdges o;
  o.id = t.id;
  for (int k = 0; k < 3; ++k) {
    o.a[k] = t.v0[k];
    o.b[k] = t.v1[k];
    o.c[k] = t.v2[k];
    o.ab[k] = __fsub_rn(t.v1[k], t.v0[k]);
    o.ac[k] = __fsub_rn(t.v2[k], t.v0[k]);
  }
  out[i] = o;
}

}  // namespace

void build_cell_entries(n2w_bvh& b) {
  const int64_t s = b.seed_n + 1, total = s * s * s;
  cell_entries_kernel<<<static_cast<unsigned>((total + 255) / 256), 256>>>(
      reinterpret_cast<const float4*>(b.d_frames), reinterpret_cast<const float4*>(b.d_edges), b.seed_lo[0],
      b.seed_lo[1], b.seed_lo[2], b.seed_h, b.seed_n, b.d_seed);
  N2W_CUDA(cudaGetLastError());
}

// Plain copies of whole cells: the BVH may be on another device than the current one,
// and the device may have no memory left.
void copy_cell_slots(const n2w_bvh& b, int64_t n, int* out) {
  constexpr int64_t kChunk = 1 << 17;
  std::vector<int4> cells(static_cast<size_t>(std::min(n, kChunk)));
  for (int64_t i = 0; i < n; i += kChunk) {
    const int64_t m = std::min(n - i, kChunk);
    N2W_CUDA(cudaMemcpy(cells.data(), b.d_seed + i, sizeof(int4) * static_cast<size_t>(m), cudaMemcpyDeviceToHost));
    for (int64_t k = 0; k < m; ++k) out[i + k] = cells[static_cast<size_t>(k)].x;
  }
}

void build_edges(n2w_bvh& b, int64_t triangles) {
  N2W_CUDA(cudaMalloc(&b.d_edges, sizeof(TriEdges) * static_cast<size_t>(triangles)));
  edges_kernel<<<static_cast<unsigned>((triangles + 255) / 256), 256>>>(b.d_tris, triangles, b.d_edges);
  N2W_CUDA(cudaGetLastError());
}

void build_frames(n2w_bvh& b, const HostBvh& h) {
  const int n = static_cast<int>(h.nodes.size());
  N2W_CUDA(cudaMalloc(&b.d_frames, sizeof(FrameNode4) * h.nodes.size()));
  TriRange* d_ranges = nullptr;
  N2W_CUDA(cudaMalloc(&d_ranges, sizeof(TriRange) * h.ranges.size()));
  const cudaError_t e =
      cudaMemcpy(d_ranges, h.ranges.data(), sizeof(TriRange) * h.ranges.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    const int64_t threads = static_cast<int64_t>(n) * 32;
    frame_nodes_kernel<<<static_cast<unsigned>((threads + kFrameBlock - 1) / kFrameBlock), kFrameBlock>>>(
        b.d_nodes, d_ranges, reinterpret_cast<const float4*>(b.d_tris), n, b.d_frames);
  }
  const cudaError_t l = cudaGetLastError();
  cudaFree(d_ranges);  // waits for the kernel
  N2W_CUDA(e);
  N2W_CUDA(l);
}

}  // namespace n2w
