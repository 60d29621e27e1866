// Device layout of the 4-wide BVH and the leaf-ordered triangle array.
//
// Node (128 B, one L2 line): six float4 rows hold the four child boxes in
// structure-of-arrays form (lo.x, hi.x, lo.y, hi.y, lo.z, hi.z), one int4 row
// holds the child references, the last 16 B are padding.
//
// Child reference r:  r >= 0      inner node index
//                     r == kEmpty  unused slot (its box is +inf/-inf)
//                     otherwise    leaf: ~r = (first_triangle << 3) | (count - 1)
//
// Triangle (48 B): three float4 rows (v0.xyz, original id as int bits),
// (v1.xyz, 0), (v2.xyz, 0).  Triangles are permuted into leaf order, so a leaf
// is a contiguous run; the original id is kept for results and tie-breaking.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define N2W_HD __host__ __device__ __forceinline__
#else
#define N2W_HD inline
#endif

namespace n2w {

constexpr int32_t kEmptyChild = INT32_MIN;
constexpr int kMaxLeafSize = 8;
constexpr int kTraversalStack = 64;
constexpr int kSeedGridCells = 128;  // seed-grid cells per axis

struct alignas(128) Node4 {
  float lo_x[4];
  float hi_x[4];
  float lo_y[4];
  float hi_y[4];
  float lo_z[4];
  float hi_z[4];
  int32_t child[4];
  int32_t pad[4];
};
static_assert(sizeof(Node4) == 128, "Node4 must be one 128-byte line");

// The same 4-wide node in 64 bytes (two sectors), with its child boxes in a frame
// of its own: the mirror image q = p - v (v.p) with |v|^2 = 2, chosen so that the
// patch of surface below the node lies flat against an axis (v.z >= 0 follows
// from v.x and v.y).  A mirror is an isometry, so distances to the boxes are
// distances in space.  Boxes around a flat patch in such a frame are thin where
// axis-aligned ones are not, so far fewer children lie within a query's best
// distance.  Box planes are o + b 2^e with a byte b per child and a power of two
// per axis (b rounded outwards).  Against 128 bytes with 32-bit planes, whose two
// further sectors kept L2 and the L1 data pipe over half busy: 4,194,304 / 262,144
// uniform queries 4.21 -> 3.62 ms / 357 -> 313 us, Laplace and Poisson walks 16.9 ->
// 15.1 and 41.5 -> 38.6 ms, batched instances 34.1 -> 31.3 ms.
struct alignas(64) FrameNode4 {
  float vx, vy;
  float o[3];
  uint32_t exps;      // biased exponents e + 127 of the axes' steps in bytes 0..2
  uint32_t plane[6];  // lo x, hi x, lo y, hi y, lo z, hi z: byte k for child k
  int32_t child[4];
};
static_assert(sizeof(FrameNode4) == 64, "FrameNode4 must be two 32-byte sectors");

struct alignas(16) TriRec {
  float v0[3];
  int32_t id;
  float v1[3];
  int32_t pad1;
  float v2[3];
  int32_t pad2;
};
static_assert(sizeof(TriRec) == 48, "TriRec must be 48 bytes");

// A triangle as the closest-point test reads it: corner a with the original id,
// the edges ab = b - a and ac = c - a (rounded once, as the test would round
// them) and the corners b and c.  64 bytes, two aligned 256-bit loads.
struct alignas(64) TriEdges {
  float a[3];
  int32_t id;
  float ab[3];
  float ac[3];
  float b[3];
  float c[3];
};
static_assert(sizeof(TriEdges) == 64, "TriEdges must be two 32-byte sectors");

N2W_HD int32_t leaf_ref(int32_t first, int32_t count) { return ~((first << 3) | (count - 1)); }
N2W_HD bool ref_is_leaf(int32_t r) { return r < 0 && r != kEmptyChild; }
N2W_HD int32_t leaf_first(int32_t r) { return (~r) >> 3; }
N2W_HD int32_t leaf_count(int32_t r) { return ((~r) & 7) + 1; }

}  // namespace n2w
