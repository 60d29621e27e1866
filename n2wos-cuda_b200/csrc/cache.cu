// Neural cache: multiresolution hash-grid encoding + small ReLU MLP, trained
// online with Adam.  Replaces tiny-cuda-nn's HashGrid + FullyFusedMLP + Adam
// as used by the reference (src/tools/eval_tcnn_nc_wos.cu:747-750,759).
//
// Encoding (Mueller, Evans, Schied, Keller, "Instant Neural Graphics
// Primitives with a Multiresolution Hash Encoding", SIGGRAPH 2022): level l has
// resolution N_l = floor(N_min * b^l); a point x in [0,1]^3 is scaled by N_l,
// its 8 lattice corners are looked up densely while (N_l+1)^3 fits the level's
// table and through the spatial hash (x*1 ^ y*2654435761 ^ z*805459861) mod T
// otherwise, and the F features are trilinearly interpolated.
//
// MLP: inputs L*F (= 32 for 16 levels x 2), hidden width W in {16, 32, 64},
// H hidden layers, scalar output, ReLU, no output activation.  FP16 weights
// and activations on mma.sync.m16n8k16 with FP32 accumulation; FP32 master
// parameters and Adam moments.
//
// Warp tiling: a warp owns 16 samples.  Lane (g = lane/4, c = lane%4) holds
// rows g and g+8 of every fragment.  It computes the encoding of exactly the
// (sample, level) pairs its layer-1 A fragment needs — levels c, c+4, c+8,
// c+12 of samples g and g+8 — so features go straight into registers; each
// layer's FP32 C fragments become the next layer's FP16 A fragments in place;
// in the backward pass dX arrives in the same (sample, level) ownership, so the
// grid-gradient scatter needs no reshuffle.  Weight fragments come from shared
// memory by ldmatrix (transposed for the backward products); rows are padded by
// 8 halves, so the eight rows of a matrix lie in different banks.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <fstream>
#include <string>
#include <vector>

#include "internal.hpp"
#include "philox.cuh"

namespace n2w {
namespace {

constexpr int kMaxLevels = 16;
constexpr int kMaxHidden = 4;
constexpr int kTrainBlock = 128;  // 4 warps
constexpr int kTrainRound = 64;   // samples staged per block round

constexpr int kPad = 8;           // halves added to every row in shared memory

struct GridMeta {
  int levels;
  int features;  // fixed to 2
  uint32_t table_size[kMaxLevels];
  uint32_t offset[kMaxLevels];  // entry offset of each level
  float scale[kMaxLevels];      // N_l
  uint32_t res[kMaxLevels];     // N_l
  uint32_t dense[kMaxLevels];   // 1 = dense indexing
};

// One level as the kernels index it.  Entry of lattice corner (x, y, z):
// dense x + y ymul + z zmul, else (x ^ y ymul ^ z zmul) mod T with T a power of two.
struct alignas(8) Level {
  float scale;
  uint32_t offset, ymul, zmul;
  uint32_t mask;
  uint32_t dense;
};

struct MlpMeta {
  int width;   // 16 / 32 / 64
  int hidden;  // hidden layers
  int in_dim;  // 16 or 32 (levels*2 padded to 16)
  // parameter offsets (elements) inside the MLP block
  int w_in;                // [width x in_dim]
  int w_hid[kMaxHidden];   // [width x width], hidden-1 of them used
  int w_out;               // [width] (output row)
  int total;
};

constexpr uint32_t kHashY = 2654435761u, kHashZ = 805459861u;

// The levels into shared memory (lanes of a warp work on different levels).
__device__ __forceinline__ void stage_levels(const GridMeta& g, Level* sl) {
  const int l = threadIdx.x;
  if (l < kMaxLevels) {
    const uint32_t s = g.res[l] + 1;
    sl[l] = Level{g.scale[l],
                  g.offset[l],
                  g.dense[l] ? s : kHashY,
                  g.dense[l] ? s * s : kHashZ,
                  g.dense[l] ? 0xffffffffu : g.table_size[l] - 1u,
                  g.dense[l]};
  }
}

// The eight corners of the cell of input u in [0,1]^3 on one level.  Corners
// come in pairs along x (dx = 0, 1); pair t has dy = t & 1, dz = t >> 1.
struct Corners {
  uint32_t x, yz[4];
  float w[3];  // fractional parts
  __device__ __forceinline__ uint32_t index(const Level& l, int t, uint32_t dx) const {
    return l.dense ? x + dx + yz[t] : ((x + dx) ^ yz[t]) & l.mask;
  }
  __device__ __forceinline__ float weight(int t, int dx) const {
    return (dx ? w[0] : 1.0f - w[0]) * ((t & 1) ? w[1] : 1.0f - w[1]) * ((t >> 1) ? w[2] : 1.0f - w[2]);
  }
};

__device__ __forceinline__ Corners level_corners(const Level& l, float ux, float uy, float uz) {
  Corners c;
  const float s = l.scale;
  const float px = ux * s, py = uy * s, pz = uz * s;
  const float fx = floorf(px), fy = floorf(py), fz = floorf(pz);
  const float lim = s - 1.0f;
  const float cx = fminf(fmaxf(fx, 0.0f), lim), cy = fminf(fmaxf(fy, 0.0f), lim), cz = fminf(fmaxf(fz, 0.0f), lim);
  c.x = static_cast<uint32_t>(cx);
  const uint32_t y0 = static_cast<uint32_t>(cy) * l.ymul, z0 = static_cast<uint32_t>(cz) * l.zmul;
  const uint32_t y1 = y0 + l.ymul, z1 = z0 + l.zmul;
  c.yz[0] = l.dense ? y0 + z0 : y0 ^ z0;
  c.yz[1] = l.dense ? y1 + z0 : y1 ^ z0;
  c.yz[2] = l.dense ? y0 + z1 : y0 ^ z1;
  c.yz[3] = l.dense ? y1 + z1 : y1 ^ z1;
  c.w[0] = px - cx;
  c.w[1] = py - cy;
  c.w[2] = pz - cz;
  return c;
}

// Encoded feature pair (F = 2) of one (sample, level).  The two corners of a
// pair are neighbours in an aligned 8 bytes whenever x is even on a hashed
// level (the hash leaves x's last bit last) or the entry is even on a dense
// one, i.e. half of the time: each pair is one 8-byte load and, for the other
// half of the lanes, a 4-byte one (levels start at multiples of 8 entries).
// The gathers and their index arithmetic bound inference: 4,000,000 inputs
// 2,278 -> 1,639 us with the pairs, the modulus as a mask and conflict-free
// weight fragments (the default network; the same bits).
__device__ __forceinline__ float2 encode_level(const Level& l, const __half2* __restrict__ table, float ux, float uy,
                                               float uz) {
  const Corners c = level_corners(l, ux, uy, uz);
  const uint32_t* t32 = reinterpret_cast<const uint32_t*>(table + l.offset);
  uint2 e[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const uint32_t i0 = c.index(l, t, 0), i1 = c.index(l, t, 1);
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(t32) + (i0 >> 1));
    e[t].x = (i0 & 1u) ? v.y : v.x;
    e[t].y = (i0 & 1u) ? v.x : v.y;
    if (i1 != (i0 ^ 1u)) e[t].y = __ldg(t32 + i1);
  }
  float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t bits = (k & 1) ? e[k >> 1].y : e[k >> 1].x;
    const float w = c.weight(k >> 1, k & 1);
    const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&bits));
    acc.x += w * v.x;
    acc.y += w * v.y;
  }
  return acc;
}

__device__ __forceinline__ void red_add(float2* p, float2 v) {
  asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void red_add(float4* p, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}

// Gradient of encode_level: the neighbouring pairs go out as one 16-byte reduction.
__device__ __forceinline__ void scatter_level(const Level& l, float2* __restrict__ grad, float ux, float uy, float uz,
                                              float2 d) {
  const Corners c = level_corners(l, ux, uy, uz);
  float2* g = grad + l.offset;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const uint32_t i0 = c.index(l, t, 0), i1 = c.index(l, t, 1);
    const float w0 = c.weight(t, 0), w1 = c.weight(t, 1);
    const float2 a = make_float2(w0 * d.x, w0 * d.y), b = make_float2(w1 * d.x, w1 * d.y);
    if (i1 == (i0 ^ 1u)) {
      const bool odd = i0 & 1u;
      red_add(reinterpret_cast<float4*>(g + (i0 & ~1u)),
              odd ? make_float4(b.x, b.y, a.x, a.y) : make_float4(a.x, a.y, b.x, b.y));
    } else {
      red_add(g + i0, a);
      red_add(g + i1, b);
    }
  }
}

__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ float2 unpack_h2(uint32_t u) {
  return __half22float2(*reinterpret_cast<const __half2*>(&u));
}

// D = A(16x16 f16, row) * B(16x8 f16, col) + C (f32).
__device__ __forceinline__ void mma16816(float* d, const uint32_t* a, const uint32_t* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Four 8x8 half matrices from shared memory; lane i gives the address of row
// i % 8 of matrix i / 8.  Plain: lane (g,c) receives elements (row g, columns
// 2c, 2c+1) of each; transposed: (rows 2c, 2c+1, column g).
__device__ __forceinline__ void ldsm4(uint32_t* r, const __half* p) {
  const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t* r, const __half* p) {
  const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}

// B fragments of the n-tiles at n0 and n0 + 8 for k-step k0, from a row-major
// matrix M with leading dimension ld: b_rows for B[k][n] = M[n][k] (forward,
// W [out x in]), b_cols for B[k][n] = M[k][n].
__device__ __forceinline__ void b_rows(uint32_t* b, const __half* M, int ld, int n0, int k0, int lane) {
  ldsm4(b, M + (n0 + (lane & 7) + ((lane & 16) >> 1)) * ld + k0 + (lane & 8));
}
__device__ __forceinline__ void b_cols(uint32_t* b, const __half* M, int ld, int n0, int k0, int lane) {
  ldsm4_t(b, M + (k0 + (lane & 15)) * ld + n0 + ((lane & 16) >> 1));
}
// A fragment A[m][k] = M[k][m] of the m-tile at m0 for k-step k0.
__device__ __forceinline__ void a_cols(uint32_t* a, const __half* M, int ld, int m0, int k0, int lane) {
  ldsm4_t(a, M + (k0 + (lane & 7) + ((lane & 16) >> 1)) * ld + m0 + (lane & 8));
}

// C fragments of n-tiles (2t, 2t+1) -> A fragment of k-step t, with ReLU.
__device__ __forceinline__ void c_to_a_relu(uint32_t* a, const float* c0, const float* c1) {
  a[0] = pack_h2(fmaxf(c0[0], 0.0f), fmaxf(c0[1], 0.0f));
  a[1] = pack_h2(fmaxf(c0[2], 0.0f), fmaxf(c0[3], 0.0f));
  a[2] = pack_h2(fmaxf(c1[0], 0.0f), fmaxf(c1[1], 0.0f));
  a[3] = pack_h2(fmaxf(c1[2], 0.0f), fmaxf(c1[3], 0.0f));
}

__device__ __forceinline__ void c_to_a(uint32_t* a, const float* c0, const float* c1) {
  a[0] = pack_h2(c0[0], c0[1]);
  a[1] = pack_h2(c0[2], c0[3]);
  a[2] = pack_h2(c1[0], c1[1]);
  a[3] = pack_h2(c1[2], c1[3]);
}

struct NetArgs {
  GridMeta grid;
  MlpMeta mlp;
  const __half2* table;   // fp16 grid features
  const __half* mlp_h;    // fp16 MLP weights
  float2* grid_grad;      // fp32 grid gradient accumulators
  float* mlp_grad;        // fp32 MLP gradient accumulators
  const float* inputs;    // [n x 3], unit cube
  const float* targets;   // [n]
  float* outputs;         // [n]
  int64_t n;
  float loss_scale;       // dL/dy = loss_scale * (y - t)
  float grad_scale;       // factor of every gradient added to the accumulators
  float* loss_sum;        // optional: sum of (y - t)^2
};

// The MLP weights in shared memory, rows padded: w_in [W x (IN + kPad)], the
// hidden matrices [W x (W + kPad)], w_out [W].
template <int W, int KS, int H>
struct Weights {
  static constexpr int kIn = 16 * KS;
  static constexpr int kLdIn = kIn + kPad, kLdHid = W + kPad;
  static constexpr int kHid = W * kLdIn;
  static constexpr int kOut = kHid + (H - 1) * W * kLdHid;
  static constexpr int kHalves = kOut + W;
};

// Copies the weights (pairs of halves; every row has an even length) and the levels.
template <int W, int KS, int H>
__device__ void stage_weights(const NetArgs& a, __half* sm, Level* sl) {
  using S = Weights<W, KS, H>;
  const uint32_t* src = reinterpret_cast<const uint32_t*>(a.mlp_h);
  uint32_t* dst = reinterpret_cast<uint32_t*>(sm);
  for (int i = threadIdx.x; i < W * S::kIn / 2; i += blockDim.x) {
    const int r = i / (S::kIn / 2), k = i % (S::kIn / 2);
    dst[r * (S::kLdIn / 2) + k] = src[a.mlp.w_in / 2 + i];
  }
  for (int h = 0; h < H - 1; ++h) {
    for (int i = threadIdx.x; i < W * W / 2; i += blockDim.x) {
      const int r = i / (W / 2), k = i % (W / 2);
      dst[(S::kHid + h * W * S::kLdHid) / 2 + r * (S::kLdHid / 2) + k] = src[a.mlp.w_hid[h] / 2 + i];
    }
  }
  for (int i = threadIdx.x; i < W / 2; i += blockDim.x) dst[S::kOut / 2 + i] = src[a.mlp.w_out / 2 + i];
  stage_levels(a.grid, sl);
  __syncthreads();
}

// Encodes the 16-sample tile into layer-1 A fragments (KS k-steps of 16 inputs).
template <int KS>
__device__ __forceinline__ void encode_tile(const NetArgs& a, const Level* sl, int64_t s0, int64_t s1, int c,
                                            uint32_t (&x)[KS][4], float (&u)[2][3]) {
  const bool v0 = s0 < a.n, v1 = s1 < a.n;
  for (int k = 0; k < 3; ++k) {
    u[0][k] = v0 ? a.inputs[3 * s0 + k] : 0.0f;
    u[1][k] = v1 ? a.inputs[3 * s1 + k] : 0.0f;
  }
#pragma unroll
  for (int kk = 0; kk < KS; ++kk) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int l = 8 * kk + c + 4 * half;
      float2 e0 = make_float2(0.0f, 0.0f), e1 = make_float2(0.0f, 0.0f);
      if (l < a.grid.levels) {
        const Level lv = sl[l];
        e0 = encode_level(lv, a.table, u[0][0], u[0][1], u[0][2]);
        e1 = encode_level(lv, a.table, u[1][0], u[1][1], u[1][2]);
      }
      x[kk][2 * half + 0] = pack_h2(e0.x, e0.y);
      x[kk][2 * half + 1] = pack_h2(e1.x, e1.y);
    }
  }
}

// Forward pass of one tile; returns activations' fragments for the backward.
template <int W, int KS, int H>
__device__ __forceinline__ void forward_tile(const __half* sm, const uint32_t (&x)[KS][4], int lane,
                                             uint32_t (&act)[H][W / 16][4], float& y0, float& y1) {
  using S = Weights<W, KS, H>;
  constexpr int NT = W / 8;
  const int g = lane >> 2, c = lane & 3;
  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
#pragma unroll
  for (int kk = 0; kk < KS; ++kk) {
#pragma unroll
    for (int j = 0; j < NT; j += 2) {
      uint32_t b[4];
      b_rows(b, sm, S::kLdIn, 8 * j, 16 * kk, lane);
      mma16816(acc[j], x[kk], b);
      mma16816(acc[j + 1], x[kk], b + 2);
    }
  }
#pragma unroll
  for (int t = 0; t < W / 16; ++t) c_to_a_relu(act[0][t], acc[2 * t], acc[2 * t + 1]);
#pragma unroll
  for (int h = 1; h < H; ++h) {
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
#pragma unroll
    for (int kk = 0; kk < W / 16; ++kk) {
#pragma unroll
      for (int j = 0; j < NT; j += 2) {
        uint32_t b[4];
        b_rows(b, sm + S::kHid + (h - 1) * W * S::kLdHid, S::kLdHid, 8 * j, 16 * kk, lane);
        mma16816(acc[j], act[h - 1][kk], b);
        mma16816(acc[j + 1], act[h - 1][kk], b + 2);
      }
    }
#pragma unroll
    for (int t = 0; t < W / 16; ++t) c_to_a_relu(act[h][t], acc[2 * t], acc[2 * t + 1]);
  }
  // output row: n-tile of 8 where only column 0 is the output neuron
  float o[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  const __half* wo = sm + S::kOut;
#pragma unroll
  for (int kk = 0; kk < W / 16; ++kk) {
    uint32_t b[2] = {0u, 0u};
    if (g == 0) {
      b[0] = *reinterpret_cast<const uint32_t*>(wo + 16 * kk + 2 * c);
      b[1] = *reinterpret_cast<const uint32_t*>(wo + 16 * kk + 2 * c + 8);
    }
    mma16816(o, act[H - 1][kk], b);
  }
  y0 = o[0];  // valid in lanes with c == 0: row g, column 0
  y1 = o[2];  // row g + 8
}

template <int W, int KS, int H>
__global__ void __launch_bounds__(kTrainBlock) infer_kernel(const NetArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __half* sm = reinterpret_cast<__half*>(smem_raw);
  __shared__ Level sl[kMaxLevels];
  stage_weights<W, KS, H>(a, sm, sl);
  const int lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  const int64_t tiles = (a.n + 15) / 16;
  for (int64_t tile = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); tile < tiles;
       tile += warps) {
    const int64_t s0 = tile * 16 + g, s1 = s0 + 8;
    uint32_t x[KS][4];
    float u[2][3];
    encode_tile<KS>(a, sl, s0, s1, c, x, u);
    uint32_t act[H][W / 16][4];
    float y0, y1;
    forward_tile<W, KS, H>(sm, x, lane, act, y0, y1);
    if (c == 0) {
      if (s0 < a.n) a.outputs[s0] = y0;
      if (s1 < a.n) a.outputs[s1] = y1;
    }
  }
}

// Shared memory of a training block: the weights, then per round of 64 samples
// X [64 x IN], the activations of all but the last hidden layer and dpre of
// every layer [64 x W], rows padded.
template <int W, int KS, int H>
struct TrainSmem {
  using S = Weights<W, KS, H>;
  static constexpr int kX = (S::kHalves + 7) / 8 * 8;
  static constexpr int kAct = kX + kTrainRound * S::kLdIn;
  static constexpr int kD = kAct + (H - 1) * kTrainRound * S::kLdHid;
  static constexpr int kHalves = kD + H * kTrainRound * S::kLdHid;
  static constexpr size_t kBytes = sizeof(__half) * kHalves;
};

// Forward + backward over rounds of 64 samples per block (16 per warp).
// Gradients: grid features by vector FP32 reductions; MLP weights accumulated per
// warp in registers (warp w owns output rows [16w, 16w+16) of each matrix) from
// the round's activations staged in shared memory, the output row's per lane over
// its own samples; both flushed at the end.  Bound by the latency of the gathers
// and the reductions at few warps per SM: staging only what the layers read back
// and one copy of the weights leave room for three blocks instead of two.  With
// the 16-byte reductions and ldmatrix fragments 65,536 samples of the default
// network take 178 -> 101 us (a bound of 128 registers for a fourth block: 112).
template <int W, int KS, int H>
__global__ void __launch_bounds__(kTrainBlock) train_kernel(const NetArgs a) {
  static_assert(W == 64 || W == 32 || W == 16, "width");
  using S = Weights<W, KS, H>;
  using T = TrainSmem<W, KS, H>;
  constexpr int NT = W / 8;
  constexpr int IN = 16 * KS;
  constexpr int MT = W / 16;  // m-tiles of a weight matrix (rows)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __half* sm = reinterpret_cast<__half*>(smem_raw);
  __half* sX = sm + T::kX;
  __half* sAct = sm + T::kAct;
  __half* sD = sm + T::kD;
  __shared__ Level sl[kMaxLevels];
  stage_weights<W, KS, H>(a, sm, sl);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  constexpr int HG = H > 1 ? H - 1 : 1;
  // weight-gradient accumulators: this warp's m-tile (rows 16*warp..) of each matrix
  float gin[IN / 8][4];
  float ghid[HG][NT][4];
  float gout[NT][2];  // output row, columns 8j + 2c, + 1 of this lane's samples
#pragma unroll
  for (int j = 0; j < IN / 8; ++j) gin[j][0] = gin[j][1] = gin[j][2] = gin[j][3] = 0.0f;
#pragma unroll
  for (int h = 0; h < HG; ++h)
#pragma unroll
    for (int j = 0; j < NT; ++j) ghid[h][j][0] = ghid[h][j][1] = ghid[h][j][2] = ghid[h][j][3] = 0.0f;
#pragma unroll
  for (int j = 0; j < NT; ++j) gout[j][0] = gout[j][1] = 0.0f;
  float loss = 0.0f;

  const int64_t rounds = (a.n + kTrainRound - 1) / kTrainRound;
  for (int64_t r = blockIdx.x; r < rounds; r += gridDim.x) {
    const int64_t s0 = r * kTrainRound + warp * 16 + g, s1 = s0 + 8;
    const int row0 = warp * 16 + g, row1 = row0 + 8;  // rows within the staged round
    uint32_t x[KS][4];
    float u[2][3];
    encode_tile<KS>(a, sl, s0, s1, c, x, u);
    uint32_t act[H][W / 16][4];
    float y0, y1;
    forward_tile<W, KS, H>(sm, x, lane, act, y0, y1);
    // dL/dy (lanes c==0 hold the outputs); broadcast to the quad
    float dy0 = 0.0f, dy1 = 0.0f;
    if (c == 0) {
      if (s0 < a.n) {
        const float e = y0 - a.targets[s0];
        dy0 = a.loss_scale * e;
        loss += e * e;
      }
      if (s1 < a.n) {
        const float e = y1 - a.targets[s1];
        dy1 = a.loss_scale * e;
        loss += e * e;
      }
      if (a.outputs) {
        if (s0 < a.n) a.outputs[s0] = y0;
        if (s1 < a.n) a.outputs[s1] = y1;
      }
    }
    dy0 = __shfl_sync(0xffffffffu, dy0, lane & ~3);
    dy1 = __shfl_sync(0xffffffffu, dy1, lane & ~3);
    // stage X and the layers' inputs
#pragma unroll
    for (int kk = 0; kk < KS; ++kk) {
      *reinterpret_cast<uint32_t*>(sX + row0 * S::kLdIn + 16 * kk + 2 * c) = x[kk][0];
      *reinterpret_cast<uint32_t*>(sX + row1 * S::kLdIn + 16 * kk + 2 * c) = x[kk][1];
      *reinterpret_cast<uint32_t*>(sX + row0 * S::kLdIn + 16 * kk + 2 * c + 8) = x[kk][2];
      *reinterpret_cast<uint32_t*>(sX + row1 * S::kLdIn + 16 * kk + 2 * c + 8) = x[kk][3];
    }
    auto stage = [&](__half* base, const uint32_t (&f)[W / 16][4]) {
#pragma unroll
      for (int t = 0; t < W / 16; ++t) {
        *reinterpret_cast<uint32_t*>(base + row0 * S::kLdHid + 16 * t + 2 * c) = f[t][0];
        *reinterpret_cast<uint32_t*>(base + row1 * S::kLdHid + 16 * t + 2 * c) = f[t][1];
        *reinterpret_cast<uint32_t*>(base + row0 * S::kLdHid + 16 * t + 2 * c + 8) = f[t][2];
        *reinterpret_cast<uint32_t*>(base + row1 * S::kLdHid + 16 * t + 2 * c + 8) = f[t][3];
      }
    };
#pragma unroll
    for (int h = 0; h < H - 1; ++h) stage(sAct + h * kTrainRound * S::kLdHid, act[h]);
    // backward: dpre of the last hidden layer = dy * w_out, masked by ReLU'
    float dpre[NT][4];
    {
      const __half* wo = sm + S::kOut;
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const float w0 = __half2float(wo[8 * j + 2 * c]), w1 = __half2float(wo[8 * j + 2 * c + 1]);
        const float2 h0 = unpack_h2(act[H - 1][j / 2][(j & 1) ? 2 : 0]);
        const float2 h1 = unpack_h2(act[H - 1][j / 2][(j & 1) ? 3 : 1]);
        gout[j][0] += dy0 * h0.x + dy1 * h1.x;
        gout[j][1] += dy0 * h0.y + dy1 * h1.y;
        dpre[j][0] = h0.x > 0.0f ? dy0 * w0 : 0.0f;
        dpre[j][1] = h0.y > 0.0f ? dy0 * w1 : 0.0f;
        dpre[j][2] = h1.x > 0.0f ? dy1 * w0 : 0.0f;
        dpre[j][3] = h1.y > 0.0f ? dy1 * w1 : 0.0f;
      }
    }
#pragma unroll
    for (int h = H - 1; h >= 0; --h) {
      uint32_t da[W / 16][4];
#pragma unroll
      for (int t = 0; t < W / 16; ++t) c_to_a(da[t], dpre[2 * t], dpre[2 * t + 1]);
      stage(sD + h * kTrainRound * S::kLdHid, da);
      if (h > 0) {
        // d act[h-1] = dpre[h] * W_hid[h-1]  (B[k][n] = W[k][n])
        float nd[NT][4];
#pragma unroll
        for (int j = 0; j < NT; ++j) nd[j][0] = nd[j][1] = nd[j][2] = nd[j][3] = 0.0f;
#pragma unroll
        for (int kk = 0; kk < W / 16; ++kk) {
#pragma unroll
          for (int j = 0; j < NT; j += 2) {
            uint32_t b[4];
            b_cols(b, sm + S::kHid + (h - 1) * W * S::kLdHid, S::kLdHid, 8 * j, 16 * kk, lane);
            mma16816(nd[j], da[kk], b);
            mma16816(nd[j + 1], da[kk], b + 2);
          }
        }
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const float2 h0 = unpack_h2(act[h - 1][j / 2][(j & 1) ? 2 : 0]);
          const float2 h1 = unpack_h2(act[h - 1][j / 2][(j & 1) ? 3 : 1]);
          dpre[j][0] = h0.x > 0.0f ? nd[j][0] : 0.0f;
          dpre[j][1] = h0.y > 0.0f ? nd[j][1] : 0.0f;
          dpre[j][2] = h1.x > 0.0f ? nd[j][2] : 0.0f;
          dpre[j][3] = h1.y > 0.0f ? nd[j][3] : 0.0f;
        }
      } else {
        // dX = dpre[0] * W_in  -> grid gradient scatter (same (sample, level) pairs as the encode)
        float dx[IN / 8][4];
#pragma unroll
        for (int j = 0; j < IN / 8; ++j) dx[j][0] = dx[j][1] = dx[j][2] = dx[j][3] = 0.0f;
#pragma unroll
        for (int kk = 0; kk < W / 16; ++kk) {
#pragma unroll
          for (int j = 0; j < IN / 8; j += 2) {
            uint32_t b[4];
            b_cols(b, sm, S::kLdIn, 8 * j, 16 * kk, lane);
            mma16816(dx[j], da[kk], b);
            mma16816(dx[j + 1], da[kk], b + 2);
          }
        }
        // n-tile j covers inputs 8j..8j+7; lane holds inputs 8j+2c, +1 = level 4j + c
        const float gs = a.grad_scale;
#pragma unroll
        for (int j = 0; j < IN / 8; ++j) {
          const int l = 4 * j + c;
          if (l < a.grid.levels) {
            const Level lv = sl[l];
            if (s0 < a.n) scatter_level(lv, a.grid_grad, u[0][0], u[0][1], u[0][2], make_float2(gs * dx[j][0], gs * dx[j][1]));
            if (s1 < a.n) scatter_level(lv, a.grid_grad, u[1][0], u[1][1], u[1][2], make_float2(gs * dx[j][2], gs * dx[j][3]));
          }
        }
      }
    }
    __syncthreads();
    // weight gradients over the staged 64 samples: G = dpre^T (W x 64) * input (64 x in)
    // this warp: rows [16*warp, 16*warp+16) of each matrix (only if warp < MT)
    if (warp < MT) {
      const int m0 = 16 * warp;
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const __half* D = sD + h * kTrainRound * S::kLdHid;                           // [64 x W] dpre of layer h
        const __half* X = (h == 0) ? sX : sAct + (h - 1) * kTrainRound * S::kLdHid;  // layer input
        constexpr int kTilesIn = IN / 8;
#pragma unroll
        for (int ks = 0; ks < kTrainRound / 16; ++ks) {
          const int k0 = 16 * ks;
          uint32_t af[4];
          a_cols(af, D, S::kLdHid, m0, k0, lane);
#pragma unroll
          for (int j = 0; j < (h == 0 ? kTilesIn : NT); j += 2) {
            uint32_t bf[4];
            b_cols(bf, X, h == 0 ? S::kLdIn : S::kLdHid, 8 * j, k0, lane);
            if (h == 0) {
              mma16816(gin[j], af, bf);
              mma16816(gin[j + 1], af, bf + 2);
            } else {
              mma16816(ghid[h - 1][j], af, bf);
              mma16816(ghid[h - 1][j + 1], af, bf + 2);
            }
          }
        }
      }
    }
    __syncthreads();
  }
  // flush this warp's weight-gradient tiles: C fragment rows m0+g, m0+g+8, cols 8j+2c..
  const float gs = a.grad_scale;
  auto flush = [&](float* G, int ld, int j, const float* f) {
    const int m0 = 16 * warp;
    red_add(reinterpret_cast<float2*>(G + (m0 + g) * ld + 8 * j + 2 * c), make_float2(gs * f[0], gs * f[1]));
    red_add(reinterpret_cast<float2*>(G + (m0 + g + 8) * ld + 8 * j + 2 * c), make_float2(gs * f[2], gs * f[3]));
  };
  if (warp < MT) {
#pragma unroll
    for (int j = 0; j < IN / 8; ++j) flush(a.mlp_grad + a.mlp.w_in, IN, j, gin[j]);
#pragma unroll
    for (int h = 1; h < H; ++h) {
#pragma unroll
      for (int j = 0; j < NT; ++j) flush(a.mlp_grad + a.mlp.w_hid[h - 1], W, j, ghid[h - 1][j]);
    }
  }
  // output row: sum over the lanes of a column (g), then over the block's warps
#pragma unroll
  for (int j = 0; j < NT; ++j) {
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      gout[j][0] += __shfl_xor_sync(0xffffffffu, gout[j][0], o);
      gout[j][1] += __shfl_xor_sync(0xffffffffu, gout[j][1], o);
    }
    if (g == 0) {
      red_add(reinterpret_cast<float2*>(a.mlp_grad + a.mlp.w_out + 8 * j + 2 * c),
              make_float2(gs * gout[j][0], gs * gout[j][1]));
    }
  }
  if (a.loss_sum) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if (lane == 0) atomicAdd(a.loss_sum, loss);
  }
}

// Adam (Kingma & Ba) on FP32 master parameters; refreshes the FP16 copy and
// clears the gradient.  Four parameters per thread in 128-bit accesses: the
// parameter count is a multiple of 8 (build_meta).  34 bytes per parameter: 12.2 M
// parameters 102 -> 79 us, 5.3 TB/s (6.4 measured copy).
struct AdamArgs {
  float lr, b1, b2, eps, bc1, bc2, gscale;
};

__device__ __forceinline__ float adam_update(float& p, float g, float& m, float& v, const AdamArgs& a) {
  const float gi = g * a.gscale;
  const float mi = a.b1 * m + (1.0f - a.b1) * gi;
  const float vi = a.b2 * v + (1.0f - a.b2) * gi * gi;
  m = mi;
  v = vi;
  const float upd = a.lr * (mi / a.bc1) / (sqrtf(vi / a.bc2) + a.eps);
  p = p - upd;
  return p;
}

__global__ void __launch_bounds__(256) adam_kernel(float4* __restrict__ p, uint2* __restrict__ ph,
                                                   float4* __restrict__ g, float4* __restrict__ m,
                                                   float4* __restrict__ v, int64_t quads, const AdamArgs a) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= quads) return;
  const float4 gi = g[i];
  float4 pi = p[i], mi = m[i], vi = v[i];
  adam_update(pi.x, gi.x, mi.x, vi.x, a);
  adam_update(pi.y, gi.y, mi.y, vi.y, a);
  adam_update(pi.z, gi.z, mi.z, vi.z, a);
  adam_update(pi.w, gi.w, mi.w, vi.w, a);
  p[i] = pi;
  m[i] = mi;
  v[i] = vi;
  ph[i] = make_uint2(pack_h2(pi.x, pi.y), pack_h2(pi.z, pi.w));
  g[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

__global__ void to_half_kernel(const float* __restrict__ p, __half* __restrict__ ph, int64_t n) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) ph[i] = __float2half_rn(p[i]);
}

__global__ void init_params_kernel(float* __restrict__ p, int64_t n_grid, const int* __restrict__ mlp_fan,
                                   int64_t n_total, uint64_t seed) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n_total) return;
  uint32_t k0, k1;
  philox_key(seed, 7u, k0, k1);
  const U4 r = philox4x32_10(U4{static_cast<uint32_t>(i), static_cast<uint32_t>(i >> 32), 0u, 0u}, k0, k1);
  const float u = 2.0f * u01(r.x) - 1.0f;
  if (i < n_grid) {
    p[i] = 1.0e-4f * u;  // hash-grid features: U(-1e-4, 1e-4)
  } else {
    // MLP weights: U(-s, s), s = sqrt(6 / (fan_in + fan_out))
    const int j = static_cast<int>(i - n_grid);
    p[i] = u * sqrtf(6.0f / static_cast<float>(mlp_fan[j]));
  }
}

}  // namespace
}  // namespace n2w

struct n2w_cache {
  n2w_cache_config cfg;
  n2w::GridMeta grid;
  n2w::MlpMeta mlp;
  int64_t n_grid = 0;  // floats of grid parameters (entries * F)
  int64_t n_total = 0;
  float* d_p = nullptr;     // fp32 master [grid | mlp]
  __half* d_ph = nullptr;   // fp16 working copy
  float* d_g = nullptr;     // fp32 gradient
  float* d_m = nullptr;
  float* d_v = nullptr;
  float* d_loss = nullptr;  // device scalar
  int64_t step = 0;
  int device = 0;
};

namespace n2w {
namespace {

void build_meta(n2w_cache& c) {
  const n2w_cache_config& k = c.cfg;
  N2W_REQUIRE(k.n_levels >= 1 && k.n_levels <= kMaxLevels, "n_levels must be in [1, 16]");
  N2W_REQUIRE(k.n_features_per_level == 2, "n_features_per_level must be 2");
  N2W_REQUIRE(k.log2_hashmap_size >= 10 && k.log2_hashmap_size <= 24, "log2_hashmap_size must be in [10, 24]");
  N2W_REQUIRE(k.base_resolution >= 2.0f, "base_resolution must be >= 2");
  N2W_REQUIRE(k.n_neurons == 16 || k.n_neurons == 32 || k.n_neurons == 64, "n_neurons must be 16, 32 or 64");
  N2W_REQUIRE(k.n_hidden_layers >= 1 && k.n_hidden_layers <= kMaxHidden, "n_hidden_layers must be in [1, 4]");
  float b = k.per_level_scale;
  if (!(b > 0.0f)) {
    N2W_REQUIRE(k.max_resolution >= k.base_resolution, "max_resolution must be >= base_resolution");
    b = k.n_levels > 1 ? std::exp((std::log(k.max_resolution) - std::log(k.base_resolution)) / (k.n_levels - 1)) : 1.0f;
  }
  c.cfg.per_level_scale = b;
  GridMeta& g = c.grid;
  std::memset(&g, 0, sizeof(g));
  g.levels = k.n_levels;
  g.features = 2;
  const uint64_t T = 1ull << k.log2_hashmap_size;
  uint64_t off = 0;
  for (int l = 0; l < k.n_levels; ++l) {
    // N_l = floor(N_min * b^l), evaluated in FP64 with a 1e-6 relative guard so
    // a level that is an exact power (e.g. 2048 = 16 * 128) is not rounded down.
    const double x = static_cast<double>(k.base_resolution) * std::pow(static_cast<double>(b), static_cast<double>(l));
    const uint32_t res = static_cast<uint32_t>(std::floor(x * (1.0 + 1e-6)));
    const uint64_t dense = static_cast<uint64_t>(res + 1) * (res + 1) * (res + 1);
    const uint64_t size = dense <= T ? ((dense + 7) / 8) * 8 : T;
    g.res[l] = res;
    g.scale[l] = static_cast<float>(res);
    g.dense[l] = dense <= T ? 1u : 0u;
    g.table_size[l] = static_cast<uint32_t>(size);
    g.offset[l] = static_cast<uint32_t>(off);
    off += size;
  }
  c.n_grid = static_cast<int64_t>(off) * 2;
  MlpMeta& m = c.mlp;
  m.width = k.n_neurons;
  m.hidden = k.n_hidden_layers;
  m.in_dim = k.n_levels * 2 <= 16 ? 16 : 32;
  int o = 0;
  m.w_in = o;
  o += m.width * m.in_dim;
  for (int h = 0; h < kMaxHidden; ++h) m.w_hid[h] = 0;
  for (int h = 0; h < m.hidden - 1; ++h) {
    m.w_hid[h] = o;
    o += m.width * m.width;
  }
  m.w_out = o;
  o += m.width;
  m.total = (o + 7) / 8 * 8;
  c.n_total = c.n_grid + m.total;
}

NetArgs net_args(const n2w_cache& c) {
  NetArgs a{};
  a.grid = c.grid;
  a.mlp = c.mlp;
  a.table = reinterpret_cast<const __half2*>(c.d_ph);
  a.mlp_h = c.d_ph + c.n_grid;
  a.grid_grad = reinterpret_cast<float2*>(c.d_g);
  a.mlp_grad = c.d_g + c.n_grid;
  a.grad_scale = 1.0f;
  return a;
}

// One Adam step on gscale times the gradient buffer.
void launch_adam(n2w_cache& c, float gscale, cudaStream_t s) {
  ++c.step;
  AdamArgs a{};
  a.lr = c.cfg.learning_rate;
  a.b1 = c.cfg.beta1;
  a.b2 = c.cfg.beta2;
  a.eps = c.cfg.epsilon;
  a.bc1 = 1.0f - std::pow(a.b1, static_cast<float>(c.step));
  a.bc2 = 1.0f - std::pow(a.b2, static_cast<float>(c.step));
  a.gscale = gscale;
  const int64_t quads = c.n_total / 4;
  const int b = 256;
  adam_kernel<<<static_cast<unsigned>((quads + b - 1) / b), b, 0, s>>>(
      reinterpret_cast<float4*>(c.d_p), reinterpret_cast<uint2*>(c.d_ph), reinterpret_cast<float4*>(c.d_g),
      reinterpret_cast<float4*>(c.d_m), reinterpret_cast<float4*>(c.d_v), quads, a);
  N2W_CUDA(cudaGetLastError());
}

template <int W, int KS, int H>
void launch_infer_t(const NetArgs& a, cudaStream_t s) {
  const size_t smem = sizeof(__half) * Weights<W, KS, H>::kHalves;
  const int64_t tiles = (a.n + 15) / 16;
  int64_t grid = std::min<int64_t>((tiles + 3) / 4, static_cast<int64_t>(sm_count_current()) * 8);
  grid = std::max<int64_t>(grid, 1);
  infer_kernel<W, KS, H><<<static_cast<unsigned>(grid), kTrainBlock, smem, s>>>(a);
  N2W_CUDA(cudaGetLastError());
}

template <int W, int KS, int H>
void launch_train_t(const NetArgs& a, cudaStream_t s) {
  const size_t smem = TrainSmem<W, KS, H>::kBytes;
  auto k = train_kernel<W, KS, H>;
  N2W_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  int occ = 0;
  N2W_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, kTrainBlock, smem));
  const int64_t rounds = (a.n + kTrainRound - 1) / kTrainRound;
  const int64_t resident = static_cast<int64_t>(sm_count_current()) * std::max(occ, 1);
  // every block the same number of rounds, as few blocks as that takes
  const int64_t per_block = (rounds + resident - 1) / resident;
  const int64_t grid = std::max<int64_t>((rounds + per_block - 1) / per_block, 1);
  k<<<static_cast<unsigned>(grid), kTrainBlock, smem, s>>>(a);
  N2W_CUDA(cudaGetLastError());
}

// Runtime (width, input k-steps, hidden layers) -> template instance.
template <template <int, int, int> class F>
void dispatch(const NetArgs& a, cudaStream_t s) {
  const int W = a.mlp.width, KS = a.mlp.in_dim / 16, H = a.mlp.hidden;
#define N2W_CACHE_CASE(w, k, h) \
  if (W == w && KS == k && H == h) return F<w, k, h>::run(a, s);
#define N2W_CACHE_H(w, k) N2W_CACHE_CASE(w, k, 1) N2W_CACHE_CASE(w, k, 2) N2W_CACHE_CASE(w, k, 3) N2W_CACHE_CASE(w, k, 4)
  N2W_CACHE_H(64, 2) N2W_CACHE_H(64, 1) N2W_CACHE_H(32, 2) N2W_CACHE_H(32, 1) N2W_CACHE_H(16, 2) N2W_CACHE_H(16, 1)
#undef N2W_CACHE_H
#undef N2W_CACHE_CASE
  throw Error(N2W_EINTERNAL, "unsupported cache network shape");
}

template <int W, int KS, int H>
struct InferL {
  static void run(const NetArgs& a, cudaStream_t s) { launch_infer_t<W, KS, H>(a, s); }
};
template <int W, int KS, int H>
struct TrainL {
  static void run(const NetArgs& a, cudaStream_t s) { launch_train_t<W, KS, H>(a, s); }
};

void launch_infer(const NetArgs& a, cudaStream_t s) { dispatch<InferL>(a, s); }
void launch_train(const NetArgs& a, cudaStream_t s) { dispatch<TrainL>(a, s); }

// fan_in + fan_out of each MLP parameter (for the uniform init bound).
std::vector<int> mlp_fans(const MlpMeta& m) {
  std::vector<int> f(static_cast<size_t>(m.total), 1);
  for (int i = 0; i < m.width * m.in_dim; ++i) f[m.w_in + i] = m.in_dim + m.width;
  for (int h = 0; h < m.hidden - 1; ++h)
    for (int i = 0; i < m.width * m.width; ++i) f[m.w_hid[h] + i] = 2 * m.width;
  for (int i = 0; i < m.width; ++i) f[m.w_out + i] = m.width + 1;
  return f;
}

void release_cache(n2w_cache* c) {
  if (!c) return;
  cudaFree(c->d_p);
  cudaFree(c->d_ph);
  cudaFree(c->d_g);
  cudaFree(c->d_m);
  cudaFree(c->d_v);
  cudaFree(c->d_loss);
  delete c;
}

constexpr uint64_t kCacheMagic = 0x31454843574E324Eull;  // "N2WCHE1"

}  // namespace
}  // namespace n2w

using namespace n2w;

extern "C" {

int n2w_cache_config_default(n2w_cache_config* out) {
  return guarded([&] {
    N2W_REQUIRE(out, "null output");
    std::memset(out, 0, sizeof(*out));
    out->n_levels = 16;
    out->n_features_per_level = 2;
    out->log2_hashmap_size = 19;
    out->base_resolution = 16.0f;
    out->max_resolution = 2048.0f;
    out->per_level_scale = 0.0f;
    out->n_neurons = 64;
    out->n_hidden_layers = 2;
    out->learning_rate = 1.0e-2f;
    out->beta1 = 0.9f;
    out->beta2 = 0.99f;
    out->epsilon = 1.0e-15f;
    out->seed = 1337;
  });
}

int n2w_cache_describe(const n2w_cache_config* cfg, int64_t* grid_params, int64_t* mlp_params,
                       int32_t* level_resolution, int32_t* level_table_size) {
  return guarded([&] {
    N2W_REQUIRE(cfg, "null config");
    n2w_cache c;
    c.cfg = *cfg;
    build_meta(c);
    if (grid_params) *grid_params = c.n_grid;
    if (mlp_params) *mlp_params = c.mlp.total;
    for (int l = 0; l < c.grid.levels; ++l) {
      if (level_resolution) level_resolution[l] = static_cast<int32_t>(c.grid.res[l]);
      if (level_table_size) level_table_size[l] = static_cast<int32_t>(c.grid.table_size[l]);
    }
  });
}

int n2w_cache_create(const n2w_cache_config* cfg, n2w_cache** out) {
  return guarded([&] {
    N2W_REQUIRE(cfg && out, "null argument");
    auto* c = new n2w_cache();
    try {
      c->cfg = *cfg;
      build_meta(*c);
      N2W_CUDA(cudaGetDevice(&c->device));
      const size_t n = static_cast<size_t>(c->n_total);
      N2W_CUDA(cudaMalloc(&c->d_p, n * sizeof(float)));
      N2W_CUDA(cudaMalloc(&c->d_ph, n * sizeof(__half)));
      N2W_CUDA(cudaMalloc(&c->d_g, n * sizeof(float)));
      N2W_CUDA(cudaMalloc(&c->d_m, n * sizeof(float)));
      N2W_CUDA(cudaMalloc(&c->d_v, n * sizeof(float)));
      N2W_CUDA(cudaMalloc(&c->d_loss, sizeof(float)));
      N2W_CUDA(cudaMemset(c->d_g, 0, n * sizeof(float)));
      N2W_CUDA(cudaMemset(c->d_m, 0, n * sizeof(float)));
      N2W_CUDA(cudaMemset(c->d_v, 0, n * sizeof(float)));
      std::vector<int> fans = mlp_fans(c->mlp);
      int* d_fans = nullptr;
      N2W_CUDA(cudaMalloc(&d_fans, fans.size() * sizeof(int)));
      N2W_CUDA(cudaMemcpy(d_fans, fans.data(), fans.size() * sizeof(int), cudaMemcpyHostToDevice));
      const int b = 256;
      init_params_kernel<<<static_cast<unsigned>((n + b - 1) / b), b>>>(c->d_p, c->n_grid, d_fans,
                                                                          c->n_total, c->cfg.seed);
      N2W_CUDA(cudaGetLastError());
      to_half_kernel<<<static_cast<unsigned>((n + b - 1) / b), b>>>(c->d_p, c->d_ph, c->n_total);
      N2W_CUDA(cudaGetLastError());
      N2W_CUDA(cudaDeviceSynchronize());
      cudaFree(d_fans);
    } catch (...) {
      release_cache(c);
      throw;
    }
    *out = c;
  });
}

void n2w_cache_destroy(n2w_cache* c) { release_cache(c); }

int n2w_cache_info(const n2w_cache* c, n2w_cache_config* cfg_out, int64_t* grid_params, int64_t* mlp_params,
                   int32_t* level_resolution, int32_t* level_table_size) {
  return guarded([&] {
    N2W_REQUIRE(c, "null cache");
    if (cfg_out) *cfg_out = c->cfg;
    if (grid_params) *grid_params = c->n_grid;
    if (mlp_params) *mlp_params = c->mlp.total;
    for (int l = 0; l < c->grid.levels; ++l) {
      if (level_resolution) level_resolution[l] = static_cast<int32_t>(c->grid.res[l]);
      if (level_table_size) level_table_size[l] = static_cast<int32_t>(c->grid.table_size[l]);
    }
  });
}

int n2w_cache_infer(const n2w_cache* c, const float* d_inputs, int64_t n, float* d_outputs, n2w_stream_t stream) {
  return guarded([&] {
    N2W_REQUIRE(c, "null cache");
    N2W_REQUIRE(n >= 0, "n must be non-negative");
    if (n == 0) return;
    N2W_REQUIRE(d_inputs && d_outputs, "null device pointer");
    NetArgs a = net_args(*c);
    a.inputs = d_inputs;
    a.outputs = d_outputs;
    a.n = n;
    launch_infer(a, stream);
  });
}

int n2w_cache_gradients(n2w_cache* c, const float* d_inputs, const float* d_targets, int64_t n, float* d_outputs,
                        n2w_stream_t stream) {
  return guarded([&] {
    N2W_REQUIRE(c, "null cache");
    N2W_REQUIRE(n > 0 && d_inputs && d_targets, "invalid arguments");
    NetArgs a = net_args(*c);
    a.inputs = d_inputs;
    a.targets = d_targets;
    a.outputs = d_outputs;
    a.n = n;
    // The backward runs on n * dL/dy = 2 (y - t): O(1) values keep FP16
    // activations' gradients out of the subnormal range; the 1/n is applied to
    // the FP32 gradients as they are added.
    a.loss_scale = 2.0f;
    a.grad_scale = 1.0f / static_cast<float>(n);
    a.loss_sum = c->d_loss;
    N2W_CUDA(cudaMemsetAsync(c->d_loss, 0, sizeof(float), stream));
    launch_train(a, stream);
  });
}

int n2w_cache_train_step(n2w_cache* c, const float* d_inputs, const float* d_targets, int64_t n, float* h_loss_out,
                         n2w_stream_t stream) {
  return guarded([&] {
    N2W_REQUIRE(c, "null cache");
    N2W_REQUIRE(n > 0 && d_inputs && d_targets, "invalid arguments");
    NetArgs a = net_args(*c);
    a.inputs = d_inputs;
    a.targets = d_targets;
    a.n = n;
    a.loss_scale = 2.0f;  // n * dL/dy; the 1/n is applied inside the Adam update
    a.loss_sum = c->d_loss;
    N2W_CUDA(cudaMemsetAsync(c->d_loss, 0, sizeof(float), stream));
    launch_train(a, stream);
    launch_adam(*c, 1.0f / static_cast<float>(n), stream);
    if (h_loss_out) {
      float l = 0.0f;
      N2W_CUDA(cudaMemcpyAsync(&l, c->d_loss, sizeof(float), cudaMemcpyDeviceToHost, stream));
      N2W_CUDA(cudaStreamSynchronize(stream));
      *h_loss_out = l / static_cast<float>(n);
    }
  });
}

int n2w_cache_gradient_buffer(n2w_cache* c, float** d_grad, int64_t* count, float** d_loss_sum) {
  return guarded([&] {
    N2W_REQUIRE(c, "null cache");
    if (d_grad) *d_grad = c->d_g;
    if (count) *count = c->n_total;
    if (d_loss_sum) *d_loss_sum = c->d_loss;
  });
}

int n2w_cache_apply_gradients(n2w_cache* c, float grad_scale, n2w_stream_t stream) {
  return guarded([&] {
    N2W_REQUIRE(c, "null cache");
    N2W_REQUIRE(std::isfinite(grad_scale) && grad_scale > 0.0f, "grad_scale must be positive");
    launch_adam(*c, grad_scale, stream);
  });
}

int n2w_cache_get_params(const n2w_cache* c, float* h_fp32, uint16_t* h_fp16, float* h_grad) {
  return guarded([&] {
    N2W_REQUIRE(c, "null cache");
    const size_t n = static_cast<size_t>(c->n_total);
    if (h_fp32) N2W_CUDA(cudaMemcpy(h_fp32, c->d_p, n * sizeof(float), cudaMemcpyDeviceToHost));
    if (h_fp16) N2W_CUDA(cudaMemcpy(h_fp16, c->d_ph, n * sizeof(__half), cudaMemcpyDeviceToHost));
    if (h_grad) N2W_CUDA(cudaMemcpy(h_grad, c->d_g, n * sizeof(float), cudaMemcpyDeviceToHost));
  });
}

int n2w_cache_set_params(n2w_cache* c, const float* h_fp32) {
  return guarded([&] {
    N2W_REQUIRE(c && h_fp32, "null argument");
    const size_t n = static_cast<size_t>(c->n_total);
    N2W_CUDA(cudaMemcpy(c->d_p, h_fp32, n * sizeof(float), cudaMemcpyHostToDevice));
    const int b = 256;
    to_half_kernel<<<static_cast<unsigned>((n + b - 1) / b), b>>>(c->d_p, c->d_ph, c->n_total);
    N2W_CUDA(cudaGetLastError());
    N2W_CUDA(cudaMemset(c->d_g, 0, n * sizeof(float)));
    N2W_CUDA(cudaDeviceSynchronize());
  });
}

int n2w_cache_copy_params(n2w_cache* dst, const n2w_cache* src, n2w_stream_t stream) {
  return guarded([&] {
    N2W_REQUIRE(dst && src, "null argument");
    const n2w_cache_config& a = dst->cfg;
    const n2w_cache_config& b = src->cfg;
    N2W_REQUIRE(dst->n_total == src->n_total && a.n_levels == b.n_levels &&
                    a.n_features_per_level == b.n_features_per_level && a.log2_hashmap_size == b.log2_hashmap_size &&
                    a.base_resolution == b.base_resolution && a.per_level_scale == b.per_level_scale &&
                    a.max_resolution == b.max_resolution && a.n_neurons == b.n_neurons &&
                    a.n_hidden_layers == b.n_hidden_layers,
                "n2w_cache_copy_params: caches of different configurations");
    if (dst == src) return;
    const size_t n = static_cast<size_t>(src->n_total);
    N2W_CUDA(cudaMemcpyAsync(dst->d_p, src->d_p, n * sizeof(float), cudaMemcpyDeviceToDevice, stream));
    N2W_CUDA(cudaMemcpyAsync(dst->d_ph, src->d_ph, n * sizeof(__half), cudaMemcpyDeviceToDevice, stream));
  });
}

int n2w_cache_zero_grad(n2w_cache* c, n2w_stream_t stream) {
  return guarded([&] {
    N2W_REQUIRE(c, "null cache");
    N2W_CUDA(cudaMemsetAsync(c->d_g, 0, static_cast<size_t>(c->n_total) * sizeof(float), stream));
  });
}

// Binary checkpoint: magic, config, step, then fp32 params, Adam m, Adam v.
int n2w_cache_save(const n2w_cache* c, const char* path) {
  return guarded([&] {
    N2W_REQUIRE(c && path, "null argument");
    const size_t n = static_cast<size_t>(c->n_total);
    std::vector<float> buf(3 * n);
    N2W_CUDA(cudaMemcpy(buf.data(), c->d_p, n * sizeof(float), cudaMemcpyDeviceToHost));
    N2W_CUDA(cudaMemcpy(buf.data() + n, c->d_m, n * sizeof(float), cudaMemcpyDeviceToHost));
    N2W_CUDA(cudaMemcpy(buf.data() + 2 * n, c->d_v, n * sizeof(float), cudaMemcpyDeviceToHost));
    std::ofstream f(path, std::ios::binary);
    if (!f) throw Error(N2W_EIO, std::string("cannot write ") + path);
    const uint64_t magic = kCacheMagic, count = n;
    const int64_t step = c->step;
    f.write(reinterpret_cast<const char*>(&magic), 8);
    f.write(reinterpret_cast<const char*>(&c->cfg), sizeof(c->cfg));
    f.write(reinterpret_cast<const char*>(&step), 8);
    f.write(reinterpret_cast<const char*>(&count), 8);
    f.write(reinterpret_cast<const char*>(buf.data()), static_cast<std::streamsize>(buf.size() * sizeof(float)));
    if (!f) throw Error(N2W_EIO, std::string("write failed: ") + path);
  });
}

int n2w_cache_load(const char* path, n2w_cache** out) {
  return guarded([&] {
    N2W_REQUIRE(path && out, "null argument");
    std::ifstream f(path, std::ios::binary);
    if (!f) throw Error(N2W_EIO, std::string("cannot read ") + path);
    uint64_t magic = 0, count = 0;
    int64_t step = 0;
    n2w_cache_config cfg{};
    f.read(reinterpret_cast<char*>(&magic), 8);
    if (magic != kCacheMagic) throw Error(N2W_EIO, "not an n2w cache checkpoint");
    f.read(reinterpret_cast<char*>(&cfg), sizeof(cfg));
    f.read(reinterpret_cast<char*>(&step), 8);
    f.read(reinterpret_cast<char*>(&count), 8);
    n2w_cache* c = nullptr;
    const int st = n2w_cache_create(&cfg, &c);
    if (st != N2W_OK) throw Error(st, n2w_last_error());
    try {
      if (count != static_cast<uint64_t>(c->n_total)) throw Error(N2W_EIO, "checkpoint size mismatch");
      std::vector<float> buf(3 * count);
      f.read(reinterpret_cast<char*>(buf.data()), static_cast<std::streamsize>(buf.size() * sizeof(float)));
      if (!f) throw Error(N2W_EIO, "truncated checkpoint");
      const size_t n = count;
      N2W_CUDA(cudaMemcpy(c->d_p, buf.data(), n * sizeof(float), cudaMemcpyHostToDevice));
      N2W_CUDA(cudaMemcpy(c->d_m, buf.data() + n, n * sizeof(float), cudaMemcpyHostToDevice));
      N2W_CUDA(cudaMemcpy(c->d_v, buf.data() + 2 * n, n * sizeof(float), cudaMemcpyHostToDevice));
      const int b = 256;
      to_half_kernel<<<static_cast<unsigned>((n + b - 1) / b), b>>>(c->d_p, c->d_ph, c->n_total);
      N2W_CUDA(cudaGetLastError());
      N2W_CUDA(cudaDeviceSynchronize());
      c->step = step;
    } catch (...) {
      release_cache(c);
      throw;
    }
    *out = c;
  });
}

}  // extern "C"
