// Rectangle-triangle tilings of a hexagon (reference: src/RectTriangle/).
//
// A vertex of the triangular lattice holds the covering codes of its six surrounding
// triangles, one hexadecimal digit each (d5..d0 as drawn at RectTriangleTiler.h:14-22).  The
// sweep has three colours, (i - j) mod 3.  One step draws a colour, offers every vertex of
// that colour a move - with probability 0.9 - and rebuilds the six digits of each vertex of
// the two other colours from its neighbours.  The offered move, and whether the weight ratio
// accepts it, follow flipTiles (recttrianglekernel.cl:25-118):
//   * the five hexagons made of triangles or of one rectangle move to the state picked by
//     the quarter of the rescaled draw;
//   * the twelve rectangle-pair hexagons toggle with their partner.
// The nine weights are runtime arguments; the reference hard-codes them at
// recttrianglekernel.cl:3-11.  MTGP mode: the reference's CUDA build's random stream (8 x 8
// blocks over the N x N/3 slots of the drawn colour, one cuRAND MTGP32 generator per block
// seeded seed + block; RectTriangleTiler.cpp:75-85, recttrianglekernel.cu:31-43).
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <curand_kernel.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <memory>
#include <random>
#include <string>
#include <vector>

#include "pdl.cuh"
#include "rng.cuh"
#include "rt_internal.h"

namespace rt {
namespace {

struct RtWeights {
  float w[16];  // by digit: 0, wt1..3, wr1..3, wr1..3, wm1..3, wm1..3 (recttrianglekernel.cl:13)
};

__host__ __device__ inline float ratio_of(const RtWeights& W, int a, int b) {
  const float* w = W.w;
  return (w[(b >> 20) & 15] * w[(b >> 16) & 15] * w[(b >> 12) & 15] * w[(b >> 8) & 15] * w[(b >> 4) & 15] * w[b & 15]) /
         (w[(a >> 20) & 15] * w[(a >> 16) & 15] * w[(a >> 12) & 15] * w[(a >> 8) & 15] * w[(a >> 4) & 15] * w[a & 15]);
}

// The five hexagons made of triangles or of one rectangle.
__host__ __device__ inline bool rt_five(int hex) {
  return hex == 0x122133 || hex == 0x331221 || hex == 0x8ebbe8 || hex == 0xfc99cf || hex == 0xa7dd7a;
}

// The state that hex is offered in quarter q of the rescaled draw (hex itself: none).
__host__ __device__ inline int rt_target(int hex, int q) {
  if (rt_five(hex)) {
    const int target = q == 0 ? 0xa7dd7a : (q == 1 ? 0xfc99cf : (q == 2 ? 0x8ebbe8 : 0x331221));
    return target == hex ? 0x122133 : target;
  }
  switch (hex) {
    case 0x47d47a: return 0xd22a33;
    case 0xd22a33: return 0x47d47a;
    case 0xa74d74: return 0x33a22d;
    case 0x33a22d: return 0xa74d74;
    case 0x8eb558: return 0x331eb1;
    case 0x331eb1: return 0x8eb558;
    case 0x855be8: return 0x1be133;
    case 0x1be133: return 0x855be8;
    case 0x6699cf: return 0xcf1221;
    case 0xcf1221: return 0x6699cf;
    case 0xfc9966: return 0x1221fc;
    case 0x1221fc: return 0xfc9966;
    default: return hex;
  }
}

// The decision of flipTiles for state hex and uniform rd in [0, 1): float arithmetic in the
// reference's order (rd / 0.9f, quarter boundaries, (rd - sc) * 4).
__host__ __device__ inline int rt_flip(int hex, float rd, const RtWeights& W) {
  if (!(rd < 0.9f)) return hex;
  rd /= 0.9f;
  const int q = rd < 0.25f ? 0 : (rd < 0.5f ? 1 : (rd < 0.75f ? 2 : 3));
  const int next = rt_target(hex, q);
  if (next == hex) return hex;  // no move offered
  const float ratio = ratio_of(W, hex, next);
  if (rt_five(hex)) rd = (rd - 0.25f * (float)q) * 4;
  return ratio >= rd ? next : hex;
}

struct RtView {
  int32_t* base;
  int N, M, P;
  size_t colour_stride;
  uint4* tmt;
  const uint4* tmt_params;  // per-generator {mat1, mat2, tmat} (LoadTinyMT), or NULL
  __device__ int32_t* colour(int c) const { return base + (size_t)c * colour_stride; }
};

// InitTinyMT (recttrianglekernel.cl:148-155): generator k, of the work item (k / M, k mod M),
// seeded seed + k with its own parameters when a table is loaded.
__global__ void k_rt_seed(uint4* st, const uint4* params, int64_t count, uint32_t seed) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  const uint4 p = params ? params[k] : make_uint4(kTmtMat1, kTmtMat2, kTmtTmat, 0);
  st[k] = tmt_seed(seed + (uint32_t)k, p.x, p.y, p.z);
}

__global__ void k_rt_flip_tmt(RtView v, int r, RtWeights W) {
  pdl_begin();
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (j >= v.M) return;
  const int64_t k = (int64_t)i * v.M + j;
  uint4 s = v.tmt[k];
  const uint4 pr = v.tmt_params ? v.tmt_params[k] : make_uint4(kTmtMat1, kTmtMat2, kTmtTmat, 0);
  const uint32_t u = tmt_next_u23(s, pr.x, pr.y, pr.z);
  v.tmt[k] = s;
  int32_t* p = v.colour(r) + (size_t)i * v.P + j;
  const int e = *p, n = rt_flip(e, (float)u * (1.0f / 8388608.0f), W);
  if (n != e) *p = n;
}

// MTGP mode: every thread of the block draws before the bounds test (recttrianglekernel.cu:35-43);
// flipTilesKernel decides as flipTiles does.
__global__ void __launch_bounds__(kMtgpBlock* kMtgpBlock) k_rt_flip_mtgp(RtView v, int r, RtWeights W,
                                                                          curandStateMtgp32* states) {
  pdl_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const float rd = curand_uniform(states + blockIdx.x * gridDim.y + blockIdx.y);
  if (i >= v.N || j >= v.M) return;
  int32_t* p = v.colour(r) + (size_t)i * v.P + j;
  const int e = *p, n = rt_flip(e, rd, W);
  if (n != e) *p = n;
}

__global__ void k_rt_flip_fast(RtView v, int r, RtWeights W, uint64_t seed, uint32_t stream, int64_t h) {
  pdl_begin();
  const int q = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (4 * q >= v.M) return;
  const uint4 d = fast_quad(seed, stream, h, (uint32_t)i, (uint32_t)q);
  const uint32_t u4[4] = {d.x, d.y, d.z, d.w};
  int32_t* row = v.colour(r) + (size_t)i * v.P;
#pragma unroll
  for (int k4 = 0; k4 < 4; ++k4) {
    const int j = 4 * q + k4;
    if (j >= v.M) break;
    const int e = row[j], n = rt_flip(e, (float)(u4[k4] >> 8) * (1.0f / 16777216.0f), W);
    if (n != e) row[j] = n;
  }
}

// updateTiles1 / updateTiles2 (recttrianglekernel.cl:120-146): the digits of colour
// (r+1) mod 3 and (r+2) mod 3 rebuilt from the rotated colour's neighbours.
__global__ void k_rt_update(RtView v, int r) {
  pdl_begin();
  const int j = blockIdx.x * blockDim.x + threadIdx.x + 1, i = blockIdx.y + 1;
  if (j > v.M - 2 || i > v.N - 2) return;
  const int32_t* A = v.colour(r);
  const int im = i % 3;
  {
    const int p1 = im == r, p2 = im == (r + 1) % 3;
    const int up = A[(size_t)(i - 1) * v.P + j], same = A[(size_t)i * v.P + j + p1], dn = A[(size_t)(i + 1) * v.P + j - p2];
    v.colour((r + 1) % 3)[(size_t)i * v.P + j] = ((up & 0xf0) << 16) | ((up & 0xf) << 16) | ((same & 0xf00000) >> 8) |
                                                  ((dn & 0x0f0000) >> 8) | ((dn & 0x00f000) >> 8) | ((same & 0xf00) >> 8);
  }
  {
    const int p1 = im == (r + 2) % 3, p2 = im == (r + 1) % 3;
    const int same = A[(size_t)i * v.P + j - p1], up = A[(size_t)(i - 1) * v.P + j + p2], dn = A[(size_t)(i + 1) * v.P + j];
    v.colour((r + 2) % 3)[(size_t)i * v.P + j] = ((same & 0xf000) << 8) | ((up & 0xf00) << 8) | ((up & 0xf0) << 8) |
                                                  ((same & 0xf) << 8) | ((dn & 0xf00000) >> 16) | ((dn & 0x0f0000) >> 16);
  }
}

// Region codes of the extremal tilings of the hexagon of side n (RectTriangleTiler.cpp:
// 480-600), then the shear of row i by n + 3 - i columns into a padded array whose side is a
// multiple of 3.
std::vector<int32_t> hex_extremal(int n, bool top) {
  const int M = 2 * n + 1;
  std::vector<int32_t> t((size_t)M * M, 0);
  auto at = [&](int i, int j) -> int32_t& { return t[(size_t)i * M + j]; };
  for (int i = 1; i < M - 1; ++i)
    for (int j = top ? 0 : 1; j < (top ? M : M - 1); ++j) {
      if (j - i > n || i - j > n) continue;
      int32_t v = 0;
      if (top) {
        if (i < n && j < n) v = 0x333333;
        else if (i < j && j > n) v = 0x111111;
        else if (i > n && i > j) v = 0x222222;
        else if (i == n && j < n) v = 0x333222;
        else if (i < n && j == n) v = 0x331311;
        else if (i == j && i > n) v = 0x211221;
        else if (i == n && j == n) v = 0x331221;
      } else {
        if (i > n && j > n) v = 0x333333;
        else if (i > j && j < n) v = 0x111111;
        else if (i < n && i < j) v = 0x222222;
        else if (i == n && j > n) v = 0x222333;
        else if (i > n && j == n) v = 0x113133;
        else if (i == j && i < n) v = 0x122112;
        else if (i == n && j == n) v = 0x122133;
      }
      at(i, j) = v;
    }
  // the rim of the hexagon: half-covered vertices
  const int32_t edge[2][6] = {{0x001011, 0x000222, 0x330300, 0x333000, 0x200220, 0x011001},
                              {0x003033, 0x000333, 0x110100, 0x222000, 0x100110, 0x022002}};
  const int32_t* e = edge[top ? 1 : 0];
  for (int i = 1; i < n; ++i) at(i, 0) = e[0], at(0, i) = e[1];
  for (int i = n + 1; i < M - 1; ++i) at(i, M - 1) = e[2], at(M - 1, i) = e[3];
  for (int i = 1; i < n; ++i) at(i, i + n) = e[4], at(i + n, i) = e[5];
  if (top) {
    at(0, 0) = 0x000033; at(n, 0) = 0x003002; at(0, n) = 0x000310;
    at(M - 1, M - 1) = 0x210000; at(n, M - 1) = 0x100100; at(M - 1, n) = 0x022000;
  } else {
    at(0, 0) = 0x000012; at(M - 1, n) = 0x013000; at(n, M - 1) = 0x200300;
    at(0, n) = 0x000220; at(n, 0) = 0x001001; at(M - 1, M - 1) = 0x330000;
  }
  const int M2 = M + 6 + (3 - M % 3) % 3;
  std::vector<int32_t> out((size_t)M2 * M2, 0);
  for (int i = 0; i < M; ++i)
    for (int j = 0; j < M; ++j) {
      const int j2 = j + n + 3 - i;
      if (j2 < M2) out[(size_t)(i + 3) * M2 + j2] = t[(size_t)i * M + j];
    }
  return out;
}

// slopeHex (RectTriangleTiler.cpp:173-478): a start tiling of the hexagon of side n with the
// hexagon split into six sloped sectors, each filled with a two-row (or two-column) periodic
// pattern of rectangles, stitched along the three main lines and the diagonal.  Every vertex
// (i, j) of the (2n+1)^2 array takes the code of the first region (in this order) that holds
// it; `alt` picks between a region's two codes.
std::vector<int32_t> hex_slope(int n) {
  const int M = 2 * n + 1;
  const bool ev = n % 2 == 0;
  std::vector<int32_t> t((size_t)M * M, 0);
  auto code = [&](int i, int j) -> int32_t {
    auto pick = [](bool odd, int32_t a, int32_t b) { return odd ? a : b; };
    const bool io = i % 2 == 1, jo = j % 2 == 1, pa = (i + j) % 2 != n % 2;
    if (i == n && j == n) return ev ? 0x213312 : 0x122133;
    if (i == n) {
      if (j < n - 1) return pick(jo, 0x1be1fc, 0xe81c91);
      if (j == n - 1) return ev ? 0x122133 : 0xe81c91;
      if (j > n + 1) return pick(jo, 0xcf1eb1, 0x19c18e);
      return ev ? 0x331221 : 0x29c38e;  // j == n + 1
    }
    if (j == n) {
      if (i < n - 1) return pick(io, 0xd22afc, 0x7af229);
      if (i == n - 1) return ev ? 0x122133 : 0x7af229;
      if (i > n + 1) return pick(io, 0xcfa22d, 0x922fa7);
      return ev ? 0x331221 : 0x913fa7;  // i == n + 1
    }
    if (i == j) {
      if (i < n - 1) return pick(io, 0x33aebd, 0xbd7833);
      if (i > n + 1) return pick(io, 0xdbea33, 0x3387db);
      if (i == n + 1) return ev ? 0x122133 : 0x3387db;
      return ev ? 0x331221 : 0xbd7812;  // i == n - 1
    }
    if (i < n && j < i) {
      if (i == n - 1 && j < i - 1) return pick(jo, 0x855be8, 0x58881b);
      if (i < n - 1 && j == i - 1) return pick(jo, 0x8eb558, 0x58388e);
      if (i == n - 1 && j == i - 1) return ev ? 0x583812 : 0x8ebbe8;
      return pick(jo, 0x855558, 0x588885);
    }
    if (i > n && j > i) {
      if (i == n + 1 && j > i + 1) return pick(jo, 0x8eb558, 0xb18885);
      if (i > n + 1 && j == i + 1) return pick(jo, 0x855be8, 0xe88385);
      if (i == n + 1 && j == i + 1) return ev ? 0x218385 : 0x8ebbe8;
      return pick(jo, 0x855558, 0x588885);
    }
    if (j < n && i < j) {
      if (j == n - 1 && i < j - 1) return pick(io, 0x47d47a, 0x7477d2);
      if (j < n - 1 && i == j - 1) return pick(io, 0xa74d74, 0x7473a7);
      if (j == n - 1 && i == j - 1) return ev ? 0x747312 : 0xa7dd7a;
      return pick(io, 0x474474, 0x747747);
    }
    if (j > n && i > j) {
      if (j == n + 1 && i > j + 1) return pick(io, 0xa74d74, 0x2d7747);
      if (j > n + 1 && i == j + 1) return pick(io, 0x47d47a, 0x7a3747);
      if (j == n + 1 && i == j + 1) return ev ? 0x213747 : 0xa7dd7a;
      return pick(io, 0x474474, 0x747747);
    }
    if (i < n && j > n && i > j - n) {
      if (i == n - 1 && j > n + 1) return pick(pa, 0x6699cf, 0x996f19);
      if (i < n - 1 && j == n + 1) return pick(pa, 0xfc9966, 0x296c99);
      if (i == n - 1 && j == n + 1) return ev ? 0x296319 : 0xfc99cf;
      return pick(pa, 0x669966, 0x996699);
    }
    if (i > n && j < n && i < j + n) {
      if (i == n + 1 && j < n - 1) return pick(pa, 0xfc9966, 0x91f699);
      if (i > n + 1 && j == n - 1) return pick(pa, 0x6699cf, 0x99c692);
      if (i == n + 1 && j == n - 1) return ev ? 0x913692 : 0xfc99cf;
      return pick(pa, 0x669966, 0x996699);
    }
    return 0;
  };
  for (int i = 1; i < M - 1; ++i)
    for (int j = 1; j < M - 1; ++j) t[(size_t)i * M + j] = code(i, j);
  auto at = [&](int i, int j) -> int32_t& { return t[(size_t)i * M + j]; };
  // the rim: runs of half-covered vertices along the six sides, then their ends
  for (int i = 2; i < n - 1; ++i) at(i, 0) = 0x008085, at(0, i) = 0x000747;
  at(1, 0) = 0x00308e, at(0, 1) = 0x0003a7, at(n - 1, 0) = 0x00801b, at(0, n - 1) = 0x0007d2;
  for (int i = n + 2; i < M - 2; ++i) at(i, M - 1) = 0x580800, at(M - 1, i) = 0x747000;
  at(n + 1, M - 1) = 0xb10800, at(M - 1, n + 1) = 0x2d7000, at(M - 2, M - 1) = 0xe80300, at(M - 1, M - 2) = 0x7a3000;
  for (int i = 2; i < n - 1; ++i) at(i, i + n) = 0x900690, at(i + n, i) = 0x096009;
  at(1, n + 1) = 0x200c90, at(n + 1, 1) = 0x01f009, at(n - 1, M - 2) = 0x900f10, at(M - 2, n - 1) = 0x09c002;
  // the six corners (n == 1: the single hexagon of triangles)
  at(0, 0) = n == 1 ? 0x000012 : 0x000033;
  at(M - 1, n) = n == 1 ? 0x013000 : 0x022000;
  at(n, M - 1) = n == 1 ? 0x200300 : 0x100100;
  at(0, n) = 0x000220, at(n, 0) = 0x001001, at(M - 1, M - 1) = 0x330000;
  const int M2 = M + 6 + (3 - M % 3) % 3;
  std::vector<int32_t> out((size_t)M2 * M2, 0);
  for (int i = 0; i < M; ++i)
    for (int j = 0; j < M; ++j) {
      const int j2 = j + n + 3 - i;
      if (j2 < M2) out[(size_t)(i + 3) * M2 + j2] = t[(size_t)i * M + j];
    }
  return out;
}

RtWeights make_weights(const double* w9) {
  // w9 = {wt1, wt2, wt3, wm1, wm2, wm3, wr1, wr2, wr3}; NULL: all 1 (the reference's values)
  float v[9];
  for (int k = 0; k < 9; ++k) v[k] = w9 ? (float)w9[k] : 1.0f;
  RtWeights W;
  const float tab[16] = {0.0f, v[0], v[1], v[2], v[6], v[7], v[8], v[6], v[7], v[8], v[3], v[4], v[5], v[3], v[4], v[5]};
  std::memcpy(W.w, tab, sizeof tab);
  return W;
}

// ---- the cluster kernel ------------------------------------------------------------------------
//
// Every triangle has three vertices, one of each colour, and a vertex's six digits are the codes
// of its six triangles.  So the triangles are the whole state: with A(i, j) the triangle of
// vertices (i, j), (i, j+1), (i-1, j+1) and B(i, j) that of (i, j), (i-1, j), (i-1, j+1), vertex
// (i, j) reads d5..d0 = A(i, j-1), B(i, j), A(i, j), B(i+1, j-1), A(i+1, j-1), B(i+1, j), and a
// move writes those six.  Vertices of one colour share no triangle: a step is one pass over the
// drawn colour, with nothing to rebuild for the two others.
//
// The arrays (two bytes a vertex) live in the shared memory of one thread-block cluster, rows
// split over its CTAs.  A CTA also holds the row of triangles below its last row of vertices, the
// first row of the CTA below; a move on either side of that seam is stored to both copies (plain
// stores through distributed shared memory; a triangle changes at most once a step).  TinyMT
// generators sit in registers, one slot (i, m) each, and a step's draws are made between arrival
// and wait of the barrier that ends the step before.  Only vertices in one of the 17 states that
// move (a 32-entry perfect hash) go on to the weights.
//
// Bound: the cluster barrier of each step.  Side 100, TinyMT: 0.6 us a step (0.9 with the weight
// products and their division at every offered move instead of the tabled ratios); the flip and
// rebuild kernels it replaces took two dependent launches and 4.1 us a step.
constexpr int kRtClCtas = 16;
constexpr int kRtClThreads = 768;  // 85 registers a thread
constexpr int kRtClSlots = 8;      // TinyMT slots a thread
constexpr uint32_t kRtHash = 0xc324c985u;  // (state * kRtHash) >> 27 differs over the 17 states

struct RtClArgs {
  uint8_t *A, *B;  // N x Np bytes each
  int N, M, Np, ctas;
  int row_start[kRtClCtas + 1];  // CTA k owns the vertices of rows [row_start[k], row_start[k + 1])
  const int* cand;               // [2][N]: first (INT_MAX: none) and last slot of each row that can move
  RtWeights W;
  uint4* tmt;                    // generators between launches (all N x M slots)
  const uint4* tmt_params;
  uint32_t seed;                 // TinyMT: generator k <- seed + k when `first`
  bool first, last;              // first (last) launch of the walk
  const uint8_t* colours;        // TinyMT: the colour of each step
  int steps;
  uint64_t fast_seed;
  uint32_t stream;
  int64_t h0;
};

__constant__ int32_t c_rt_states[17] = {0x122133, 0x331221, 0x8ebbe8, 0xfc99cf, 0xa7dd7a, 0x47d47a,
                                        0xd22a33, 0xa74d74, 0x33a22d, 0x8eb558, 0x331eb1, 0x855be8,
                                        0x1be133, 0x6699cf, 0xcf1221, 0xfc9966, 0x1221fc};

__device__ __forceinline__ uint32_t rt_remote(const void* p, int rank) {
  uint32_t r;
  const uint32_t x = (uint32_t)__cvta_generic_to_shared(p);
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(rank));
  return r;
}
__device__ __forceinline__ void rt_store_remote(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.u8 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// K: TinyMT slots a thread (0: fast mode, column quads through a list in shared memory).
template <int K, bool kParams>
__global__ void __launch_bounds__(kRtClThreads, 1) k_rt_cluster(const __grid_constant__ RtClArgs a) {
  extern __shared__ __align__(16) uint8_t rsm[];
  // by state (its hash): the state; by state and quarter of the draw: the state it moves to and the
  // weight ratio (rt_flip's, computed once)
  __shared__ int32_t table[32];
  __shared__ int2 target[32][4];
  constexpr bool kFast = K == 0;
  const int tid = threadIdx.x, T = blockDim.x;
  const int rank = (int)cooperative_groups::this_cluster().block_rank();
  const int r0 = a.row_start[rank], r1 = a.row_start[rank + 1], rows = r1 - r0, Np = a.Np;
  uint8_t* const sA = rsm;
  uint8_t* const sB = rsm + (size_t)(rows + 1) * Np;
  // rows' first unit (slot or quad), then, fast mode, the units
  int* const row_at = reinterpret_cast<int*>(rsm + (size_t)2 * (rows + 1) * Np);
  if (tid < 32) table[tid] = -1;
  __syncthreads();
  for (int k = tid; k < 17 * 4; k += T) {
    const int32_t hex = c_rt_states[k >> 2];
    const uint32_t at = ((uint32_t)hex * kRtHash) >> 27;
    table[at] = hex;
    const int32_t next = rt_target(hex, k & 3);
    target[at][k & 3] = make_int2(next, __float_as_int(ratio_of(a.W, hex, next)));
  }
  for (int k = tid; k < (rows + 1) * (Np / 16); k += T) {
    const size_t g = (size_t)r0 * (Np / 16) + k;
    reinterpret_cast<uint4*>(sA)[k] = reinterpret_cast<const uint4*>(a.A)[g];
    reinterpret_cast<uint4*>(sB)[k] = reinterpret_cast<const uint4*>(a.B)[g];
  }
  auto first_of = [&](int i) { return kFast ? a.cand[i] >> 2 : a.cand[i]; };
  auto last_of = [&](int i) { return kFast ? a.cand[a.N + i] >> 2 : a.cand[a.N + i]; };
  if (tid == 0) {
    int at = 0;
    for (int i = r0; i < r1; ++i) {
      row_at[i - r0] = at;
      if (a.cand[i] != INT_MAX) at += last_of(i) - first_of(i) + 1;
    }
    row_at[rows] = at;
  }
  __syncthreads();
  const int units = row_at[rows];
  // Unit u as row (low 16 bits) and slot or quad.
  auto unit_at = [&](int u) -> uint32_t {
    int lo = 0, hi = rows;  // row_at[lo] <= u < row_at[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) / 2;
      if (row_at[mid] <= u) lo = mid;
      else hi = mid;
    }
    return (uint32_t)lo | (uint32_t)(first_of(r0 + lo) + u - row_at[lo]) << 16;
  };
  const uint32_t upA = rank > 0 ? rt_remote(sA, rank - 1) : 0u;
  const uint32_t dnA = rank + 1 < a.ctas ? rt_remote(sA, rank + 1) : 0u;
  const int rows_up = rank > 0 ? r0 - a.row_start[rank - 1] : 0;
  const int rows_dn = rank + 1 < a.ctas ? a.row_start[rank + 2] - r1 : 0;
  const uint32_t upB = upA + (uint32_t)(rows_up + 1) * Np, dnB = dnA + (uint32_t)(rows_dn + 1) * Np;
  auto state = [&](int ad) -> int32_t {
    return (sA[ad - 1] << 20) | (sB[ad] << 16) | (sA[ad] << 12) | (sB[ad + Np - 1] << 8) | (sA[ad + Np - 1] << 4) |
           sB[ad + Np];
  };
  auto moves = [&](int32_t hex) { return table[((uint32_t)hex * kRtHash) >> 27] == hex; };
  // rt_flip for a state that moves: the same float operations on the tabled ratio
  auto flip = [&](int32_t hex, float rd) -> int32_t {
    if (!(rd < 0.9f)) return hex;
    rd /= 0.9f;
    const int q = (rd < 0.25f ? 0 : 1) + (rd < 0.5f ? 0 : 1) + (rd < 0.75f ? 0 : 1);
    const int2 to = target[((uint32_t)hex * kRtHash) >> 27][q];
    if (rt_five(hex)) rd = (rd - 0.25f * (float)q) * 4;
    return __int_as_float(to.y) >= rd ? to.x : hex;
  };
  auto store = [&](int row, int ad, int32_t n) {
    sA[ad - 1] = (uint8_t)(n >> 20);
    sB[ad] = (uint8_t)((n >> 16) & 15);
    sA[ad] = (uint8_t)((n >> 12) & 15);
    sB[ad + Np - 1] = (uint8_t)((n >> 8) & 15);
    sA[ad + Np - 1] = (uint8_t)((n >> 4) & 15);
    sB[ad + Np] = (uint8_t)(n & 15);
    if (row == 0 && rank > 0) {  // the row below the last row of the CTA above
      const int x = ad + rows_up * Np;
      rt_store_remote(upA + x - 1, (uint32_t)n >> 20);
      rt_store_remote(upB + x, (uint32_t)(n >> 16) & 15u);
      rt_store_remote(upA + x, (uint32_t)(n >> 12) & 15u);
    }
    if (row == rows - 1 && rank + 1 < a.ctas) {  // the first row of the CTA below
      const int x = ad + Np - rows * Np;
      rt_store_remote(dnB + x - 1, (uint32_t)(n >> 8) & 15u);
      rt_store_remote(dnA + x - 1, (uint32_t)(n >> 4) & 15u);
      rt_store_remote(dnB + x, (uint32_t)n & 15u);
    }
  };
  // column offset of colour r's vertex in slot m of row i: j = 3 m + (i - r mod 3)
  auto offset = [](int imod, int r) { return imod - r + (imod < r ? 3 : 0); };

  uint4 gen[kFast ? 1 : K];
  uint32_t unit[kFast ? 1 : K];  // row | slot << 16
  uint32_t draw[kFast ? 1 : K];
  int n_mine = 0;
  if constexpr (!kFast) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int u = tid + k * T;
      gen[k] = make_uint4(0u, 0u, 0u, 0u);
      unit[k] = 0u;
      if (u >= units) continue;
      n_mine = k + 1;
      unit[k] = unit_at(u);
      const int64_t g = (int64_t)(r0 + (int)(unit[k] & 0xffffu)) * a.M + (unit[k] >> 16);
      if (a.first) {
        const uint4 p = kParams ? a.tmt_params[g] : make_uint4(kTmtMat1, kTmtMat2, kTmtTmat, 0);
        gen[k] = tmt_seed(a.seed + (uint32_t)g, p.x, p.y, p.z);
      } else {
        gen[k] = a.tmt[g];
      }
    }
  } else {
    uint32_t* const list = reinterpret_cast<uint32_t*>(row_at + rows + 1);
    for (int u = tid; u < units; u += T) list[u] = unit_at(u);
    __syncthreads();
  }
  auto draw_all = [&] {
    if constexpr (!kFast) {
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (k >= n_mine) continue;
        uint4 p = make_uint4(kTmtMat1, kTmtMat2, kTmtTmat, 0);
        if (kParams) p = __ldg(&a.tmt_params[(int64_t)(r0 + (int)(unit[k] & 0xffffu)) * a.M + (unit[k] >> 16)]);
        draw[k] = tmt_next_u23(gen[k], p.x, p.y, p.z);
      }
    }
  };
  auto colour_at = [&](int s) -> int {
    if (kFast) return (int)((a.h0 + s) % 3);
    return s < a.steps ? (int)__ldg(&a.colours[s]) : 0;
  };
  if (a.steps > 0) draw_all();
  int r = colour_at(0), r_next = colour_at(1);
  cooperative_groups::this_cluster().sync();  // the windows are loaded
  for (int s = 0; s < a.steps; ++s) {
    const int r_after = colour_at(s + 2);
    if constexpr (!kFast) {
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (k >= n_mine) continue;
        const int row = (int)(unit[k] & 0xffffu);
        const int ad = row * Np + 3 * (int)(unit[k] >> 16) + offset((r0 + row) % 3, r);
        const int32_t hex = state(ad);
        if (!moves(hex)) continue;
        const int32_t n = flip(hex, (float)draw[k] * (1.0f / 8388608.0f));
        if (n != hex) store(row, ad, n);
      }
    } else {
      const uint32_t* const list = reinterpret_cast<const uint32_t*>(row_at + rows + 1);
      for (int u = tid; u < units; u += T) {
        const uint32_t e = list[u];
        const int row = (int)(e & 0xffffu), q = (int)(e >> 16), i = r0 + row;
        const int ad0 = row * Np + 12 * q + offset(i % 3, r);
        int32_t hex[4];
        bool any = false;
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) {
          const int m = 4 * q + k4;
          hex[k4] = m >= 1 && m < a.M ? state(ad0 + 3 * k4) : 0;
          if (!moves(hex[k4])) hex[k4] = 0;
          any = any || hex[k4];
        }
        if (!any) continue;
        const uint4 d = fast_quad(a.fast_seed, a.stream, a.h0 + s, (uint32_t)i, (uint32_t)q);
        const uint32_t u4[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) {
          if (!hex[k4]) continue;
          const int32_t n = flip(hex[k4], (float)(u4[k4] >> 8) * (1.0f / 16777216.0f));
          if (n != hex[k4]) store(row, ad0 + 3 * k4, n);
        }
      }
    }
    r = r_next;
    r_next = r_after;
    const bool more = s + 1 < a.steps;
    if (a.ctas == 1) {
      if (more) draw_all();
      __syncthreads();
    } else {
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
      if (more) draw_all();
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
  }
  // (the row below the last vertices belongs to the next CTA, or to the last one)
  const int out_rows = rank + 1 < a.ctas ? rows : rows + 1;
  for (int k = tid; k < out_rows * (Np / 16); k += T) {
    const size_t g = (size_t)r0 * (Np / 16) + k;
    reinterpret_cast<uint4*>(a.A)[g] = reinterpret_cast<const uint4*>(sA)[k];
    reinterpret_cast<uint4*>(a.B)[g] = reinterpret_cast<const uint4*>(sB)[k];
  }
  if constexpr (!kFast) {
    if (a.last) return;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (k < n_mine) a.tmt[(int64_t)(r0 + (int)(unit[k] & 0xffffu)) * a.M + (unit[k] >> 16)] = gen[k];
  }
}

// Tiling (N x N) -> triangle bytes; flag[0] is set when the digits of a triangle differ between its
// vertices, or a vertex in the rows and columns that the reference never rebuilds (row 0 and N - 1,
// slot 0 and M - 1) has a digit: such a state is left to the per-step kernels.  cand as RtClArgs.
__global__ void k_rt_pack(const int32_t* t, int N, int Np, uint8_t* A, uint8_t* B, int* cand, int* flag) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (j >= Np) return;
  int32_t v = 0;
  if (j < N) {
    v = t[(size_t)i * N + j];
    auto digit = [&](int y, int x, int k) { return y >= 0 && x >= 0 && y < N && x < N ? (t[(size_t)y * N + x] >> (4 * k)) & 15 : 0; };
    bool bad = ((v >> 20) & 15) != digit(i, j - 1, 3) || ((v >> 4) & 15) != digit(i + 1, j - 1, 3) ||
               ((v >> 8) & 15) != digit(i + 1, j - 1, 4) || (v & 15) != digit(i + 1, j, 4);
    const int m = j / 3;
    if (v != 0 && (i < 1 || i > N - 2 || m < 1 || m > N / 3 - 2)) bad = true;
    if (bad) *flag = 1;
    bool full = true;
#pragma unroll
    for (int k = 0; k < 6; ++k) full = full && ((v >> (4 * k)) & 15);
    if (full) {
      atomicMin(&cand[i], m);
      atomicMax(&cand[N + i], m);
    }
  }
  A[(size_t)i * Np + j] = (uint8_t)((v >> 12) & 15);
  B[(size_t)i * Np + j] = (uint8_t)((v >> 16) & 15);
}

__global__ void k_rt_unpack(const uint8_t* A, const uint8_t* B, int N, int Np, int32_t* t) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (j >= N) return;
  const size_t x = (size_t)i * Np + j;
  int32_t v = (B[x] << 16) | (A[x] << 12);
  if (j > 0) v |= A[x - 1] << 20;
  if (i + 1 < N) {
    v |= B[x + Np];
    if (j > 0) v |= (B[x + Np - 1] << 8) | (A[x + Np - 1] << 4);
  }
  t[(size_t)i * N + j] = v;
}

void* rt_cluster_kernel(bool fast, bool params, int K) {
  if (fast) return (void*)k_rt_cluster<0, false>;
  switch (K) {
    case 1: return params ? (void*)k_rt_cluster<1, true> : (void*)k_rt_cluster<1, false>;
    case 2: return params ? (void*)k_rt_cluster<2, true> : (void*)k_rt_cluster<2, false>;
    case 3:
    case 4: return params ? (void*)k_rt_cluster<4, true> : (void*)k_rt_cluster<4, false>;
    default: return params ? (void*)k_rt_cluster<8, true> : (void*)k_rt_cluster<8, false>;
  }
}

// Units a step (TinyMT: generator slots; fast mode: column quads) up to which one CTA is faster
// than a cluster and its barrier.
constexpr int kRtOneCta = 1024;

struct RtClPlan {
  bool ok = false;
  int ctas = 0, threads = 0, K = 0;
  int row_start[kRtClCtas + 1] = {};
  size_t smem = 0;
  void* kernel = nullptr;
};

// Rows [first candidate row, last] over the CTAs, the largest share of units as small as possible.
RtClPlan rt_cluster_plan(const int* lo, const int* hi, int N, int Np, bool fast, bool params) {
  RtClPlan p;
  std::vector<int> cnt(N, 0);
  int first = -1, last = -1;
  int64_t total = 0;
  for (int i = 0; i < N; ++i)
    if (lo[i] != INT_MAX) {
      cnt[i] = fast ? (hi[i] >> 2) - (lo[i] >> 2) + 1 : hi[i] - lo[i] + 1;
      total += cnt[i];
      if (first < 0) first = i;
      last = i;
    }
  if (total == 0 || N > 0xffff) return p;
  p.ctas = total <= kRtOneCta ? 1 : std::min(kRtClCtas, last - first + 1);
  auto pack = [&](int64_t cap) -> bool {
    int k = 0;
    int64_t in = 0;
    p.row_start[0] = first;
    for (int i = first; i <= last; ++i) {
      if (in > 0 && in + cnt[i] > cap) {
        if (++k >= p.ctas) return false;
        p.row_start[k] = i;
        in = 0;
      }
      in += cnt[i];
    }
    for (int q = k + 1; q <= p.ctas; ++q) p.row_start[q] = last + 1;
    return true;
  };
  int64_t a = 1, b = total;
  while (a < b) {
    const int64_t mid = (a + b) / 2;
    if (pack(mid)) b = mid;
    else a = mid + 1;
  }
  pack(a);
  while (p.ctas > 1 && p.row_start[p.ctas - 1] > last) --p.ctas;
  int rows_max = 0;
  int64_t units = 0;
  for (int k = 0; k < p.ctas; ++k) {
    rows_max = std::max(rows_max, p.row_start[k + 1] - p.row_start[k]);
    int64_t u = 0;
    for (int i = p.row_start[k]; i < p.row_start[k + 1]; ++i) u += cnt[i];
    units = std::max(units, u);
  }
  p.K = (int)((units + kRtClThreads - 1) / kRtClThreads);
  if (!fast && p.K > kRtClSlots) return p;
  if (!fast) p.K = p.K == 3 ? 4 : p.K > 4 ? 8 : p.K;
  p.threads = p.K > 1 ? kRtClThreads : (int)(units + 31) / 32 * 32;
  p.smem = (size_t)2 * (rows_max + 1) * Np + (size_t)(rows_max + 1) * sizeof(int) + (fast ? (size_t)units * 4 : 0) + 16;
  p.kernel = rt_cluster_kernel(fast, params, p.K);
  if (p.smem > 200 * 1024 ||
      dev_allow_smem(p.kernel, p.smem) != cudaSuccess ||
      cudaFuncSetAttribute(p.kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return p;
  }
  p.ok = true;
  return p;
}

struct RtClLaunch {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  RtClLaunch(const RtClPlan& p, cudaStream_t st) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)p.ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)p.ctas);
    cfg.blockDim = dim3((unsigned)p.threads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
  }
};

// The walk in one cluster; *done stays false (and the tiling as it was) where the state or the
// size is not the cluster kernel's.
rt_status rt_cluster_walk(int32_t* tiling, int N, int64_t steps, int64_t seed, const RtWeights& W, const rt_walk_opts& o,
                          cudaStream_t st, bool* done) {
  *done = false;
  const int M = N / 3, Np = (N + 3 + 15) / 16 * 16;
  const bool fast = o.rng_mode == RT_RNG_FAST;
  const size_t plane = (size_t)(N + 1) * Np, cells = (size_t)N * N;
  struct Buffers {
    cudaStream_t st;
    std::vector<void*> p;
    ~Buffers() {
      for (void* q : p) dev_free(q, st);
    }
    rt_status get(void** out, size_t bytes) {
      const rt_status s = dev_alloc(out, bytes, st);
      if (s == RT_OK) p.push_back(*out);
      return s;
    }
  } buf{st, {}};
  int32_t* d_t = nullptr;
  uint8_t* d_planes = nullptr;
  int* d_cand = nullptr;  // [2][N], flag
  if (rt_status s = buf.get((void**)&d_t, cells * sizeof(int32_t))) return s;
  if (rt_status s = buf.get((void**)&d_planes, 2 * plane)) return s;
  if (rt_status s = buf.get((void**)&d_cand, (2 * (size_t)N + 1) * sizeof(int))) return s;
  std::vector<int> cand(2 * (size_t)N + 1, -1);
  std::fill(cand.begin(), cand.begin() + N, INT_MAX);
  cand[2 * (size_t)N] = 0;
  cudaMemcpyAsync(d_t, tiling, cells * sizeof(int32_t), cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(d_cand, cand.data(), cand.size() * sizeof(int), cudaMemcpyHostToDevice, st);
  cudaMemsetAsync(d_planes, 0, 2 * plane, st);
  const dim3 gp((Np + 127) / 128, N);
  k_rt_pack<<<gp, 128, 0, st>>>(d_t, N, Np, d_planes, d_planes + plane, d_cand, d_cand + 2 * (size_t)N);
  cudaMemcpyAsync(cand.data(), d_cand, cand.size() * sizeof(int), cudaMemcpyDeviceToHost, st);
  cudaError_t e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return fail(RT_ERR_CUDA, std::string("recttri walk: ") + cudaGetErrorString(e));
  if (cand[2 * (size_t)N]) return RT_OK;
  const RtClPlan plan = rt_cluster_plan(cand.data(), cand.data() + N, N, Np, fast, o.tinymt_params != nullptr);
  if (!plan.ok) return RT_OK;
  RtClLaunch launch(plan, st);
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, plan.kernel, &launch.cfg) != cudaSuccess || clusters < 1) {
    cudaGetLastError();
    return RT_OK;
  }
  const int64_t chunk_max = (int64_t)1 << 20;  // steps a launch
  RtClArgs a{};
  a.A = d_planes;
  a.B = d_planes + plane;
  a.N = N;
  a.M = M;
  a.Np = Np;
  a.ctas = plan.ctas;
  std::copy(plan.row_start, plan.row_start + kRtClCtas + 1, a.row_start);
  a.cand = d_cand;
  a.W = W;
  a.seed = (uint32_t)seed;
  a.fast_seed = (uint64_t)seed;
  a.stream = o.fast_stream;
  std::vector<uint8_t> col;
  uint8_t* d_col = nullptr;
  uint4* params = nullptr;
  struct FreeParams {
    uint4*& p;
    ~FreeParams() {
      if (p) cudaFree(p);
    }
  } free_params{params};
  if (!fast) {
    if (rt_status s = tmt_param_table(o, (int64_t)N * M, &params, st)) return s;
    a.tmt_params = params;
    if (steps > chunk_max) {
      if (rt_status s = buf.get((void**)&a.tmt, (size_t)N * M * sizeof(uint4))) return s;
    }
    // RectTriangleTiler.cpp:74-76: colours from default_random_engine(seed)
    std::default_random_engine gen;
    std::uniform_int_distribution<int> dist(0, 2);
    gen.seed(seed);
    col.resize((size_t)steps);
    for (uint8_t& c : col) c = (uint8_t)dist(gen);
    if (rt_status s = buf.get((void**)&d_col, std::max<size_t>(1, col.size()))) return s;
    cudaMemcpyAsync(d_col, col.data(), col.size(), cudaMemcpyHostToDevice, st);
  }
  for (int64_t s0 = 0; s0 < steps; s0 += chunk_max) {
    a.steps = (int)std::min(chunk_max, steps - s0);
    a.first = s0 == 0;
    a.last = s0 + a.steps >= steps;
    a.colours = d_col ? d_col + s0 : nullptr;
    a.h0 = s0;
    void* args[] = {&a};
    e = cudaLaunchKernelExC(&launch.cfg, plan.kernel, args);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return fail(RT_ERR_CUDA, std::string("recttri walk launch: ") + cudaGetErrorString(e));
    }
  }
  k_rt_unpack<<<dim3((N + 127) / 128, N), 128, 0, st>>>(d_planes, d_planes + plane, N, Np, d_t);
  cudaMemcpyAsync(tiling, d_t, cells * sizeof(int32_t), cudaMemcpyDeviceToHost, st);
  e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return fail(RT_ERR_CUDA, std::string("recttri walk: ") + cudaGetErrorString(e));
  *done = true;
  return RT_OK;
}

}  // namespace
}  // namespace rt

using namespace rt;

extern "C" {

RT_API rt_status rt_recttri_hex_tiling(int32_t n, int32_t top, int32_t* out, int64_t cap, int32_t* side) {
  clear_error();
  if (n < 2 || !side || top < 0 || top > 2) return fail(RT_ERR_INVALID_ARGUMENT, "recttri hex_tiling: side n >= 2, top 0, 1 or 2");
  std::vector<int32_t> t = top == 2 ? hex_slope(n) : hex_extremal(n, top != 0);
  const int s = (int)std::lround(std::sqrt((double)t.size()));
  *side = s;
  if (!out || cap < (int64_t)t.size()) return fail(RT_ERR_BUFFER_TOO_SMALL, "recttri hex_tiling: output too small");
  std::memcpy(out, t.data(), t.size() * sizeof(int32_t));
  return RT_OK;
}

// Each lozenge triangle of the domain becomes one triangle of the rectangle-triangle tiling,
// its digit (1, 2, 3) the orientation of the lozenge covering it, written into the three
// vertices around it (RectTriangleTiler.cpp:602-644).  Up triangles (even domain column)
// touch vertices (i, j/2), (i, j/2 + 1), (i + 1, j/2); down triangles (odd column) touch
// (i, j/2 + 1), (i + 1, j/2), (i + 1, j/2 + 1).
RT_API rt_status rt_recttri_from_lozenge(const int32_t* lozenge, int32_t n_side, const int32_t* domain, int32_t m_rows,
                                         int32_t* out) {
  clear_error();
  if (!lozenge || !domain || !out || n_side < 1 || m_rows < 1)
    return fail(RT_ERR_INVALID_ARGUMENT, "recttri from_lozenge: NULL buffer or empty size");
  const int N = n_side, M = m_rows;
  std::fill(out, out + (size_t)N * N, 0);
  for (int i = 0; i < M; ++i)
    for (int j = 0; j < 2 * M; ++j) {
      if (domain[(size_t)i * 2 * M + j] != 1) continue;
      const int64_t a = (int64_t)i * N + j / 2 + (j & 1);  // the vertex whose edge mask is read
      const int64_t v[3] = {a, j & 1 ? a + N - 1 : a + 1, a + N};
      const int sh[3] = {j & 1 ? 4 : 0, j & 1 ? 12 : 8, j & 1 ? 20 : 16};
      if (i + 1 >= N || j / 2 + 1 >= N) return fail(RT_ERR_INVALID_ARGUMENT, "recttri from_lozenge: domain needs padding");
      const int e = lozenge[a];
      const int d = (j & 1) ? ((e & 16) ? 2 : (e & 32) ? 3 : 1) : ((e & 8) ? 1 : (e & 32) ? 3 : 2);
      for (int k = 0; k < 3; ++k) out[v[k]] += d << sh[k];
    }
  return RT_OK;
}

RT_API rt_status rt_recttri_mtgp_draws(int32_t n_side, int64_t seed, int64_t launches, float* out) {
  clear_error();
  if (n_side < 9 || n_side % 3 || n_side > 32766 || launches < 0 || (launches > 0 && !out))
    return fail(RT_ERR_INVALID_ARGUMENT, "recttri mtgp_draws: n_side a multiple of 3 in [9, 32766], launches >= 0");
  return mtgp_draws_grid(n_side, n_side / 3, seed, launches, out);
}

RT_API rt_status rt_recttri_walk(int32_t* tiling, int32_t n_side, int64_t steps, int64_t seed, const double* weights9,
                                 const rt_walk_opts* opts) {
  clear_error();
  rt_walk_opts o;
  rt_walk_opts_default(&o);
  if (opts) o = *opts;
  if (!tiling || steps < 0) return fail(RT_ERR_INVALID_ARGUMENT, "recttri walk: NULL tiling or negative steps");
  if (n_side < 9 || n_side % 3 || n_side > 32766)
    return fail(RT_ERR_INVALID_ARGUMENT, "recttri tiling side must be a multiple of 3 in [9, 32766]");
  if (o.rng_mode != RT_RNG_TINYMT && o.rng_mode != RT_RNG_FAST && o.rng_mode != RT_RNG_MTGP)
    return fail(RT_ERR_INVALID_ARGUMENT, "unknown rng mode");
  if (o.rng_mode == RT_RNG_FAST && o.fast_stream >= 65536u) return fail(RT_ERR_INVALID_ARGUMENT, "fast_stream must be < 65536");
  if (o.tinymt_params && o.rng_mode != RT_RNG_TINYMT)
    return fail(RT_ERR_INVALID_ARGUMENT, "recttri walk: a TinyMT parameter table needs the TinyMT mode");
  uint32_t high = 0;
  for (size_t p = 0; p < (size_t)n_side * n_side; ++p) high |= (uint32_t)tiling[p];
  if (high > 0xffffffu) return fail(RT_ERR_INVALID_ARGUMENT, "recttri tiling values must be six hex digits");
  int devs = 0;
  if (cudaGetDeviceCount(&devs) != cudaSuccess || devs == 0) {
    cudaGetLastError();
    return fail(RT_ERR_CUDA, "no CUDA device: the sweep has no CPU fallback");
  }
  const int N = n_side, M = N / 3, P = (M + 3) / 4 * 4;
  const RtWeights W = make_weights(weights9);
  cudaStream_t stream = (cudaStream_t)o.cuda_stream;
  // The cluster kernel's set-up (packing, a wait for the candidates, a plan) is longer than what a few steps take on a
  // small array (us a call, fast mode, per-step kernels / cluster kernel: N = 12, 1 step 36 / 66, 7 steps 64 / 66; N = 48,
  // 1 step 44 / 72, 7 steps 74 / 72; N = 93, 1 step 68 / 90, 4 steps 87 / 90; N = 144 the cluster at any number).
  const bool few = steps < (N <= 48 ? 8 : N <= 96 ? 4 : 0);
  if (o.rng_mode != RT_RNG_MTGP && steps > 0 && !few) {
    bool done = false;
    if (rt_status st = rt_cluster_walk(tiling, N, steps, seed, W, o, stream, &done)) return st;
    if (done) return RT_OK;
  }
  int32_t* base = nullptr;
  uint4 *tmt = nullptr, *tmt_params = nullptr;
  void* mtgp = nullptr;
  const MtgpGrid mg = mtgp_grid(N, M);
  auto cleanup = [&]() {
    for (void* p : {(void*)base, (void*)tmt, mtgp}) dev_free(p, stream);
    if (tmt_params) cudaFree(tmt_params);
  };
  const size_t cs = (size_t)N * P;
  rt_status status = RT_OK;
  do {
    if (dev_alloc(&base, 3 * cs * sizeof(int32_t), stream) ||
        (o.rng_mode == RT_RNG_TINYMT && dev_alloc(&tmt, (size_t)N * M * sizeof(uint4), stream)) ||
        (o.rng_mode == RT_RNG_MTGP && dev_alloc(&mtgp, mtgp_state_bytes(mg.count()), stream))) {
      status = fail(RT_ERR_OUT_OF_MEMORY, "recttri walk: device allocation failed");
      break;
    }
    // colour split on the host (the reference does the same, RectTriangleTiler.cpp:35-51)
    std::vector<int32_t> h(3 * cs, 0);
    for (int i = 0; i < N; ++i)
      for (int j = 0; j < N; ++j) h[(size_t)(((i - j) % 3 + 3) % 3) * cs + (size_t)i * P + j / 3] = tiling[(size_t)i * N + j];
    cudaMemcpyAsync(base, h.data(), h.size() * sizeof(int32_t), cudaMemcpyHostToDevice, stream);
    if (o.rng_mode == RT_RNG_TINYMT && (status = tmt_param_table(o, (int64_t)N * M, &tmt_params, stream)) != RT_OK) break;
    RtView v{base, N, M, P, cs, tmt, tmt_params};
    const dim3 gr((M + 127) / 128, N), gq(((M + 3) / 4 + 127) / 128, N), gu((M + 127) / 128, N - 2);
    if (o.rng_mode == RT_RNG_TINYMT) {
      const int64_t count = (int64_t)N * M;
      k_rt_seed<<<(unsigned)((count + 255) / 256), 256, 0, stream>>>(tmt, tmt_params, count, (uint32_t)seed);
      // RectTriangleTiler.cpp:74-76: colours from default_random_engine(seed)
      std::default_random_engine gen;
      std::uniform_int_distribution<int> dist(0, 2);
      gen.seed(seed);
      for (int64_t s = 0; s < steps; ++s) {
        const int r = dist(gen);
        pdl_launch(k_rt_flip_tmt, gr, dim3(128), stream, v, r, W);
        pdl_launch(k_rt_update, gu, dim3(128), stream, v, r);
      }
    } else if (o.rng_mode == RT_RNG_MTGP) {
      // RectTriangleTiler.cpp:75-85 (CUDA branch): block generator k seeded seed + k; the
      // colours as above.
      if ((status = mtgp_seed(mtgp, mg.count(), seed, stream)) != RT_OK) break;
      std::default_random_engine gen;
      std::uniform_int_distribution<int> dist(0, 2);
      gen.seed(seed);
      for (int64_t s = 0; s < steps; ++s) {
        const int r = dist(gen);
        pdl_launch(k_rt_flip_mtgp, dim3(mg.gx, mg.gy), dim3(kMtgpBlock, kMtgpBlock), stream, v, r, W,
                   static_cast<curandStateMtgp32*>(mtgp));
        pdl_launch(k_rt_update, gu, dim3(128), stream, v, r);
      }
    } else {
      for (int64_t s = 0; s < steps; ++s) {
        const int r = (int)(s % 3);
        pdl_launch(k_rt_flip_fast, gq, dim3(128), stream, v, r, W, (uint64_t)seed, o.fast_stream, s);
        pdl_launch(k_rt_update, gu, dim3(128), stream, v, r);
      }
    }
    cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) {
      status = fail(RT_ERR_CUDA, std::string("recttri walk: ") + cudaGetErrorString(le));
      break;
    }
    cudaMemcpyAsync(h.data(), base, h.size() * sizeof(int32_t), cudaMemcpyDeviceToHost, stream);
    cudaError_t se = cudaStreamSynchronize(stream);
    if (se != cudaSuccess) {
      status = fail(RT_ERR_CUDA, std::string("recttri walk: ") + cudaGetErrorString(se));
      break;
    }
    for (int i = 0; i < N; ++i)
      for (int j = 0; j < N; ++j) tiling[(size_t)i * N + j] = h[(size_t)(((i - j) % 3 + 3) % 3) * cs + (size_t)i * P + j / 3];
  } while (false);
  cleanup();
  return status;
}

}  // extern "C"
