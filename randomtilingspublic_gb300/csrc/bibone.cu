// Bibone tilings: dimer coverings of regions of the triangular lattice (reference:
// src/TriangleDimer/, class TriangleDimerTiler).
//
// The reference stores, per lattice edge, the states of the edges around it in eight arrays
// (three lozenge, two triangle, three butterfly orientations) and re-derives all of them
// after each move with up to 11 kernels.  Here the state is the dimer configuration itself,
// one byte per vertex (bit 1: H(a,b) = (a,b)-(a,b+1), bit 2: L(a,b) = (a,b)-(a-1,b), bit 4:
// R(a,b) = (a,b)-(a-1,b+1)), and every move of the reference is the toggle of an alternating
// cycle of edges: lozenges (4-cycles, triangledimerkernel.cl:4-22), side-2 triangles
// (6-cycles, :191-211) and butterflies (8-cycles, :331-353).  A step is one kernel: each
// site of the chosen class whose cycle has one half covered flips with probability 1/2.
// Same-class cycles are edge-disjoint (the reference's colourings), and two cycles that can
// flip together share no vertex, so byte read-modify-writes never race.
#include <cuda_runtime.h>
#include <curand_kernel.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "pdl.cuh"
#include "rng.cuh"
#include "rt_internal.h"

namespace rt {
namespace {

enum : uint8_t { kH = 1, kL = 2, kR = 4 };

struct TdEdge {
  int8_t da, db;
  uint8_t bit;
};
struct TdCycle {
  int n;
  TdEdge a[4], b[4];  // the two alternating halves; a = state 5 / 45 / 85, b = 10 / 54 / 170
};

// Cycles by class: lozenge H, L, R (eH/eL/eR of the reference), triangle up / down (tU/tD),
// butterfly H, L, R (bH/bL/bR), at site (a, b).
__constant__ TdCycle c_cycles[8] = {
    {2, {{-1, 0, kR}, {0, 0, kR}}, {{-1, 1, kL}, {0, 0, kL}}},
    {2, {{-1, 0, kH}, {0, -1, kH}}, {{0, 0, kR}, {0, -1, kR}}},
    {2, {{-1, 0, kH}, {0, 0, kH}}, {{0, 1, kL}, {0, 0, kL}}},
    {3, {{-1, 0, kH}, {0, 1, kR}, {1, 0, kL}}, {{0, 0, kL}, {-1, 1, kH}, {1, 0, kR}}},
    {3, {{0, -1, kH}, {0, 1, kL}, {-1, 0, kR}}, {{0, -1, kR}, {0, 0, kH}, {-1, 1, kL}}},
    {4, {{-1, 0, kL}, {-2, 1, kH}, {0, 1, kL}, {0, -1, kH}}, {{-2, 0, kH}, {-1, 1, kR}, {0, 0, kH}, {0, -1, kR}}},
    {4, {{-1, 0, kR}, {0, 1, kL}, {1, -1, kR}, {0, -1, kL}}, {{-1, 1, kL}, {0, 0, kH}, {1, -1, kL}, {-1, -1, kH}}},
    {4, {{-1, 0, kR}, {-1, 1, kH}, {1, 0, kR}, {0, -1, kH}}, {{-1, 1, kL}, {0, 1, kR}, {1, 0, kL}, {0, -1, kR}}},
};

// One step's class: move type (0 lozenge, 1 triangle, 2 butterfly), orientation / colour r1,
// colour r2, butterfly slice p1 and parity p2 (TriangleDimerTiler.cpp:269-276, 459-460).
struct TdStep {
  int type, r1, r2, p1, p2;
};

__host__ __device__ inline int td_cycle_of(const TdStep& s) {
  return s.type == 0 ? s.r1 : s.type == 1 ? (s.r2 == 1 ? 4 : 3) : 5 + s.r1;
}

__host__ __device__ inline bool td_in_class(const TdStep& s, int a, int b) {
  if (s.type == 0) return (((1 - (s.r1 & 1)) * a + ((1 + s.r1) / 2) * b) % 2) == s.r2;
  if (s.type == 1) return (((b - a) % 3 + 3) % 3) == s.r1;
  const int b1 = 1 - (s.r1 & 1), b2 = (1 + s.r1) / 2, b3 = s.r1 & 1;
  return ((b1 * a + b2 * b) % 3) == s.p1 && ((b1 * b + b3 * a) & 1) == s.p2;
}

__device__ __forceinline__ void td_try_flip(uint8_t* D, int M, int c, int a, int b) {
  const TdCycle& C = c_cycles[c];
  bool ha = true, hb = true;
  for (int k = 0; k < C.n; ++k) {
    const int xa = a + C.a[k].da, ya = b + C.a[k].db, xb = a + C.b[k].da, yb = b + C.b[k].db;
    // cycles reaching past the array never move (the padding keeps every domain cycle inside)
    if (xa < 0 || ya < 0 || xa >= M || ya >= M || xb < 0 || yb < 0 || xb >= M || yb >= M) return;
    ha = ha && (D[(size_t)xa * M + ya] & C.a[k].bit);
    hb = hb && (D[(size_t)xb * M + yb] & C.b[k].bit);
  }
  if (!ha && !hb) return;
  for (int k = 0; k < C.n; ++k) {
    D[(size_t)(a + C.a[k].da) * M + b + C.a[k].db] ^= C.a[k].bit;
    D[(size_t)(a + C.b[k].da) * M + b + C.b[k].db] ^= C.b[k].bit;
  }
}

// InitTinyMT (triangledimerkernel.cl:749-756): generator k, of the work item (k / M, k mod M),
// seeded seed + k with its own parameters when a table is loaded.
__global__ void k_td_seed(uint4* st, const uint4* params, int64_t count, uint32_t seed) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  const uint4 p = params ? params[k] : make_uint4(kTmtMat1, kTmtMat2, kTmtTmat, 0);
  st[k] = tmt_seed(seed + (uint32_t)k, p.x, p.y, p.z);
}

// TinyMT mode: every generator draws (as every work item of the reference's rotate kernel
// does); sites of the class flip when rd < 0.5, i.e. the 23-bit draw is below 2^22.
__global__ void k_td_step_tmt(uint8_t* D, uint4* tmt, const uint4* params, int M, TdStep s) {
  pdl_begin();
  const int b = blockIdx.x * blockDim.x + threadIdx.x, a = blockIdx.y;
  if (b >= M) return;
  const size_t k = (size_t)a * M + b;
  uint4 g = tmt[k];
  const uint4 p = params ? params[k] : make_uint4(kTmtMat1, kTmtMat2, kTmtTmat, 0);
  const uint32_t u = tmt_next_u23(g, p.x, p.y, p.z);
  tmt[k] = g;
  if (u < (1u << 22) && td_in_class(s, a, b)) td_try_flip(D, M, td_cycle_of(s), a, b);
}

// MTGP mode: the reference's CUDA launch (8 x 8 blocks over the M x M sites, row a from
// the x index, one cuRAND MTGP32 generator per block, TriangleDimerTiler.cpp:279-291); every
// thread draws before its tests (triangledimerkernel.cu, the three Rotate*Kernel).
__global__ void __launch_bounds__(kMtgpBlock* kMtgpBlock) k_td_step_mtgp(uint8_t* D, int M, TdStep s,
                                                                          curandStateMtgp32* states) {
  pdl_begin();
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y * blockDim.y + threadIdx.y;
  const float rd = curand_uniform(states + blockIdx.x * gridDim.y + blockIdx.y);
  if (a >= M || b >= M) return;
  if (rd < 0.5f && td_in_class(s, a, b)) td_try_flip(D, M, td_cycle_of(s), a, b);
}

// Fast mode: a thread owns columns 4q .. 4q+3 of row a and one Philox block of draws.
__global__ void k_td_step_fast(uint8_t* D, int M, TdStep s, uint64_t seed, uint32_t stream, int64_t h) {
  pdl_begin();
  const int q = blockIdx.x * blockDim.x + threadIdx.x, a = blockIdx.y * blockDim.y + threadIdx.y;
  if (4 * q >= M || a >= M) return;
  bool any = false;
#pragma unroll
  for (int k = 0; k < 4; ++k) any |= (4 * q + k < M) && td_in_class(s, a, 4 * q + k);
  if (!any) return;
  const uint4 d = fast_quad(seed, stream, h, (uint32_t)a, (uint32_t)q);
  const uint32_t u[4] = {d.x, d.y, d.z, d.w};
  const int c = td_cycle_of(s);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int b = 4 * q + k;
    if (b < M && u[k] < 0x80000000u && td_in_class(s, a, b)) td_try_flip(D, M, c, a, b);
  }
}

// ---- the resident kernel -----------------------------------------------------------------------
//
// The dimers as bit planes: per vertex row three planes of 32-bit words (H, L, R), bit k of word w
// for column 32 w + k.  A step is then a handful of logic operations per word: the cycles of 32
// sites have their halves covered where the AND of 2-4 shifted plane words is set, the class is a
// periodic mask, and a flip toggles 4-8 shifted words.  Same-class cycles share no edge, so the
// words are read and toggled (shared-memory XOR) within one step without order, and one barrier
// separates steps.
//
// The rows live in the shared memory of every SM, a band of site rows [own0, own1) per CTA.  A step's sites of
// row a read and change vertex rows a - 2 .. a + 1, so what a band knows shrinks by three rows on each side
// with every step: it starts a period of `depth` steps from 3 depth rows around its own (taken from the
// bands that own them, as 64-bit words tagged with the period, through L2; every wait bounded) and makes
// the steps of its neighbours' sites with its own, draws included.  A small region is one CTA's.
//
// Draws.  Fast mode: only quads of columns with a site that can flip need their Philox block, so a warp
// lists those of its words (about a tenth of them), then draws for the list.  TinyMT: every site's
// generator is in a register of the lane of its column, and a ballot gives a word's acceptance bits.
//
// Bound: the dependent instructions of a step.  Rhombus 512 with one launch per step and a byte per vertex:
// 5.3 us a step on the device, 7.8 in the call; with the rows in one cluster and a cluster barrier per
// step, 2.6 us (TinyMT beyond its registers: 5.1).  Now 1.67 us, TinyMT 1.90; rhombus 300 1.45 (before 2.26) and
// 1.39 (1.94), 66 x 186 1.39 (1.88) and 1.14 (1.19), 20 x 20 0.92 (1.09) and 0.54 (0.61).
constexpr int kTdThreads = 512;  // up to 128 registers a thread
constexpr int kTdSlots = 16;     // TinyMT words a warp

struct TdClArgs {
  uint8_t* D;  // M x M dimer bytes
  int M, bands;
  int w0, words;               // words that hold sites
  int row_lo, row_hi, depth;   // site rows; steps between exchanges
  uint4* tmt;                  // generators between launches
  const uint4* tmt_params;
  uint32_t seed;
  bool first, last;
  const uint8_t* sched;        // packed TdStep per step
  int steps, per_warp;         // per_warp: words of a pass that a warp lists (fast mode)
  uint64_t fast_seed;
  uint32_t stream;
  int64_t h0;
  uint64_t* xbuf;  // [period parity][row from row_lo - 2][word][plane H, L, R], tags cleared
  int* error;
  long max_spin;
  int silent_plus1;  // test hook: this band, less one, publishes nothing
};

// First site row of band b.
__host__ __device__ __forceinline__ int td_band_row(int b, int bands, int lo, int hi) {
  return lo + (int)((int64_t)(hi - lo + 1) * b / bands);
}
constexpr int kTdMove = 4;  // words of an exchange a thread sends, and takes

inline uint8_t td_pack_step(const TdStep& s) {
  return (uint8_t)(s.type | s.r1 << 2 | s.r2 << 4 | s.p1 << 5 | s.p2 << 7);
}
__device__ __forceinline__ TdStep td_unpack_step(uint32_t v) {
  return TdStep{(int)(v & 3u), (int)((v >> 2) & 3u), (int)((v >> 4) & 1u), (int)((v >> 5) & 3u), (int)((v >> 7) & 1u)};
}

// The cycles of c_cycles, edge by edge: f(half, da, db, plane).
template <int V>
struct TdI {
  static constexpr int v = V;
};
template <int kHalf, int kDa, int kDb, int kP, class F>
__device__ __forceinline__ void td_edge(F& f) {
  f(TdI<kHalf>{}, TdI<kDa>{}, TdI<kDb>{}, TdI<kP>{});
}
template <int C, class F>
__device__ __forceinline__ void td_edges(F f) {
  constexpr int H = 0, L = 1, R = 2;
  if constexpr (C == 0) {
    td_edge<0, -1, 0, R>(f), td_edge<0, 0, 0, R>(f);
    td_edge<1, -1, 1, L>(f), td_edge<1, 0, 0, L>(f);
  } else if constexpr (C == 1) {
    td_edge<0, -1, 0, H>(f), td_edge<0, 0, -1, H>(f);
    td_edge<1, 0, 0, R>(f), td_edge<1, 0, -1, R>(f);
  } else if constexpr (C == 2) {
    td_edge<0, -1, 0, H>(f), td_edge<0, 0, 0, H>(f);
    td_edge<1, 0, 1, L>(f), td_edge<1, 0, 0, L>(f);
  } else if constexpr (C == 3) {
    td_edge<0, -1, 0, H>(f), td_edge<0, 0, 1, R>(f), td_edge<0, 1, 0, L>(f);
    td_edge<1, 0, 0, L>(f), td_edge<1, -1, 1, H>(f), td_edge<1, 1, 0, R>(f);
  } else if constexpr (C == 4) {
    td_edge<0, 0, -1, H>(f), td_edge<0, 0, 1, L>(f), td_edge<0, -1, 0, R>(f);
    td_edge<1, 0, -1, R>(f), td_edge<1, 0, 0, H>(f), td_edge<1, -1, 1, L>(f);
  } else if constexpr (C == 5) {
    td_edge<0, -1, 0, L>(f), td_edge<0, -2, 1, H>(f), td_edge<0, 0, 1, L>(f), td_edge<0, 0, -1, H>(f);
    td_edge<1, -2, 0, H>(f), td_edge<1, -1, 1, R>(f), td_edge<1, 0, 0, H>(f), td_edge<1, 0, -1, R>(f);
  } else if constexpr (C == 6) {
    td_edge<0, -1, 0, R>(f), td_edge<0, 0, 1, L>(f), td_edge<0, 1, -1, R>(f), td_edge<0, 0, -1, L>(f);
    td_edge<1, -1, 1, L>(f), td_edge<1, 0, 0, H>(f), td_edge<1, 1, -1, L>(f), td_edge<1, -1, -1, H>(f);
  } else {
    td_edge<0, -1, 0, R>(f), td_edge<0, -1, 1, H>(f), td_edge<0, 1, 0, R>(f), td_edge<0, 0, -1, H>(f);
    td_edge<1, -1, 1, L>(f), td_edge<1, 0, 1, R>(f), td_edge<1, 1, 0, L>(f), td_edge<1, 0, -1, R>(f);
  }
}
// The sites of class s among columns 32 w .. 32 w + 31 of row a (td_in_class); a3, w3: a and w mod 3.
__device__ __forceinline__ uint32_t td_class_mask(const TdStep& s, int a, int a3, int w3) {
  auto every3 = [](int x) -> uint32_t { return 0x49249249u << (x - (x >= 3 ? 3 : 0) - (x >= 6 ? 3 : 0)); };  // x < 9
  auto parity = [](int p) -> uint32_t { return p ? 0xaaaaaaaau : 0x55555555u; };  // (32 w is even, and 32 = 2 mod 3)
  if (s.type == 0) {
    if (s.r1 == 0) return (a & 1) == s.r2 ? ~0u : 0u;
    return parity(s.r1 == 1 ? s.r2 : (s.r2 ^ a) & 1);
  }
  if (s.type == 1) return every3(s.r1 + a3 + w3);
  if (s.r1 == 0) return a3 == s.p1 ? parity(s.p2) : 0u;
  if (s.r1 == 1) return (a & 1) == s.p2 ? every3(s.p1 + w3) : 0u;
  return every3(s.p1 + w3 + (a3 ? 3 - a3 : 0)) & parity(s.p2);
}

// K: TinyMT words a warp (0: fast mode).
template <int K, bool kParams>
__global__ void __launch_bounds__(kTdThreads, 1) k_td_bands(const __grid_constant__ TdClArgs a) {
  extern __shared__ __align__(16) uint32_t tsm[];
  __shared__ uint32_t s_mask[2][18];
  constexpr bool kFast = K == 0;
  const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = T >> 5;
  const int rank = (int)blockIdx.x;
  const int own0 = td_band_row(rank, a.bands, a.row_lo, a.row_hi), own1 = td_band_row(rank + 1, a.bands, a.row_lo, a.row_hi);
  const int reach = a.bands > 1 ? 3 * a.depth : 3;
  const int r0 = max(own0 - reach + 2, a.row_lo), r1 = min(own1 + reach - 1, a.row_hi + 1);  // site rows held
  const int rows = r1 - r0, words = a.words, Wp = words + 2;
  // Window row y is vertex row r0 - 2 + y; word x is column word w0 - 1 + x; planes H, L, R, -.
  uint32_t* const planes = tsm;
  uint32_t* const list = tsm + (size_t)(rows + 3) * Wp * 4;
  auto word = [&](int y, int x, int p) -> uint32_t& { return planes[(y * Wp + x) * 4 + p]; };
  for (int it = warp; it < (rows + 3) * Wp; it += nwarps) {
    const int y = it / Wp, x = it - y * Wp, row = r0 - 2 + y, col = 32 * (a.w0 - 1 + x) + lane;
    const uint32_t v = row >= 0 && row < a.M && col >= 0 && col < a.M ? a.D[(size_t)row * a.M + col] : 0u;
    const uint32_t h = __ballot_sync(~0u, v & kH), l = __ballot_sync(~0u, v & kL), r = __ballot_sync(~0u, v & kR);
    if (lane < 4) word(y, x, lane) = lane == 0 ? h : lane == 1 ? l : lane == 2 ? r : 0u;
  }
  const uint32_t self = (uint32_t)__cvta_generic_to_shared(planes);
  auto toggle_word = [&](int y, int x, int p, uint32_t m) {  // (predicated, not branched)
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %1, 0;\n\t@q red.shared.xor.b32 [%0], %1;\n\t}" ::"r"(
                     self + (uint32_t)((y * Wp + x) * 4 + p) * 4u),
                 "r"(m)
                 : "memory");
  };
  // Sites of the word at `at` whose cycle has a half covered.
  const int pitch = Wp * 4;
  auto covered = [&](auto c, const uint32_t* at) -> uint32_t {
    uint32_t half[2] = {~0u, ~0u};
    td_edges<decltype(c)::v>([&](auto hf, auto da, auto db, auto p) {
      constexpr int d = decltype(db)::v;
      const uint32_t* q = at + decltype(da)::v * pitch + decltype(p)::v;
      const uint32_t v = *q;
      if constexpr (d == 0) half[decltype(hf)::v] &= v;
      else if constexpr (d == 1) half[decltype(hf)::v] &= __funnelshift_r(v, q[4], 1);
      else half[decltype(hf)::v] &= __funnelshift_l(q[-4], v, 1);
    });
    return half[0] | half[1];
  };
  // Flips the sites m of row r0 + i, word x (a cycle spans window rows i .. i + 3).
  auto toggle = [&](auto c, int i, int x, uint32_t m) {
    td_edges<decltype(c)::v>([&](auto, auto da, auto db, auto p) {
      constexpr int d = decltype(db)::v, pl = decltype(p)::v;
      const int yy = i + 2 + decltype(da)::v;
      if constexpr (d == 0) {
        toggle_word(yy, x, pl, m);
      } else if constexpr (d == 1) {
        toggle_word(yy, x, pl, m << 1);
        toggle_word(yy, x + 1, pl, m >> 31);
      } else {
        toggle_word(yy, x, pl, m >> 1);
        toggle_word(yy, x - 1, pl, m << 31);
      }
    });
  };
  auto by_cycle = [](int c, auto f) {  // c is the same for the whole grid
    switch (c) {
      case 0: f(TdI<0>{}); break;
      case 1: f(TdI<1>{}); break;
      case 2: f(TdI<2>{}); break;
      case 3: f(TdI<3>{}); break;
      case 4: f(TdI<4>{}); break;
      case 5: f(TdI<5>{}); break;
      case 6: f(TdI<6>{}); break;
      default: f(TdI<7>{}); break;
    }
  };
  // An item: row r0 + i, word x; its first plane word and its entry of the class masks.
  struct Item {
    int i, x, mask;
    const uint32_t* at;
  };
  auto item_at = [&](int it) -> Item {
    const int i = it / words, x = 1 + it - i * words;
    return Item{i, x, ((r0 + i) % 6) * 3 + (a.w0 - 1 + x) % 3, planes + ((i + 2) * Wp + x) * 4};
  };
  // Its sites that can flip in this step.  (A cycle with a half covered has all its vertices covered,
  // so it lies inside the array.)
  auto sites = [&](int c, int b, const Item& e) -> uint32_t {
    uint32_t m = s_mask[b][e.mask];
    if (m) by_cycle(c, [&](auto cc) { m &= covered(cc, e.at); });
    return m;
  };
  // The class masks of a step by (row mod 6, word mod 3), lane l of a warp the l-th.
  auto make_masks = [&](uint32_t packed, int b) {
    if (lane < 18) s_mask[b][lane] = td_class_mask(td_unpack_step(packed), lane / 3, lane / 3 % 3, lane % 3);
  };
  const int items = rows * words;

  // TinyMT: slot k of a warp is item warp + k * nwarps; lane l keeps the generator of its column l.
  uint4 gen[kFast ? 1 : K];
  uint32_t acc = 0u;  // lane k: the acceptance word of slot k
  auto gen_index = [&](int k, bool* valid) -> int64_t {
    const int it = warp + k * nwarps, row = r0 + it / words, col = 32 * (a.w0 + it % words) + lane;
    *valid = it < items && col < a.M;
    return (int64_t)row * a.M + col;
  };
  if constexpr (!kFast) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      bool v;
      const int64_t g = gen_index(k, &v);
      gen[k] = make_uint4(0u, 0u, 0u, 0u);
      if (!v) continue;
      if (a.first) {
        const uint4 p = kParams ? a.tmt_params[g] : make_uint4(kTmtMat1, kTmtMat2, kTmtTmat, 0);
        gen[k] = tmt_seed(a.seed + (uint32_t)g, p.x, p.y, p.z);
      } else {
        gen[k] = a.tmt[g];
      }
    }
  }
  auto draw = [&] {
    if constexpr (!kFast) {
      uint32_t mine = 0u;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        uint4 p = make_uint4(kTmtMat1, kTmtMat2, kTmtTmat, 0);
        if (kParams) {
          bool v;
          const int64_t g = gen_index(k, &v);
          p = __ldg(&a.tmt_params[v ? g : 0]);
        }
        // the 23-bit draw is below 2^22: the top bit of the tempered word is clear
        const uint32_t ok = __ballot_sync(~0u, (int)tmt_next_t0_mad(gen[k], p.x, p.y, p.z) >= 0);
        mine = lane == k ? ok : mine;
      }
      acc = mine;
    }
  };
  // This thread's item (fast mode: of a step that starts with the first row).
  const int pw = a.per_warp;
  const Item first = item_at(min(kFast ? warp * pw + lane : warp + lane * nwarps, items - 1));
  // The rows of sites, and their items, of a step with `left` steps to go to the exchange, this one included.
  auto row_from = [&](int left) { return max(own0 - 3 * left + 2, r0) - r0; };
  auto row_to = [&](int left) { return min(own1 + 3 * left - 1, r1) - r0; };
  bool dead = false;  // a wait gave up: no more waits, the launch runs to its end
  int send_at[kTdMove], send_to[kTdMove], take_at[kTdMove], take_to[kTdMove];
  const int row_elements = Wp * 3;
  {
    // a vertex row belongs to the band with its site row; the two rows above the first to the first, the row
    // below the last to the last
    const int v0 = rank == 0 ? own0 - 2 : own0, v1 = rank + 1 == a.bands ? own1 + 1 : own1;
    const int mine = min(v1 - v0, 2 * reach);
#pragma unroll
    for (int m = 0; m < kTdMove; ++m) {
      send_at[m] = take_at[m] = -1;
      send_to[m] = take_to[m] = 0;
      const int e = tid + m * T, y = e / row_elements, q = e - y * row_elements, x = q / 3, p = q - 3 * x;
      if (y < mine && rank + 1 != a.silent_plus1) {
        const int row = v1 - v0 <= 2 * reach || y < reach ? v0 + y : v1 - 2 * reach + y;
        send_at[m] = ((row - r0 + 2) * Wp + x) * 4 + p;
        send_to[m] = (row - a.row_lo + 2) * row_elements + q;
      }
      if (y < 2 * reach) {
        const int row = y < reach ? v0 - reach + y : v1 + y - reach;
        if (row >= r0 - 2 && row <= r1 && row >= a.row_lo - 2 && row <= a.row_hi + 1) {
          take_at[m] = ((row - r0 + 2) * Wp + x) * 4 + p;
          take_to[m] = (row - a.row_lo + 2) * row_elements + q;
        }
      }
    }
  }
  auto exchange = [&](uint32_t period) {
    uint64_t* const buf = a.xbuf + (period & 1u) * (uint32_t)((a.row_hi - a.row_lo + 4) * row_elements);
    uint64_t v[kTdMove];
#pragma unroll
    for (int m = 0; m < kTdMove; ++m)
      if (send_at[m] >= 0)
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(buf + send_to[m]),
                     "l"(((uint64_t)(period + 1u) << 32) | planes[send_at[m]])
                     : "memory");
#pragma unroll
    for (int m = 0; m < kTdMove; ++m)
      if (take_at[m] >= 0) asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v[m]) : "l"(buf + take_to[m]) : "memory");
#pragma unroll
    for (int m = 0; m < kTdMove; ++m) {
      if (take_at[m] < 0) continue;
      for (long it = 0; !dead && (uint32_t)(v[m] >> 32) != period + 1u; ++it) {
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v[m]) : "l"(buf + take_to[m]) : "memory");
        if (it >= a.max_spin) {
          dead = true;
          atomicExch(a.error, 1);
        } else if ((it & 1023) == 1023 && *static_cast<volatile int*>(a.error)) {
          dead = true;
        }
      }
      if (!dead) planes[take_at[m]] = (uint32_t)v[m];
    }
    __syncthreads();
  };
  if (a.steps > 0) draw();
  uint32_t step = a.steps > 0 ? __ldg(&a.sched[0]) : 0u, next = a.steps > 1 ? __ldg(&a.sched[1]) : 0u;
  if (warp == nwarps - 1) make_masks(step, 0);
  __syncthreads();  // the window is loaded
  int left = min(a.depth, a.steps);
  uint32_t period = 0;
  for (int s = 0; s < a.steps; ++s) {
    if (left == 0) {
      exchange(period++);
      left = min(a.depth, a.steps - s);
    }
    const int i_lo = row_from(left), i_hi = row_to(left), it_lo = i_lo * words, it_hi = i_hi * words;
    --left;
    const int c = td_cycle_of(td_unpack_step(step));
    step = next;
    next = s + 2 < a.steps ? __ldg(&a.sched[s + 2]) : 0u;
    if constexpr (kFast) {
      if (warp == nwarps - 1) make_masks(step, (s + 1) & 1);
      // A warp's quads with a site that can flip: (row << 20) | (quad << 4) | sites.  (Sites of a class share no edge:
      // the toggles need not wait for the other warps' lists.)
      uint32_t* const mine = list + warp * 8 * pw;
      for (int it0 = it_lo + warp * pw; it0 < it_hi; it0 += nwarps * pw) {
        Item e = first;
        if (it0 >= it_lo + nwarps * pw) {
          e = item_at(min(it0 + lane, items - 1));
        } else if (i_lo) {  // the first item of the whole range, i_lo rows further on
          e.i += i_lo;
          e.mask = ((r0 + e.i) % 6) * 3 + (a.w0 - 1 + e.x) % 3;
          e.at += i_lo * pitch;
        }
        const uint32_t m = lane < pw && it0 + lane < it_hi ? sites(c, s & 1, e) : 0u;
        uint32_t quads = (m | (m >> 1) | (m >> 2) | (m >> 3)) & 0x11111111u;
        int at = __popc(quads);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int before = __shfl_up_sync(~0u, at, o);
          if (lane >= o) at += before;
        }
        const int n = __shfl_sync(~0u, at, 31);
        uint32_t* to = mine + at - __popc(quads);
        const uint32_t tag = (uint32_t)e.i << 20 | (uint32_t)e.x << 7;
        for (; quads; quads &= quads - 1) {
          const int k = __ffs((int)quads) - 1;
          *to++ = tag | (uint32_t)k << 2 | ((m >> k) & 15u);
        }
        __syncwarp();
        for (int q = lane; q < n; q += 32) {
          const uint32_t v = mine[q];
          const int i = (int)(v >> 20), qx = (int)((v >> 4) & 0xffffu), x = qx >> 3, k = qx & 7;
          const uint4 d = fast_quad(a.fast_seed, a.stream, a.h0 + s, (uint32_t)(r0 + i), (uint32_t)(8 * (a.w0 - 1) + qx));
          const uint32_t ok = (~d.x >> 31) | ((~d.y >> 31) << 1) | ((~d.z >> 31) << 2) | ((~d.w >> 31) << 3);
          const uint32_t f = (v & ok & 15u) << (4 * k);
          if (f) by_cycle(c, [&](auto cc) { toggle(cc, i, x, f); });
        }
        __syncwarp();
      }
    } else {
      if (warp == nwarps - 1) make_masks(step, (s + 1) & 1);
      const int it = warp + lane * nwarps;
      if (lane < K && it >= it_lo && it < it_hi) {
        const uint32_t m = sites(c, s & 1, first) & acc;
        if (m) by_cycle(c, [&](auto cc) { toggle(cc, first.i, first.x, m); });
      }
      __syncwarp();
    }
    if (s + 1 < a.steps) draw();
    __syncthreads();
  }
  // No band writes back before the bands around it have loaded.
  if (a.bands > 1 && a.steps > 0) exchange(period);
  for (int it = warp; it < (own1 - own0) * words; it += nwarps) {
    const int i = own0 - r0 + it / words, x = 1 + it % words, col = 32 * (a.w0 - 1 + x) + lane;
    if (col >= a.M) continue;
    uint32_t v = 0;
#pragma unroll
    for (int p = 0; p < 3; ++p) v |= ((word(i + 2, x, p) >> lane) & 1u) << p;
    a.D[(size_t)(r0 + i) * a.M + col] = (uint8_t)v;
  }
  if constexpr (!kFast) {
    if (a.last) return;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      bool v;
      const int64_t g = gen_index(k, &v);
      const int row = r0 + (warp + k * nwarps) / words;
      if (v && row >= own0 && row < own1) a.tmt[g] = gen[k];
    }
  }
}

// ---- between the reference's tiling format and the dimer bytes, on the device ---------------------

// What k_td_pack finds: bit 0 of flags a state that is not a dimer configuration's, bit 1 two dimers
// at a vertex, bit 2 a dimer that leaves the array; the rows and columns of the covered vertices; their number by (row, column) mod 6.
struct TdScan {
  unsigned flags;
  int row_lo, row_hi, col_lo, col_hi;
  unsigned long long by_residue[36];
};

inline TdScan td_no_scan(int M) {
  TdScan scan{};
  scan.row_lo = scan.col_lo = M;
  scan.row_hi = scan.col_hi = -1;
  return scan;
}

__device__ __forceinline__ uint32_t td_byte(const int32_t* t, int N, int M, int a, int b) {
  if (a < 0 || b < 0 || a >= M || b >= M) return 0u;
  const int eR = t[(size_t)(2 * a + 1) * N + 2 * b + 1], eH = t[(size_t)(2 * a) * N + 2 * b + 1];
  return ((eR & 4) ? kH : 0) | ((eR & 8) ? kL : 0) | ((eH & 4) ? kR : 0);
}

// td_from_tiling, and the checks of a walk's input (td_to_tiling gives the tiling back, at most
// one dimer at a vertex).
__global__ void k_td_pack(const int32_t* t, int N, uint8_t* D, TdScan* scan) {
  __shared__ unsigned hist[36];
  __shared__ int s_lo, s_hi;  // this block's covered columns
  const int M = N / 2, b = blockIdx.x * blockDim.x + threadIdx.x, a = blockIdx.y;
  for (int k = threadIdx.x; k < 36; k += blockDim.x) hist[k] = 0u;
  if (threadIdx.x == 0) s_lo = M, s_hi = -1;
  __syncthreads();
  if (b < M) {
    auto bit = [&](int y, int x, uint32_t k) -> int { return (td_byte(t, N, M, y, x) & k) ? 1 : 0; };
    const uint32_t v = td_byte(t, N, M, a, b);
    D[(size_t)a * M + b] = (uint8_t)v;
    const int h = (v & kH) ? 1 : 0, l = (v & kL) ? 1 : 0, r = (v & kR) ? 1 : 0;
    const int nR = bit(a - 1, b, kR), nH = bit(a - 1, b, kH), wH = bit(a, b - 1, kH), wR = bit(a, b - 1, kR);
    const int eL = bit(a, b + 1, kL), neL = bit(a - 1, b + 1, kL);
    unsigned flags = 0;
    if (t[(size_t)(2 * a) * N + 2 * b + 1] != nR + 2 * neL + 4 * r + 8 * l) flags |= 1u;
    if (t[(size_t)(2 * a + 1) * N + 2 * b] != nH + 2 * r + 4 * wH + 8 * wR) flags |= 1u;
    if (t[(size_t)(2 * a + 1) * N + 2 * b + 1] != nH + 2 * eL + 4 * h + 8 * l) flags |= 1u;
    const int cover = h + l + r + wH + bit(a + 1, b, kL) + bit(a + 1, b - 1, kR);
    if (cover > 1) flags |= 2u;
    if ((a == 0 && (l || r)) || (b == M - 1 && (h || r))) flags |= 4u;
    if (flags) atomicOr(&scan->flags, flags);
    if (cover) {
      atomicMin(&s_lo, b);
      atomicMax(&s_hi, b);
      atomicAdd(&hist[(a % 6) * 6 + b % 6], 1u);
    }
  }
  __syncthreads();
  for (int k = threadIdx.x; k < 36; k += blockDim.x)
    if (hist[k]) atomicAdd(&scan->by_residue[k], (unsigned long long)hist[k]);
  if (threadIdx.x == 0 && s_hi >= 0) {
    atomicMin(&scan->row_lo, a);
    atomicMax(&scan->row_hi, a);
    atomicMin(&scan->col_lo, s_lo);
    atomicMax(&scan->col_hi, s_hi);
  }
}

// td_to_tiling on the device (the (even, even) entries stay).
__global__ void k_td_unpack(const uint8_t* D, int N, int32_t* t) {
  const int M = N / 2, b = blockIdx.x * blockDim.x + threadIdx.x, a = blockIdx.y;
  if (b >= M) return;
  auto bit = [&](int y, int x, int k) -> int {
    return (y >= 0 && x >= 0 && y < M && x < M && (D[(size_t)y * M + x] & k)) ? 1 : 0;
  };
  const int nH = bit(a - 1, b, kH), r = bit(a, b, kR), l = bit(a, b, kL);
  t[(size_t)(2 * a) * N + 2 * b + 1] = bit(a - 1, b, kR) + 2 * bit(a - 1, b + 1, kL) + 4 * r + 8 * l;
  t[(size_t)(2 * a + 1) * N + 2 * b] = nH + 2 * r + 4 * bit(a, b - 1, kH) + 8 * bit(a, b - 1, kR);
  t[(size_t)(2 * a + 1) * N + 2 * b + 1] = nH + 2 * bit(a, b + 1, kL) + 4 * bit(a, b, kH) + 8 * l;
}

struct TdClPlan {
  bool ok = false;
  int bands = 0, threads = 0, K = 0, w0 = 0, words = 0, depth = 0, per_warp = 1;
  size_t smem = 0, xbuf_words = 0;
  void* kernel = nullptr;
};

void* td_kernel(bool fast, bool params, int K) {
  if (fast) return (void*)k_td_bands<0, false>;
  switch (K) {
    case 1: return params ? (void*)k_td_bands<1, true> : (void*)k_td_bands<1, false>;
    case 2: return params ? (void*)k_td_bands<2, true> : (void*)k_td_bands<2, false>;
    case 4: return params ? (void*)k_td_bands<4, true> : (void*)k_td_bands<4, false>;
    case 8: return params ? (void*)k_td_bands<8, true> : (void*)k_td_bands<8, false>;
    default: return params ? (void*)k_td_bands<16, true> : (void*)k_td_bands<16, false>;
  }
}

// Bands of equally many rows with an exchange every `depth` steps.
TdClPlan td_plan_of(const TdScan& sc, bool fast, bool params, int bands, int depth) {
  TdClPlan p;
  const int rows = sc.row_hi - sc.row_lo + 1;
  p.w0 = sc.col_lo / 32;
  p.words = sc.col_hi / 32 - p.w0 + 1;
  p.bands = std::min(bands, rows);
  p.depth = depth;
  int held = 0, own = 0;
  for (int k = 0; k < p.bands; ++k) {
    const int o0 = td_band_row(k, p.bands, sc.row_lo, sc.row_hi), o1 = td_band_row(k + 1, p.bands, sc.row_lo, sc.row_hi);
    held = std::max(held, std::min(o1 + 3 * depth - 1, sc.row_hi + 1) - std::max(o0 - 3 * depth + 2, sc.row_lo));
    own = std::max(own, o1 - o0 + 2);
  }
  const int64_t items = (int64_t)held * p.words;
  p.smem = (size_t)(held + 3) * (p.words + 2) * 16;
  int64_t threads = std::min<int64_t>(kTdThreads, (items + 31) / 32 * 32);
  if (p.bands > 1) {
    const int64_t moves = (int64_t)6 * depth * (p.words + 2) * 3;
    if (moves > (int64_t)kTdMove * kTdThreads) return p;
    threads = std::max(threads, (moves + kTdMove * 32 - 1) / (kTdMove * 32) * 32);
  }
  if (fast) {
    threads = std::min<int64_t>(kTdThreads, std::max<int64_t>(threads, std::min<int64_t>(items, 16) * 32));
    p.threads = (int)threads;
    p.per_warp = (int)std::min<int64_t>(32, (items + p.threads / 32 - 1) / (p.threads / 32));
    p.smem += (size_t)(p.threads / 32) * 8 * p.per_warp * sizeof(uint32_t);
    if (held > 4095 || p.words + 2 > 8191) return p;
  } else {
    const int64_t K = (items + kTdThreads / 32 - 1) / (kTdThreads / 32);
    if (K > kTdSlots) return p;
    p.K = K <= 1 ? 1 : K <= 2 ? 2 : K <= 4 ? 4 : K <= 8 ? 8 : 16;
    p.threads = K <= 1 ? (int)std::max(threads, items * 32) : kTdThreads;
  }
  p.xbuf_words = (size_t)2 * (rows + 3) * (p.words + 2) * 3;
  p.kernel = td_kernel(fast, params, p.K);
  int per_sm = 0;
  if (p.smem > 200 * 1024 ||
      dev_allow_smem(p.kernel, p.smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, p.kernel, p.threads, p.smem) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    return p;
  }
  p.ok = true;
  return p;
}

TdClPlan td_plan(const TdScan& sc, bool fast, bool params) {
  int dev = 0, sms = 0, coop = 0;
  if (sc.row_hi < sc.row_lo || sc.flags || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess) {
    cudaGetLastError();
    return TdClPlan{};
  }
  // One CTA where that is faster than any exchange (us per step, rhombus 20 x 20: fast mode 0.92, bands 0.96 at
  // best; TinyMT 0.54 and 0.61; 60 x 60: 1.27 and 1.26, 1.15 and 0.87).  Else a band per SM, and the deeper the fewer
  // words a band then holds, whose draws with TinyMT are all made:
  //   fast    66 x 186: depth 2 1.54, 3 1.42, 4 1.39    300 x 300: 1.58, 1.50, 1.45    512 x 512: 1.77, 1.70, 1.67
  //   TinyMT  60 x 60 (40 words): 2 0.95, 3 0.87    66 x 186 (66): 1 1.45, 2 1.14, 3 1.24    300 x 300 (120): 1.56,
  //           1.39, 1.91    512 x 512 (238 at depth 2): 1.90, 2.21
  const int rows = sc.row_hi - sc.row_lo + 1, words = sc.col_hi / 32 - sc.col_lo / 32 + 1;
  TdClPlan p;
  if (!coop || rows * words <= (fast ? 128 : 32)) {
    p = td_plan_of(sc, fast, params, 1, 1);
    if (p.ok || !coop) return p;
  }
  const auto held = [&](int d) { return ((rows + sms - 1) / sms + 6 * d - 3) * words; };
  int depth = fast ? 4 : (held(3) <= 51 ? 3 : (held(2) <= 128 ? 2 : 1));
  for (; depth > 0 && !p.ok; --depth) p = td_plan_of(sc, fast, params, sms, depth);
  return p;
}

struct TdClLaunch {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  TdClLaunch(const TdClPlan& p, cudaStream_t st) {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.gridDim = dim3((unsigned)p.bands);
    cfg.blockDim = dim3((unsigned)p.threads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = p.bands > 1 ? 1 : 0;
  }
};

// Philox4x32-10 on the host (the fast-mode step schedule).
void philox_host(uint32_t c[4], uint32_t k0, uint32_t k1) {
  for (int r = 0; r < 10; ++r) {
    const uint64_t p0 = (uint64_t)0xD2511F53u * c[0], p1 = (uint64_t)0xCD9E8D57u * c[2];
    const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c[1] ^ k0, n1 = (uint32_t)p1, n2 = (uint32_t)(p0 >> 32) ^ c[3] ^ k1,
                   n3 = (uint32_t)p0;
    c[0] = n0, c[1] = n1, c[2] = n2, c[3] = n3;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
}

// Fast-mode schedule: step h's class from Philox(ctr = {~0, ~0, lo32(h), hi16(h) | s << 16}).
TdStep td_fast_step(uint64_t seed, uint32_t stream, int64_t h) {
  uint32_t c[4] = {0xffffffffu, 0xffffffffu, (uint32_t)(uint64_t)h,
                   ((uint32_t)((uint64_t)h >> 32) & 0xffffu) | (stream << 16)};
  philox_host(c, (uint32_t)seed, (uint32_t)(seed >> 32));
  return TdStep{(int)(c[0] % 3u), (int)(c[1] % 3u), (int)(c[2] & 1u), (int)((c[3] >> 1) % 3u), (int)(c[3] & 1u)};
}

void td_from_tiling(const int32_t* t, int N, uint8_t* D) {
  const int M = N / 2;
  for (int a = 0; a < M; ++a)
    for (int b = 0; b < M; ++b) {
      const int eR = t[(size_t)(2 * a + 1) * N + 2 * b + 1], eH = t[(size_t)(2 * a) * N + 2 * b + 1];
      D[(size_t)a * M + b] = (uint8_t)(((eR & 4) ? kH : 0) | ((eR & 8) ? kL : 0) | ((eH & 4) ? kR : 0));
    }
}

// Lozenge states from the dimers (the reference's tiling format); the (even, even) entries,
// which hold no state, are left as they are.
void td_to_tiling(const uint8_t* D, int N, int32_t* t) {
  const int M = N / 2;
  auto bit = [&](int a, int b, int k) -> int {
    return (a >= 0 && b >= 0 && a < M && b < M && (D[(size_t)a * M + b] & k)) ? 1 : 0;
  };
  for (int a = 0; a < M; ++a)
    for (int b = 0; b < M; ++b) {
      t[(size_t)(2 * a) * N + 2 * b + 1] = bit(a - 1, b, kR) + 2 * bit(a - 1, b + 1, kL) + 4 * bit(a, b, kR) + 8 * bit(a, b, kL);
      t[(size_t)(2 * a + 1) * N + 2 * b] = bit(a - 1, b, kH) + 2 * bit(a, b, kR) + 4 * bit(a, b - 1, kH) + 8 * bit(a, b - 1, kR);
      t[(size_t)(2 * a + 1) * N + 2 * b + 1] = bit(a - 1, b, kH) + 2 * bit(a, b + 1, kL) + 4 * bit(a, b, kH) + 8 * bit(a, b, kL);
    }
}

// Number of dimers at each vertex: 0 off the domain, 1 on it for a dimer covering.
std::vector<int> td_cover(const uint8_t* D, int M) {
  std::vector<int> c((size_t)M * M, 0);
  auto add = [&](int a, int b) {
    if (a >= 0 && b >= 0 && a < M && b < M) ++c[(size_t)a * M + b];
  };
  for (int a = 0; a < M; ++a)
    for (int b = 0; b < M; ++b) {
      const uint8_t v = D[(size_t)a * M + b];
      if (v & kH) add(a, b), add(a, b + 1);
      if (v & kL) add(a, b), add(a - 1, b);
      if (v & kR) add(a, b), add(a - 1, b + 1);
    }
  return c;
}

// Side of the vertex array up to which a walk's conversions are made on the host: two launches, a wait and two pool
// blocks less, 10 ns a vertex more (walk of one step, fast mode, host / device: side 10 47 / 74 us, 46 72 / 81, 70
// 115 / 106, 106 169 / 110).
constexpr int kTdHostSide = 48;

// k_td_pack on the host.
TdScan td_pack_host(const int32_t* tiling, int N, std::vector<uint8_t>* bytes) {
  const int M = N / 2;
  std::vector<uint8_t>& D = *bytes;
  D.resize((size_t)M * M);
  td_from_tiling(tiling, N, D.data());
  TdScan scan = td_no_scan(M);
  std::vector<int32_t> back(tiling, tiling + (size_t)N * N);
  td_to_tiling(D.data(), N, back.data());
  if (!std::equal(back.begin(), back.end(), tiling)) scan.flags |= 1u;
  const std::vector<int> cover = td_cover(D.data(), M);
  for (int a = 0; a < M; ++a)
    for (int b = 0; b < M; ++b) {
      const uint8_t v = D[(size_t)a * M + b];
      if ((a == 0 && (v & (kL | kR))) || (b == M - 1 && (v & (kH | kR)))) scan.flags |= 4u;
      if (!cover[(size_t)a * M + b]) continue;
      if (cover[(size_t)a * M + b] > 1) scan.flags |= 2u;
      scan.row_lo = std::min(scan.row_lo, a);
      scan.row_hi = std::max(scan.row_hi, a);
      scan.col_lo = std::min(scan.col_lo, b);
      scan.col_hi = std::max(scan.col_hi, b);
      ++scan.by_residue[(a % 6) * 6 + b % 6];
    }
  return scan;
}

rt_status td_check(const TdScan& scan) {
  if (scan.flags & 1u)
    return fail(RT_ERR_INVALID_ARGUMENT, "bibone walk: tiling states are not those of a dimer configuration");
  if (scan.flags & 2u) return fail(RT_ERR_INVALID_ARGUMENT, "bibone walk: two dimers share a vertex");
  return RT_OK;
}

}  // namespace
}  // namespace rt

using namespace rt;

extern "C" {

RT_API rt_status rt_td_icecream_cone(int32_t n, int32_t m, int32_t* out, int64_t cap, int32_t* side) {
  clear_error();
  if (n < 1 || m < 0 || !side) return fail(RT_ERR_INVALID_ARGUMENT, "bibone icecream_cone: n >= 1, m >= 0");
  const int E = n + 4, T = 2 * E, k = ((n + 1) * (n + 2) / 2) % 2;
  *side = T;
  if (!out || cap < (int64_t)T * T) return fail(RT_ERR_BUFFER_TOO_SMALL, "bibone icecream_cone: output too small");
  // As the reference, the layout is built even when m > n - 1 or the vertex count is odd (it
  // prints a warning and covers the domain less its top-right vertex).
  // The reference's dimer layout (TriangleDimerTiler.cpp:714-740): horizontal dimers in every
  // other column, the slanted right side closed by L / R dimers, the cut corner staggered
  std::vector<uint8_t> D((size_t)E * E, 0);
  auto set = [&](int a, int b, uint8_t bit) {
    if (a >= 0 && a < E) D[(size_t)a * E + b] |= bit;
  };
  for (int i = 2; i < E - 2; ++i)
    for (int j = 2; j < E - i; ++j) {
      if (i < m + 2) {
        if ((i + j) % 2 == m % 2 && (m != 0 && j > m + 3 - i)) set(i - 1, j, kH);
        if ((n - m) % 2 == 0 && (i % 2) == 0 && j == E - i - 1) set(i, j, kR);
      } else {
        const bool closes_l = i % 4 == (3 + n % 2 + 2 * k) % 4 && j == E - i - 1;
        if (j % 2 == 0 && !closes_l) set(i - 1, j, kH);
        if (closes_l) set(i, j, kL);
        if (i % 4 == (2 + n % 2 + 2 * k) % 4 && j == E - i - 1) set(i, j, kR);
      }
    }
  std::vector<int32_t> t((size_t)T * T, 0);
  td_to_tiling(D.data(), T, t.data());
  for (int i = 0; i < T; ++i)
    for (int j = 0; j < T; ++j)
      out[(size_t)i * T + j] = (i >= 3 && j >= 3 && i < T - 1 && j < T - 1) ? t[(size_t)i * T + j] : 0;
  return RT_OK;
}

// TriangleDimerTiler::TestButterfly(type) (TriangleDimerTiler.cpp:795-845): one butterfly of
// orientation type (0 H, 1 L, 2 R) of four dimers in a side-16 tiling; other types give the
// all-zero tiling (the reference prints a message).
RT_API rt_status rt_td_test_butterfly(int32_t type, int32_t* out, int64_t cap, int32_t* side) {
  clear_error();
  const int E = 8, T = 2 * E;
  if (!side) return fail(RT_ERR_INVALID_ARGUMENT, "test_butterfly: side is NULL");
  *side = T;
  if (!out || cap < (int64_t)T * T) return fail(RT_ERR_BUFFER_TOO_SMALL, "test_butterfly: output too small");
  std::fill(out, out + (size_t)T * T, 0);
  if (type < 0 || type > 2) return RT_OK;
  std::vector<uint8_t> D((size_t)E * E, 0);
  auto set = [&](int a, int b, uint8_t bit) { D[(size_t)a * E + b] |= bit; };
  // the reference's h edges sit one vertex row below the edge they stand for
  if (type == 0) set(1, 3, kH), set(3, 3, kH), set(2, 4, kR), set(3, 2, kR);
  else if (type == 1) set(2, 3, kR), set(4, 2, kR), set(3, 2, kL), set(3, 4, kL);
  else set(2, 4, kL), set(4, 3, kL), set(3, 2, kR), set(3, 4, kR);
  std::vector<int32_t> t((size_t)T * T, 0);
  td_to_tiling(D.data(), T, t.data());
  for (int i = 3; i < T - 1; ++i)
    for (int j = 3; j < T - 1; ++j) out[(size_t)i * T + j] = t[(size_t)i * T + j];
  return RT_OK;
}

// TriangleDimerTiler::TilingToTriangleFlips (:846-873): (N/2) x N; row i, even column j the
// state of the down triangle, odd column the up triangle, as three base-4 digits (the edge of
// each neighbouring triangle that holds a dimer: 1, 2, 3, or 0), read from the lozenge states.
RT_API rt_status rt_td_triangle_flips(const int32_t* t, int32_t n_side, int32_t* out) {
  clear_error();
  if (!t || !out || n_side < 4 || n_side % 2) return fail(RT_ERR_INVALID_ARGUMENT, "triangle_flips: even side >= 4");
  const int N = n_side;
  auto at = [&](int i, int j) { return t[(size_t)i * N + j]; };
  std::fill(out, out + (size_t)(N / 2) * N, 0);
  for (int i = 1; i < N / 2 - 1; ++i)
    for (int j = 1; j < N - 1; ++j) {
      const int eL = at(2 * i + 1, j), eR = at(2 * i + 1, j + 1), eU = at(2 * i, j + 1);  // j even: down triangle
      int v;
      if (j % 2 == 0) {
        v = (((eL >> 2) & 1) + 2 * ((eL >> 3) & 1) + 3 * ((eR >> 3) & 1)) +
            4 * (((eR >> 2) & 1) + 2 * ((eL >> 1) & 1) + 3 * ((eR >> 1) & 1)) +
            16 * (2 * (eU & 1) + (eL & 1) + 3 * ((eU >> 1) & 1));
      } else {
        const int r = at(2 * i + 1, j), l = at(2 * i + 1, j + 1), h = at(2 * i + 2, j);  // odd: up triangle
        v = ((r & 1) + 2 * ((r >> 3) & 1) + 3 * ((l >> 3) & 1)) + 4 * ((l & 1) + 2 * ((r >> 1) & 1) + 3 * ((l >> 1) & 1)) +
            16 * (2 * ((h >> 3) & 1) + 3 * ((h >> 2) & 1) + ((r >> 2) & 1));
      }
      out[(size_t)i * N + j] = v;
    }
  return RT_OK;
}

// TriangleDimerTiler::TilingToButterflyFlips (:875-921): N x N, at each H / L / R position
// the four neighbouring triangles' digits (weights 1, 4, 16, 64) and the centre edge (256).
RT_API rt_status rt_td_butterfly_flips(const int32_t* t, int32_t n_side, int32_t* out) {
  clear_error();
  if (!t || !out || n_side < 4 || n_side % 2) return fail(RT_ERR_INVALID_ARGUMENT, "butterfly_flips: even side >= 4");
  const int N = n_side;
  auto at = [&](int i, int j) { return t[(size_t)i * N + j]; };
  auto bit = [](int v, int k) { return (v >> k) & 1; };
  std::fill(out, out + (size_t)N * N, 0);
  for (int i = 2; i < N - 2; ++i)
    for (int j = 2; j < N - 2; ++j) {
      const int c0 = at(i, j);
      int f1, f4, f16, f64, c;
      if (i % 2 == 0) {
        if (j % 2 == 0) continue;
        const int up = at(i - 1, j), upr = at(i - 1, j + 1), dn = at(i + 1, j), dnl = at(i + 1, j - 1);
        f1 = bit(up, 3) + 2 * bit(up, 0) + 3 * bit(c0, 0);
        f4 = bit(upr, 0) + 2 * bit(upr, 1) + 3 * bit(c0, 1);
        f16 = bit(dn, 1) + 2 * bit(dn, 2) + 3 * bit(c0, 2);
        f64 = bit(dnl, 2) + 2 * bit(dnl, 3) + 3 * bit(c0, 3);
        c = bit(upr, 2);
      } else if (j % 2 == 0) {
        const int ur = at(i - 1, j + 1), rr = at(i, j + 1), dl = at(i + 1, j - 1), ll = at(i, j - 1);
        f1 = bit(ur, 0) + 2 * bit(ur, 1) + 3 * bit(c0, 0);
        f4 = bit(rr, 1) + 2 * bit(rr, 2) + 3 * bit(c0, 1);
        f16 = bit(dl, 2) + 2 * bit(dl, 3) + 3 * bit(c0, 2);
        f64 = bit(ll, 3) + 2 * bit(ll, 0) + 3 * bit(c0, 3);
        c = bit(rr, 3);
      } else {
        const int uu = at(i - 1, j), rr = at(i, j + 1), dd = at(i + 1, j), ll = at(i, j - 1);
        f1 = bit(uu, 0) + 2 * bit(uu, 1) + 3 * bit(c0, 0);
        f4 = bit(rr, 0) + 2 * bit(rr, 1) + 3 * bit(c0, 1);
        f16 = bit(dd, 2) + 2 * bit(dd, 3) + 3 * bit(c0, 2);
        f64 = bit(ll, 2) + 2 * bit(ll, 3) + 3 * bit(c0, 3);
        c = bit(rr, 3);
      }
      out[(size_t)i * N + j] = f1 + 4 * f4 + 16 * f16 + 64 * f64 + 256 * c;
    }
  return RT_OK;
}

RT_API rt_status rt_td_rhombus_brick(int32_t rows, int32_t cols, int32_t* out, int64_t cap, int32_t* side) {
  clear_error();
  if (rows < 1 || cols < 2 || cols % 2 || !side)
    return fail(RT_ERR_INVALID_ARGUMENT, "bibone rhombus: rows >= 1 and an even number of columns >= 2");
  const int M = std::max(rows, cols) + 6, T = 2 * M;
  *side = T;
  if (!out || cap < (int64_t)T * T) return fail(RT_ERR_BUFFER_TOO_SMALL, "bibone rhombus: output too small");
  std::vector<uint8_t> D((size_t)M * M, 0);
  for (int a = 0; a < rows; ++a)
    for (int b = 0; b < cols; b += 2) D[(size_t)(a + 3) * M + b + 3] = kH;
  std::fill(out, out + (size_t)T * T, 0);
  td_to_tiling(D.data(), T, out);
  return RT_OK;
}

RT_API rt_status rt_td_dimers(const int32_t* t, int32_t n_side, uint8_t* out) {
  clear_error();
  if (!t || !out || n_side < 2 || n_side % 2) return fail(RT_ERR_INVALID_ARGUMENT, "bibone dimers: even side >= 2");
  td_from_tiling(t, n_side, out);
  return RT_OK;
}

RT_API rt_status rt_td_from_dimers(const uint8_t* dimers, int32_t n_side, int32_t* out) {
  clear_error();
  if (!dimers || !out || n_side < 2 || n_side % 2) return fail(RT_ERR_INVALID_ARGUMENT, "bibone from_dimers: even side >= 2");
  td_to_tiling(dimers, n_side, out);
  return RT_OK;
}

// TriangleDimerTiler::TilingToVertices (TriangleDimerTiler.cpp:923-949): an (N/2+1)^2 grid,
// entry (i, j) (2 <= i, j < N/2 - 1) is 1 when vertex (i-1, j) is covered by a dimer.
RT_API rt_status rt_td_vertices(const int32_t* tiling, int32_t n_side, int32_t* out) {
  clear_error();
  if (!tiling || !out || n_side < 4 || n_side % 2) return fail(RT_ERR_INVALID_ARGUMENT, "bibone vertices: even side >= 4");
  const int M = n_side / 2, V = M + 1;
  std::vector<uint8_t> D((size_t)M * M);
  td_from_tiling(tiling, n_side, D.data());
  const std::vector<int> c = td_cover(D.data(), M);
  std::fill(out, out + (size_t)V * V, 0);
  for (int i = 2; i < V - 2; ++i)
    for (int j = 2; j < V - 2; ++j) out[(size_t)i * V + j] = c[(size_t)(i - 1) * M + j] > 0;
  return RT_OK;
}

// TriangleDimerTiler::TilingToDomain (:951-982): (V-1) x 2(V-1) triangles over the vertex grid
// above, even columns the triangle (i, j/2), (i, j/2+1), (i+1, j/2), odd columns
// (i, j/2+1), (i+1, j/2), (i+1, j/2+1); 1 when all three vertices are covered.
RT_API rt_status rt_td_domain(const int32_t* tiling, int32_t n_side, int32_t* out) {
  clear_error();
  if (!tiling || !out || n_side < 4 || n_side % 2) return fail(RT_ERR_INVALID_ARGUMENT, "bibone domain: even side >= 4");
  const int V = n_side / 2 + 1;
  std::vector<int32_t> v((size_t)V * V);
  rt_td_vertices(tiling, n_side, v.data());
  auto at = [&](int i, int j) { return v[(size_t)i * V + j]; };
  for (int i = 0; i < V - 1; ++i)
    for (int j = 0; j < 2 * (V - 1); ++j) {
      const bool in = j % 2 == 0 ? (at(i, j / 2) && at(i, j / 2 + 1) && at(i + 1, j / 2))
                                 : (at(i, j / 2 + 1) && at(i + 1, j / 2) && at(i + 1, j / 2 + 1));
      out[(size_t)i * 2 * (V - 1) + j] = in ? 1 : 0;
    }
  return RT_OK;
}

// TriangleDimerTiler::DimerIndicator(t, c) (:35-99): M x M, for c = 0 the horizontal dimers
// (entry (a, b) is the edge (a-1, b)-(a-1, b+1)), c = 1 the up-left ones (a, b)-(a-1, b),
// c = 2 the up-right ones (a, b)-(a-1, b+1).
RT_API rt_status rt_td_dimer_indicator(const int32_t* tiling, int32_t n_side, int32_t c, int32_t* out) {
  clear_error();
  if (!tiling || !out || n_side < 4 || n_side % 2 || c < 0 || c > 2)
    return fail(RT_ERR_INVALID_ARGUMENT, "bibone dimer_indicator: even side >= 4, c in {0, 1, 2}");
  const int M = n_side / 2;
  std::vector<uint8_t> D((size_t)M * M);
  td_from_tiling(tiling, n_side, D.data());
  for (int a = 0; a < M; ++a)
    for (int b = 0; b < M; ++b) {
      const int v = c == 0 ? (a > 0 ? (D[(size_t)(a - 1) * M + b] & kH) : 0)
                           : (D[(size_t)a * M + b] & (c == 1 ? kL : kR));
      out[(size_t)a * M + b] = v ? 1 : 0;
    }
  return RT_OK;
}

RT_API rt_status rt_td_mtgp_draws(int32_t n_side, int64_t seed, int64_t launches, float* out) {
  clear_error();
  if (n_side < 8 || n_side % 2 || n_side > 2 * 32767 || launches < 0 || (launches > 0 && !out))
    return fail(RT_ERR_INVALID_ARGUMENT, "bibone mtgp_draws: even n_side in [8, 65534], launches >= 0");
  return mtgp_draws_grid(n_side / 2, n_side / 2, seed, launches, out);
}

RT_API rt_status rt_td_walk(int32_t* tiling, int32_t n_side, int64_t steps, int64_t seed, const rt_walk_opts* opts,
                            rt_cftp_stats* stats) {
  clear_error();
  rt_walk_opts o;
  rt_walk_opts_default(&o);
  if (opts) o = *opts;
  if (!tiling || steps < 0) return fail(RT_ERR_INVALID_ARGUMENT, "bibone walk: NULL tiling or negative steps");
  if (n_side < 8 || n_side % 2 || n_side > 2 * 32767)
    return fail(RT_ERR_INVALID_ARGUMENT, "bibone tiling side must be even, in [8, 65534]");
  if (o.rng_mode != RT_RNG_TINYMT && o.rng_mode != RT_RNG_FAST && o.rng_mode != RT_RNG_MTGP)
    return fail(RT_ERR_INVALID_ARGUMENT, "unknown rng mode");
  if (o.rng_mode == RT_RNG_FAST && o.fast_stream >= 65536u) return fail(RT_ERR_INVALID_ARGUMENT, "fast_stream must be < 65536");
  if (o.tinymt_params && o.rng_mode != RT_RNG_TINYMT)
    return fail(RT_ERR_INVALID_ARGUMENT, "bibone walk: a TinyMT parameter table needs the TinyMT mode");
  const int N = n_side, M = N / 2;
  int devs = 0;
  if (cudaGetDeviceCount(&devs) != cudaSuccess || devs == 0) {
    cudaGetLastError();
    std::vector<uint8_t> bytes;
    if (rt_status cs = td_check(td_pack_host(tiling, N, &bytes))) return cs;  // an input is refused before a missing device
    return fail(RT_ERR_CUDA, "no CUDA device: the sweep has no CPU fallback");
  }
  cudaStream_t st = (cudaStream_t)o.cuda_stream;
  const bool fast = o.rng_mode == RT_RNG_FAST;
  const size_t cells = (size_t)N * N;
  int32_t* d_t = nullptr;
  uint8_t* dD = nullptr;
  TdScan* d_scan = nullptr;
  uint8_t* d_sched = nullptr;
  uint4 *tmt = nullptr, *tmt_params = nullptr;
  uint64_t* xbuf = nullptr;
  int* d_error = nullptr;
  void* mtgp = nullptr;
  const MtgpGrid mg = mtgp_grid(M, M);
  auto cleanup = [&]() {
    for (void* q : {(void*)d_t, (void*)dD, (void*)d_scan, (void*)d_sched, (void*)tmt, (void*)xbuf, (void*)d_error, mtgp})
      dev_free(q, st);
    if (tmt_params) cudaFree(tmt_params);
  };
  auto out_of_memory = [&]() {
    cleanup();
    return fail(RT_ERR_OUT_OF_MEMORY, "bibone walk: device allocation failed");
  };
  TdScan scan = td_no_scan(M);
  std::vector<uint8_t> bytes;
  const dim3 g_all((M + 127) / 128, M), g_quad(((M + 3) / 4 + 31) / 32, (M + 7) / 8);
  // (on the host too where the device has no room for the tiling's words, 16 times the bytes)
  const bool on_device = M > kTdHostSide && !dev_alloc(&d_t, cells * sizeof(int32_t), st) &&
                         !dev_alloc(&d_scan, sizeof(TdScan), st);
  clear_error();
  if (!on_device) {
    scan = td_pack_host(tiling, N, &bytes);
    if (rt_status cs = td_check(scan)) {
      cleanup();
      return cs;
    }
  }
  if (dev_alloc(&dD, (size_t)M * M, st)) return out_of_memory();
  if (on_device) {
    cudaMemcpyAsync(d_t, tiling, cells * sizeof(int32_t), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(d_scan, &scan, sizeof scan, cudaMemcpyHostToDevice, st);
    k_td_pack<<<g_all, 128, 0, st>>>(d_t, N, dD, d_scan);
    cudaMemcpyAsync(&scan, d_scan, sizeof scan, cudaMemcpyDeviceToHost, st);
    const cudaError_t pe = cudaStreamSynchronize(st);
    if (pe != cudaSuccess) {
      cleanup();
      return fail(RT_ERR_CUDA, std::string("bibone walk: ") + cudaGetErrorString(pe));
    }
    if (rt_status cs = td_check(scan)) {
      cleanup();
      return cs;
    }
  } else {
    cudaMemcpyAsync(dD, bytes.data(), bytes.size(), cudaMemcpyHostToDevice, st);
  }
  TdClPlan plan;
  if (o.rng_mode != RT_RNG_MTGP && steps > 0) {
    plan = td_plan(scan, fast, o.tinymt_params != nullptr);
  }
  TdClLaunch launch(plan, st);
  const bool resident = plan.ok, exchanges = plan.ok && plan.bands > 1;
  constexpr int64_t chunk_max = (int64_t)1 << 18;  // steps of a launch
  if ((o.rng_mode == RT_RNG_TINYMT && (!resident || steps > chunk_max) &&
       dev_alloc(&tmt, (size_t)M * M * sizeof(uint4), st)) ||
      (resident && dev_alloc(&d_sched, (size_t)steps, st)) ||
      (exchanges && (dev_alloc(&xbuf, plan.xbuf_words * sizeof(uint64_t), st) || dev_alloc(&d_error, sizeof(int), st))) ||
      (o.rng_mode == RT_RNG_MTGP && dev_alloc(&mtgp, mtgp_state_bytes(mg.count()), st)))
    return out_of_memory();
  if (o.rng_mode == RT_RNG_TINYMT) {
    if (rt_status ps = tmt_param_table(o, (int64_t)M * M, &tmt_params, st)) {
      cleanup();
      return ps;
    }
  }
  std::vector<TdStep> sched((size_t)steps);
  if (o.rng_mode != RT_RNG_FAST) {
    // TriangleDimerTiler.cpp:269-276, 459-460: type, r1, r2 (and p1, p2 for butterflies)
    std::default_random_engine gen;
    std::uniform_int_distribution<int> d1(0, 2), d2(0, 1);
    gen.seed(seed);
    for (auto& s : sched) {
      s.type = d1(gen);
      s.r1 = d1(gen);
      s.r2 = d2(gen);
      s.p1 = s.p2 = 0;
      if (s.type == 2) s.p1 = d1(gen), s.p2 = d2(gen);
    }
  } else {
    for (int64_t h = 0; h < steps; ++h) sched[(size_t)h] = td_fast_step((uint64_t)seed, o.fast_stream, h);
  }
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  if (o.rng_mode == RT_RNG_TINYMT && !resident) {
    const int64_t count = (int64_t)M * M;
    k_td_seed<<<(unsigned)((count + 255) / 256), 256, 0, st>>>(tmt, tmt_params, count, (uint32_t)seed);
  } else if (o.rng_mode == RT_RNG_MTGP) {
    // TriangleDimerTiler.cpp:287-289: block generator k seeded seed + k
    if (rt_status ms = mtgp_seed(mtgp, mg.count(), seed, st)) {
      cudaEventDestroy(e0);
      cudaEventDestroy(e1);
      cleanup();
      return ms;
    }
  }
  std::vector<uint8_t> packed;
  if (resident) {
    packed.resize((size_t)steps);
    for (int64_t h = 0; h < steps; ++h) packed[(size_t)h] = td_pack_step(sched[(size_t)h]);
    cudaMemcpyAsync(d_sched, packed.data(), packed.size(), cudaMemcpyHostToDevice, st);
  }
  cudaError_t le = cudaSuccess;
  cudaEventRecord(e0, st);
  for (int64_t s0 = 0; resident && s0 < steps && le == cudaSuccess; s0 += chunk_max) {
    TdClArgs a{};
    a.D = dD;
    a.M = M;
    a.bands = plan.bands;
    a.w0 = plan.w0;
    a.words = plan.words;
    a.tmt = tmt;
    a.tmt_params = tmt_params;
    a.seed = (uint32_t)seed;
    a.first = s0 == 0;
    a.steps = (int)std::min(chunk_max, steps - s0);
    a.last = s0 + a.steps >= steps;
    a.sched = d_sched + s0;
    a.per_warp = plan.per_warp;
    a.fast_seed = (uint64_t)seed;
    a.stream = o.fast_stream;
    a.h0 = s0;
    a.depth = exchanges ? plan.depth : a.steps;
    a.row_lo = scan.row_lo;
    a.row_hi = scan.row_hi;
    a.xbuf = xbuf;
    a.error = d_error;
    a.max_spin = test_silence().spin(1L << 22);
    a.silent_plus1 = test_silence().next_plus1();
    if (exchanges) {
      if (s0 == 0) cudaMemsetAsync(d_error, 0, sizeof(int), st);
      cudaMemsetAsync(xbuf, 0, plan.xbuf_words * sizeof(uint64_t), st);  // no stale tags
    }
    void* args[] = {&a};
    le = cudaLaunchKernelExC(&launch.cfg, plan.kernel, args);
  }
  for (int64_t h = 0; !resident && h < steps; ++h) {
    if (o.rng_mode == RT_RNG_TINYMT)
      pdl_launch(k_td_step_tmt, g_all, dim3(128), st, dD, tmt, (const uint4*)tmt_params, M, sched[(size_t)h]);
    else if (o.rng_mode == RT_RNG_MTGP)
      pdl_launch(k_td_step_mtgp, dim3(mg.gx, mg.gy), dim3(kMtgpBlock, kMtgpBlock), st, dD, M, sched[(size_t)h],
                 static_cast<curandStateMtgp32*>(mtgp));
    else
      pdl_launch(k_td_step_fast, g_quad, dim3(32, 8), st, dD, M, sched[(size_t)h], (uint64_t)seed, o.fast_stream, h);
  }
  cudaEventRecord(e1, st);
  if (on_device) k_td_unpack<<<g_all, 128, 0, st>>>(dD, N, d_t);
  if (le == cudaSuccess) le = cudaGetLastError();
  int gave_up = 0;
  if (exchanges && le == cudaSuccess) {  // before the caller's tiling changes
    cudaMemcpyAsync(&gave_up, d_error, sizeof gave_up, cudaMemcpyDeviceToHost, st);
    le = cudaStreamSynchronize(st);
    if (gave_up && le == cudaSuccess) {
      cudaEventDestroy(e0);
      cudaEventDestroy(e1);
      cleanup();
      return fail(RT_ERR_TIMEOUT, "bibone walk: a band gave up waiting for a neighbour's rows");
    }
  }
  if (le == cudaSuccess && on_device) cudaMemcpyAsync(tiling, d_t, cells * sizeof(int32_t), cudaMemcpyDeviceToHost, st);
  if (le == cudaSuccess && !on_device) cudaMemcpyAsync(bytes.data(), dD, bytes.size(), cudaMemcpyDeviceToHost, st);
  const cudaError_t se = cudaStreamSynchronize(st);
  float ms = 0.f;
  if (se == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cleanup();
  if (le != cudaSuccess || se != cudaSuccess)
    return fail(RT_ERR_CUDA, std::string("bibone walk: ") + cudaGetErrorString(le != cudaSuccess ? le : se));
  if (!on_device) td_to_tiling(bytes.data(), N, tiling);
  if (stats) {
    std::memset(stats, 0, sizeof *stats);
    // per class, the sites whose anchor vertex is covered: the classes have periods 2 and 3
    int64_t attempts = 0;
    std::vector<int64_t> per_class(3 * 3 * 2 * 3 * 2, -1);
    for (const TdStep& s : sched) {
      const size_t key = (((size_t)s.type * 3 + s.r1) * 2 + s.r2) * 6 + (s.type == 2 ? s.p1 * 2 + s.p2 : 0);
      if (per_class[key] < 0) {
        int64_t c = 0;
        for (int a = 0; a < 6; ++a)
          for (int b = 0; b < 6; ++b)
            if (td_in_class(s, a, b)) c += (int64_t)scan.by_residue[a * 6 + b];
        per_class[key] = c;
      }
      attempts += per_class[key];
    }
    stats->attempts = 1;
    stats->total_steps = steps;
    stats->final_steps = steps;
    stats->flip_attempts = attempts;
    stats->seconds = ms * 1e-3;
  }
  return RT_OK;
}

}  // extern "C"
