// One CTA's coupled chains as bit planes: the look-back of one attempt of a domino or lozenge
// instance (batch_cftp.cu).
//
// State: one bit per lattice edge, as in domino_cluster.cu and lozenge_bits.cu, both chains of a word
// side by side; a flip toggles a vertex's edges and there is no passive colour to rebuild.  Only
// inputs whose edges agree at both ends and whose flip candidates border no cell that the reference
// never rebuilds are held this way (bp_load tells); the others keep the byte kernels (batch_cftp.cuh).
//
// Warps of their own draw, a few half-sweeps (steps) ahead; the others apply the moves.  Draws are made for bytes of
// eight cells that hold a candidate, one lane a Philox block (four cells), so a diamond draws for half of its bounding
// box.
//
// Bound: the issue of the draws, about 220 cycles of a scheduler for 32 blocks (160 of them Philox's
// products), and in a CTA alone on its SM an update's latency.  Measured (GB300): hexagon of side 32, one CTA,
// attempts side by side, 23.1 ms (bytes of both chains with a rebuild pass: 253 ms, attempts in turn); 64 mixed
// diamonds (orders 16-48) and hexagons (sides 8-32) 34 ms (226), 512 of them 65 (246).  Every warp drawing and updating
// in turn, a barrier a step: 29.5, 39.4 and 73-82 ms; 192 or 256 update threads of the 512: 27.6 and 25.4 ms for the hexagon.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "batch_cftp.cuh"
#include "rng.cuh"

namespace rt {

// Shared memory of one instance, offsets in 32-bit words.
struct BpLayout {
  int W;                                           // 32-cell words a row
  int period;                                      // steps between the barriers of the whole CTA
  int planes, valid, moves, items, units, stage;  // stage shares its words with moves, items and units
  int words;                                       // all
};
constexpr int kBpUpdate = 128;      // threads that update, of a CTA; the others draw
constexpr int kBpDominoWord = 8;    // [2 chains]{VD0, VD1, HE, HO}
constexpr int kBpLozengeWord = 24;  // [2 chains]{E0-2, NE0-2, N0-2, three of padding}

// smem: bytes to keep within, if fewer steps a period do (a smaller side may ask for more than a larger one, whose
// period is shorter).
__host__ __device__ inline BpLayout bp_layout(int model, int N, int P, size_t smem = ~(size_t)0) {
  BpLayout L;
  const int PW = model == 0 ? kBpDominoWord : kBpLozengeWord;
  L.W = ((model == 0 ? N / 2 : N / 3) + 31) / 32;
  L.planes = PW;  // a word of padding in front, one after each row
  L.valid = L.planes + (N + (model == 0 ? 0 : 1)) * (L.W + 1) * PW;
  L.moves = L.stage = (L.valid + N * L.W + 3) & ~3;
  // As many steps a period as 32 KB of moves hold, but 2 to 8: a hexagon of side 32 alone 29.5 ms with 1, 24.0 with 4, 23.1
  // with 8.
  const int staged = L.stage + (model == 0 ? 2 : 3) * N * P / 4;
  for (L.period = N * L.W <= 256 ? 8 : N * L.W <= 512 ? 4 : 2;; L.period /= 2) {
    L.items = L.moves + 2 * L.period * 2 * N * L.W;  // [period parity][step][word] pairs of words
    L.units = L.items + N * L.W;
    L.words = L.units + 4 * N * L.W;
    if (L.words < staged) L.words = staged;
    if (L.period == 2 || (size_t)L.words * 4 <= smem) return L;
  }
}
inline size_t bp_bytes(int model, int N, int P) { return (size_t)bp_layout(model, N, P).words * 4; }

// The byte of cell (i, m) of a colour from the planes (domino: colour t; lozenge: residue q of the column).
__device__ __forceinline__ uint32_t bp_domino_cell(const uint32_t* sm, const BpLayout& L, int c, int t, int i, int m) {
  const uint32_t* me = sm + L.planes + (i * (L.W + 1) + (m >> 5)) * kBpDominoWord + 4 * c;
  const int b = m & 31;
  const uint32_t up = i > 0 ? (me[-(L.W + 1) * kBpDominoWord + 1 - t] >> b) & 1u : 0u, dn = (me[t] >> b) & 1u;
  const uint32_t he = (me[2] >> b) & 1u;
  uint32_t left, right;
  if ((i + 1 - t) & 1) {
    left = he;
    right = (me[3] >> b) & 1u;
  } else {
    left = b ? (me[3] >> (b - 1)) & 1u : me[3 - kBpDominoWord] >> 31;
    right = he;
  }
  return up | (dn << 1) | (left << 2) | (right << 3);
}
__device__ __forceinline__ uint32_t bp_lozenge_cell(const uint32_t* sm, const BpLayout& L, int c, int q, int i, int m) {
  const uint32_t* p = sm + L.planes + (i * (L.W + 1) + (m >> 5)) * kBpLozengeWord + 12 * c;
  const uint32_t* d = p + (L.W + 1) * kBpLozengeWord;
  const int b = m & 31, qw = q == 0 ? 2 : q - 1;
  auto west = [&](const uint32_t* at) {  // the bit of column j - 1
    return q ? (at[0] >> b) & 1u : b ? (at[0] >> (b - 1)) & 1u : at[-kBpLozengeWord] >> 31;
  };
  return ((p[q] >> b) & 1u) * 8u + ((p[3 + q] >> b) & 1u) * 2u + ((p[6 + q] >> b) & 1u) + west(p + qw) * 4u +
         west(d + 3 + qw) * 16u + ((d[6 + q] >> b) & 1u) * 32u;
}

// Four bytes (word w of a chain's colour arrays) of chain c.
__device__ __forceinline__ uint32_t bp_bytes_of(const uint32_t* sm, const BpLayout& L, const DevInstance& in, int c, int w) {
  const int per_row = in.P / 4, k = w / (in.N * per_row), i = (w / per_row) % in.N, m = 4 * (w % per_row);
  uint32_t v = 0;
  for (int b = 0; b < 4; ++b) {
    if (m + b >= 32 * L.W) break;
    v |= (in.model == 0 ? bp_domino_cell(sm, L, c, k, i, m + b)
                        : bp_lozenge_cell(sm, L, c, (i + k) % 3, i, m + b)) << (8 * b);
  }
  return v;
}

// Loads both chains (0: from the min tiling, 1: from the max tiling); cnt: three shared words.  False
// (for every thread) where the planes cannot hold them.
template <int kThreads>
__device__ bool bp_load(uint32_t* sm, const BpLayout& L, const DevInstance& in, const uint32_t* gmax, const uint32_t* gmin,
                        int* cnt) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int N = in.N, P = in.P, W = L.W;
  const bool domino = in.model == 0;
  const int rows = domino ? N : N + 1, words = (domino ? 2 : 3) * N * P / 4;
  if (tid < 3) cnt[tid] = 0;
  for (int k = tid; k < L.planes; k += kThreads) sm[k] = 0u;
  const uint8_t* const stage = reinterpret_cast<const uint8_t*>(sm + L.stage);
  // byte of vertex (i, j)
  auto at = [&](int i, int j) -> uint32_t {
    if (i < 0 || j < 0 || i >= N || j >= N) return 0u;
    return domino ? stage[((((i + j) & 1) ? 0 : 1) * N + i) * P + (j >> 1)]
                  : stage[((((j - i) % 3 + 3) % 3) * N + i) * P + j / 3];
  };
  for (int c = 0; c < 2; ++c) {
    __syncthreads();
    const uint32_t* g = c ? gmax : gmin;
    for (int k = tid; k < words; k += kThreads) sm[L.stage + k] = __ldcv(g + k);
    __syncthreads();
    bool bad = false;
    for (int it = warp; it < rows * (W + 1); it += kThreads / 32) {
      const int i = it / (W + 1), x = it - i * (W + 1), m = 32 * x + lane;
      uint32_t* const p = sm + L.planes + it * (domino ? kBpDominoWord : kBpLozengeWord) + (domino ? 4 : 12) * c;
      if (x == W || i == N) {
        if (lane < (domino ? 4 : 12)) p[lane] = 0u;
        continue;
      }
      const bool inside = m < P;
      bool cand = false;
      if (domino) {
        const uint32_t b0 = inside ? stage[i * P + m] : 0u, b1 = inside ? stage[(N + i) * P + m] : 0u;
        const uint32_t bo = (i & 1) ? b1 : b0;  // the colour whose cells sit at odd lattice columns
        const uint32_t vd0 = __ballot_sync(~0u, b0 & 2u), vd1 = __ballot_sync(~0u, b1 & 2u);
        const uint32_t he = __ballot_sync(~0u, bo & 4u), ho = __ballot_sync(~0u, bo & 8u);
        if (lane < 4) p[lane] = lane == 0 ? vd0 : lane == 1 ? vd1 : lane == 2 ? he : ho;
        bad = bad || (i == N - 1 && ((b0 | b1) & 2u)) || (m == N / 2 - 1 && (bo & 8u));  // edges that leave the array
        if (i >= 1 && i <= N - 2 && m >= 1 && m <= N / 2 - 2) {
          auto sq = [&](int a, int b) { return (at(a, b) & 10u) || (at(a + 1, b + 1) & 5u); };  // a covered square
          const int j = 2 * m;
          const bool mid = sq(i - 1, j) && sq(i, j);
          const bool even = mid && sq(i - 1, j - 1) && sq(i, j - 1), odd = mid && sq(i - 1, j + 1) && sq(i, j + 1);
          cand = even || odd;
          bad = bad || (cand && (i < 2 || i > N - 3)) || (even && m < 2) || (odd && m > N / 2 - 3);
        }
      } else {
        uint32_t bits[9];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const int col = (q + 3 - i % 3) % 3, j = 3 * m + q;  // colour of residue q in row i
          const uint32_t v = inside ? stage[(col * N + i) * P + m] : 0u;
          bits[q] = __ballot_sync(~0u, v & 8u);
          bits[3 + q] = __ballot_sync(~0u, v & 2u);
          bits[6 + q] = __ballot_sync(~0u, v & 1u);
          bad = bad || (i == 0 && (v & 3u)) || (j == N - 1 && (v & 10u));
          auto A = [&](int y, int z) { return (at(y, z) & 10u) || (at(y, z + 1) & 1u); };
          auto B = [&](int y, int z) { return (at(y, z) & 3u) || (at(y - 1, z) & 8u); };
          if (j < N && A(i, j) && B(i, j) && A(i, j - 1) && A(i + 1, j - 1) && B(i + 1, j - 1) && B(i + 1, j)) {
            cand = true;
            bad = bad || i < 2 || i > N - 3 || j < 4 || (j + 1) / 3 > in.cols - 2;
          }
        }
        uint32_t mine = 0u;
#pragma unroll
        for (int k = 0; k < 9; ++k) mine = lane == k ? bits[k] : mine;
        if (lane < 12) p[lane] = mine;
      }
      const uint32_t v = __ballot_sync(~0u, cand);
      if (lane == 0) sm[L.valid + i * W + x] = c ? sm[L.valid + i * W + x] | v : v;
    }
    __syncthreads();
    for (int k = tid; k < words; k += kThreads) bad = bad || bp_bytes_of(sm, L, in, c, k) != sm[L.stage + k];
    if (bad) cnt[2] = 1;
  }
  __syncthreads();
  if (cnt[2]) return false;
  for (int k = tid; k < N * W; k += kThreads) {
    const uint32_t v = sm[L.valid + k];
    if (!v) continue;
    const int i = k / W, x = k - i * W;
    sm[L.items + atomicAdd(&cnt[0], 1)] = (uint32_t)i << 16 | (uint32_t)x;
    for (int b = 0; b < 4; ++b)
      if ((v >> (8 * b)) & 255u) sm[L.units + atomicAdd(&cnt[1], 1)] = (uint32_t)i << 16 | (uint32_t)(4 * x + b);
  }
  __syncthreads();
  return true;
}

// Draws of half-sweep h into one set of moves: bit k of x (y) set where cell k, in state 3 or 25 (12 or 38), is in
// it (in the other) after the half-sweep.
struct BpUnit {
  uint32_t row, quad, to;  // to: byte offset in a set of moves
};
__device__ __forceinline__ BpUnit bp_unit(const uint32_t* sm, const BpLayout& L, int u, int units) {
  const uint32_t e = units ? sm[L.units + min(u, units - 1)] : 0u, byte = e & 0xffffu;
  BpUnit b;
  b.row = e >> 16;
  b.quad = 2 * byte + (threadIdx.x & 1);
  b.to = (b.row * (uint32_t)L.W + (byte >> 2)) * 8 + (byte & 3);
  return b;
}
__device__ __forceinline__ void bp_moves_of(const uint4& d, uint8_t* moves, const BpUnit& b, bool on, uint3 t) {
  auto nib = [](bool p, bool q, bool r, bool s) { return (p ? 1u : 0u) | (q ? 2u : 0u) | (r ? 4u : 0u) | (s ? 8u : 0u); };
  const uint32_t up = nib(d.x < t.x, d.y < t.x, d.z < t.x, d.w < t.x);
  const uint32_t dn = nib(d.x - t.y < t.z, d.y - t.y < t.z, d.z - t.y < t.z, d.w - t.y < t.z);
  const uint32_t mine = (up ^ 15u) | (dn << 16);
  const uint32_t pair = mine | (__shfl_down_sync(~0u, mine, 1) << 4);
  if (on && !(threadIdx.x & 1)) {
    moves[b.to] = (uint8_t)pair;
    moves[b.to + 4] = (uint8_t)(pair >> 16);
  }
}

// The steps [-look, 0) of an attempt: the first kBpUpdate threads update, the others draw, a period of
// L.period steps ahead, two steps' Philox blocks side by side; the update warps alone meet after every step.
// update(k, step, moves): the moves of one set applied to item k (a word of a chain); test(row, step): {width up,
// low down, width down}; stop() is asked (by every thread, after a barrier) every 256 steps.  False where it stopped.
template <int kThreads, int period, class Update, class Test, class Stop>
__device__ bool bp_steps_of(uint32_t* sm, const BpLayout& L, const DevInstance& in, int64_t look, int units, Update update,
                         Test test, Stop stop) {
  const int tid = threadIdx.x, lane = tid & 31;
  const int set = 2 * in.N * L.W;  // words of a set of moves
  constexpr int ask = 256 / period - 1;
  const int64_t periods = (look + period - 1) / period;
  const uint64_t seed = in.seed;
  const uint32_t stream = in.stream;
  const int u_warp = ((tid - kBpUpdate) >> 5) * 16, u0 = u_warp + (lane >> 1);
  const BpUnit unit0 = tid >= kBpUpdate ? bp_unit(sm, L, u0, units) : BpUnit{0, 0, 0};
  auto draw = [&](int64_t q) {
    uint8_t* const to = reinterpret_cast<uint8_t*>(sm + L.moves + (int)(q & 1) * period * set);
    for (int u = u_warp; u < units; u += (kThreads - kBpUpdate) / 2) {
      const BpUnit b = u == u_warp ? unit0 : bp_unit(sm, L, u + (lane >> 1), units);
      const bool on = u + (lane >> 1) < units;
#pragma unroll
      for (int r = 0; r < period; r += 2) {
        const int64_t h = -look + q * period + r;  // (draws of steps past the end are not used)
        const uint4 d0 = fast_quad(seed, stream, h, b.row, b.quad), d1 = fast_quad(seed, stream, h + 1, b.row, b.quad);
        bp_moves_of(d0, to + 4 * r * set, b, on, test(b.row, h));
        bp_moves_of(d1, to + 4 * (r + 1) * set, b, on, test(b.row, h + 1));
      }
    }
  };
  if (tid >= kBpUpdate) draw(0);
  __syncthreads();
  for (int64_t q = 0; q < periods; ++q) {
    if (tid < kBpUpdate) {
      const uint32_t* moves = sm + L.moves + (int)(q & 1) * period * set;
      const int len = (int)min((int64_t)period, look - q * period);
      for (int r = 0; r < len; ++r, moves += set) {
        update(-look + q * period + r, moves);
        asm volatile("bar.sync 1, %0;" ::"n"(kBpUpdate) : "memory");
      }
    } else if (q + 1 < periods) {
      draw(q + 1);
    }
    __syncthreads();
    if ((q & ask) == ask && stop()) return false;
  }
  return true;
}

template <int kThreads, class Update, class Test, class Stop>
__device__ __forceinline__ bool bp_steps(uint32_t* sm, const BpLayout& L, const DevInstance& in, int64_t look, int units,
                                         Update update, Test test, Stop stop) {
  return L.period == 8   ? bp_steps_of<kThreads, 8>(sm, L, in, look, units, update, test, stop)
         : L.period == 4 ? bp_steps_of<kThreads, 4>(sm, L, in, look, units, update, test, stop)
                         : bp_steps_of<kThreads, 2>(sm, L, in, look, units, update, test, stop);
}

// A loaded domino instance.
template <int kThreads, class Stop>
__device__ bool bp_domino(uint32_t* sm, const BpLayout& L, const DevInstance& in, int64_t look, int items, int units,
                          Stop stop) {
  const int tid = threadIdx.x, W = L.W, up_row = (W + 1) * kBpDominoWord;
  struct Item {
    int here, move;
    bool odd;
    uint32_t valid;
  };
  auto item = [&](int k) {
    const uint32_t e = k < 2 * items ? sm[L.items + (k >> 1)] : 1u << 16;
    const int i = (int)(e >> 16), x = (int)(e & 0xffffu);
    return Item{L.planes + (i * (W + 1) + x) * kBpDominoWord + 4 * (k & 1), 2 * (i * W + x), (i & 1) != 0,
                k < 2 * items ? sm[L.valid + i * W + x] : 0u};
  };
  auto apply = [&](const Item& it, int t, const uint32_t* moves) {
    uint32_t* const here = sm + it.here;
    uint32_t* const above = here - up_row;
    const uint2 move = *reinterpret_cast<const uint2*>(moves + it.move);
    const uint4 me = *reinterpret_cast<const uint4*>(here);
    const uint32_t U = above[1 - t], west = here[3 - kBpDominoWord];
    const bool aligned = it.odd == (t != 0);  // left HE, right HO of the same word
    const uint32_t D = t ? me.y : me.x;
    const uint32_t lft = aligned ? me.z : __funnelshift_l(west, me.w, 1), rgt = aligned ? me.w : me.z;
    // Flippable: up = down, left = right, up != left (states 3 and 12).
    const uint32_t flip = ~(U ^ D) & ~(lft ^ rgt) & (U ^ lft) & it.valid;
    const uint32_t T = flip & ((U & ~move.x) | (~U & move.y));
    if (T) {
      above[1 - t] = U ^ T;
      here[t] = D ^ T;
      here[2] = me.z ^ T;
      // HO: the word itself, or bit k - 1 of this word and bit 31 of the word to the left, whose other bits belong
      // to that word's cells.
      atomicXor(here + 3, aligned ? T : T >> 1);
      if (!aligned && (T & 1u)) atomicXor(here + 3 - kBpDominoWord, 0x80000000u);
    }
  };
  const Item item0 = item(tid < kBpUpdate ? tid : 2 * items), item1 = item(tid < kBpUpdate ? tid + kBpUpdate : 2 * items);
  return bp_steps<kThreads>(
      sm, L, in, look, units,
      [&](int64_t h, const uint32_t* moves) {
        const int t = (h & 1) ? 0 : 1;
        if (item0.valid) apply(item0, t, moves);
        if (item1.valid) apply(item1, t, moves);
        for (int k = tid + 2 * kBpUpdate; k < 2 * items; k += kBpUpdate) apply(item(k), t, moves);
      },
      [&](uint32_t row, int64_t h) {
        const int c = (int)(row & 1u) | ((h & 1) ? 0 : 2);
        return make_uint3(in.w_up[c], in.lo_dn[c], in.w_dn[c]);
      },
      stop);
}

template <int kThreads, class Stop>
__device__ bool bp_lozenge(uint32_t* sm, const BpLayout& L, const DevInstance& in, int64_t look, uint32_t c4, uint32_t c8,
                           int items, int units, Stop stop) {
  const int tid = threadIdx.x, W = L.W, left = kBpLozengeWord, dn_row = (W + 1) * kBpLozengeWord;
  struct Item {
    int here, move, q;
    uint32_t valid;
  };
  auto item = [&](int k) {
    const uint32_t e = k < 2 * items ? sm[L.items + (k >> 1)] : 0u;
    const int i = (int)(e >> 16), x = (int)(e & 0xffffu);
    return Item{L.planes + (i * (W + 1) + x) * kBpLozengeWord + 12 * (k & 1), 2 * (i * W + x), i % 3,
                k < 2 * items ? sm[L.valid + i * W + x] : 0u};
  };
  auto apply = [&](const Item& it, int r, const uint32_t* moves) {
    const int q = it.q + r >= 3 ? it.q + r - 3 : it.q + r, qw = q == 0 ? 2 : q - 1;
    uint32_t* const own = sm + it.here + q;
    uint32_t* const west = sm + it.here + qw;
    uint32_t* const south = own + dn_row + 6;
    uint32_t* const sw = west + dn_row + 3;
    const uint2 move = *reinterpret_cast<const uint2*>(moves + it.move);
    const uint32_t e = own[0], ne = own[3], n = own[6], s = south[0], w_l = west[-left], ws_l = sw[-left];
    uint32_t w = west[0], ws = sw[0];
    if (q == 0) {
      w = __funnelshift_l(w_l, w, 1);
      ws = __funnelshift_l(ws_l, ws, 1);
    }
    // Flippable: E, N, SW equal, NE, W, S their complement.
    const uint32_t flip = ~(n ^ e) & ~(n ^ ws) & (n ^ ne) & (n ^ w) & (n ^ s) & it.valid;
    const uint32_t T = flip & ((n & ~move.x) | (~n & move.y));
    if (T) {
      own[0] = e ^ T;
      own[3] = ne ^ T;
      own[6] = n ^ T;
      south[0] = s ^ T;
      // one slot to the left where the column to the west is in the slot before
      atomicXor(west, q == 0 ? T >> 1 : T);
      atomicXor(sw, q == 0 ? T >> 1 : T);
      if (q == 0 && (T & 1u)) {
        atomicXor(west - left, 0x80000000u);
        atomicXor(sw - left, 0x80000000u);
      }
    }
  };
  const Item item0 = item(tid < kBpUpdate ? tid : 2 * items), item1 = item(tid < kBpUpdate ? tid + kBpUpdate : 2 * items);
  int r = 0;  // the step's colour: look is a multiple of three
  return bp_steps<kThreads>(
      sm, L, in, look, units,
      [&](int64_t, const uint32_t* moves) {
        if (item0.valid) apply(item0, r, moves);
        if (item1.valid) apply(item1, r, moves);
        for (int k = tid + 2 * kBpUpdate; k < 2 * items; k += kBpUpdate) apply(item(k), r, moves);
        r = r == 2 ? 0 : r + 1;
      },
      [&](uint32_t, int64_t) { return make_uint3(c4, c4, c8 - c4); }, stop);
}

// Words in which the two chains differ, of this thread's share.
template <int kThreads>
__device__ uint32_t bp_differ(const uint32_t* sm, const BpLayout& L, const DevInstance& in) {
  const int pw = in.model == 0 ? kBpDominoWord : kBpLozengeWord, half = pw / 2;
  const int n = (L.valid - L.planes) / 2;
  uint32_t differ = 0;
  for (int k = threadIdx.x; k < n; k += kThreads) {
    const uint32_t* p = sm + L.planes + k / half * pw + k % half;
    differ += p[0] != p[half];
  }
  return differ;
}

}  // namespace rt
