// Six-vertex model: heat-bath sweep and coupling from the past on the height function.
//
// The reference has no six-vertex model; the definition is the library's own:
//   * n x n vertices, height points (y, x), 0 <= y, x <= n; h(below) - h(above) = +1 across a
//     horizontal edge whose arrow points right, h(right) - h(left) = +1 across a vertical
//     edge whose arrow points up;
//   * vertex types from the corner heights NW, NE, SW, SE: a (NE == SW, NW != SE), b (NW ==
//     SE, NE != SW), c (both equal), weights a, b, c;
//   * four point classes (x mod 2, y mod 2); sub-sweep s updates class s mod 4 by heat bath at
//     every interior point whose four edge neighbours share one height h': h' + 1 with
//     probability P(k1, k2), h' - 1 otherwise (k1, k2: diagonal points equal to h' + 1 on the
//     a/c and on the b/c diagonals), drawn as u < T[3 k1 + k2], u from 32 Philox bit planes.
//
// Layout in HBM.  Heights are kept mod 4; within a class the parity of x + y is fixed, so one
// bit per point is enough (sigma = ((h - parity) / 2) mod 2).  One chain = 4 class arrays,
// each R = n/2 + 1 rows of P 32-bit words; word 0 and the words past the data are zero guards,
// bit b of data word w is point k = 32 w + b of the class row (x = 2k + px, y = 2r + py).
// A thread owns one word: 32 points updated with bitwise logic, the random comparison done
// bit-sliced from the most significant plane down and stopped once every lane is decided.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "pdl.cuh"
#include "rng.cuh"
#include "rt_internal.h"

namespace rt {
namespace {

struct SvGeom {
  int n, R, P;           // side, rows per class, words per row (with guards)
  size_t class_words;    // R * P
  size_t chain_words;    // 4 * R * P
};

SvGeom sv_geom(int n) {
  SvGeom g;
  g.n = n;
  g.R = n / 2 + 1;
  g.P = (n / 2 + 1 + 31) / 32 + 2;
  g.class_words = (size_t)g.R * g.P;
  g.chain_words = 4 * g.class_words;
  return g;
}

struct SvLaunch {
  uint32_t* base;   // chain 0; chain c at base + c * chain_words
  size_t chain_words, class_words;
  int P, n;
  int px, py, r_lo, words, rows;  // the class being updated and its interior extent
  int k_lo, k_hi;
  uint32_t leaf[32][9];  // leaf[j][m]: all ones where bit j of threshold T[m] is set (sv_leaves)
  uint64_t seed;
  uint32_t stream;
  int64_t s;
};

// Per-plane leaf words of the nine heat-bath thresholds: leaf[j][m] is all ones where bit j
// of T[m] is set, so that a point's threshold bit in plane j is the OR over the nine
// vertex-weight classes m of (class mask & leaf[j][m]) - one three-input logic operation
// each, with the leaf a constant operand once the plane loop is unrolled.
inline void sv_leaves(const uint32_t* T, uint32_t (&leaf)[32][9]) {
  for (int j = 0; j < 32; ++j)
    for (int m = 0; m < 9; ++m) leaf[j][m] = ((T[m] >> j) & 1u) ? 0xffffffffu : 0u;
}

__device__ __forceinline__ uint32_t west_of(const uint32_t* row, int idx, int px) {
  return px ? row[idx] : __funnelshift_l(row[idx - 1], row[idx], 1);
}
__device__ __forceinline__ uint32_t east_of(const uint32_t* row, int idx, int px) {
  return px ? __funnelshift_r(row[idx], row[idx + 1], 1) : row[idx];
}

// The rows one word update reads and writes: the word's own row F (class px, py), the same
// row of class (1-px, py) (west/east neighbours), rows above/below of class (px, 1-py)
// (north/south) and of class (1-px, 1-py) (diagonals).
struct SvRows {
  uint32_t* F;
  const uint32_t *H, *Vn, *Vs, *Dn, *Ds;
};

// Planes 4 q .. 4 q + 3 (the most significant first) of the draws of word w of row r.
__device__ __forceinline__ uint4 sv_block(uint32_t w, uint32_t r, int q, uint32_t c2, uint32_t c3, uint64_t seed) {
  return philox4x32_10(make_uint4(w | ((uint32_t)q << 24), r, c2, c3), (uint32_t)seed, (uint32_t)(seed >> 32));
}

// Updates data word w (index idx = w + 1) of class row r.
__device__ __forceinline__ void sv_update_word(const SvRows& R, int idx, int px, int py, uint32_t imask, uint32_t w,
                                               uint32_t r, const uint32_t (&leaf)[32][9], uint64_t seed, uint32_t c2,
                                               uint32_t c3) {
  const uint32_t f = R.F[idx], wv = west_of(R.H, idx, px), ev = east_of(R.H, idx, px);
  const uint32_t flip = ~(wv ^ ev) & ~(wv ^ R.Vn[idx]) & ~(wv ^ R.Vs[idx]) & imask;
  if (!flip) return;
  const uint32_t sup = (px ^ py) ? wv : ~wv;  // sigma of h' + 1 (neighbour parity 1 - (px ^ py))
  const uint32_t e1a = ~(west_of(R.Dn, idx, px) ^ sup), e1b = ~(east_of(R.Ds, idx, px) ^ sup);
  const uint32_t e2a = ~(east_of(R.Dn, idx, px) ^ sup), e2b = ~(west_of(R.Ds, idx, px) ^ sup);
  const uint32_t a0 = ~(e1a | e1b), a1 = e1a ^ e1b, a2 = e1a & e1b;
  const uint32_t b0 = ~(e2a | e2b), b1 = e2a ^ e2b, b2 = e2a & e2b;
  const uint32_t mk[9] = {a0 & b0, a0 & b1, a0 & b2, a1 & b0, a1 & b1, a1 & b2, a2 & b0, a2 & b1, a2 & b2};
  uint32_t lt = 0, und = flip;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    if (!und) break;
    const uint4 Rq = sv_block(w, r, q, c2, c3, seed);
    const uint32_t planes[4] = {Rq.x, Rq.y, Rq.z, Rq.w};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int j = 31 - (4 * q + t);
      uint32_t Tj = 0;  // bit j of each point's threshold
#pragma unroll
      for (int m = 0; m < 9; ++m) Tj |= mk[m] & leaf[j][m];
      lt |= und & ~planes[t] & Tj;
      und &= ~(planes[t] ^ Tj);
    }
  }
  R.F[idx] = (f & ~flip) | (flip & ~(lt ^ sup));
}

__device__ __forceinline__ uint32_t interior_mask(int w, int k_lo, int k_hi) {
  const int k0 = 32 * w;
  const int lo = max(k_lo - k0, 0), hi = min(k_hi - k0, 31);
  if (hi < lo) return 0u;
  return (hi - lo == 31 ? 0xffffffffu : ((1u << (hi - lo + 1)) - 1u)) << lo;
}

// One sub-sweep of one class over global memory; blockIdx.y is the chain.
__global__ void __launch_bounds__(128) k_sv_sub(SvLaunch L) {
  pdl_begin();
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= L.words * L.rows) return;
  const int w = g % L.words, r = L.r_lo + g / L.words;
  const int px = L.px, py = L.py, cls = px | (py << 1);
  const uint32_t imask = interior_mask(w, L.k_lo, L.k_hi);
  if (!imask) return;
  uint32_t* chain = L.base + (size_t)blockIdx.y * L.chain_words;
  const uint32_t* V = chain + (size_t)(cls ^ 2) * L.class_words;
  const uint32_t* D = chain + (size_t)(cls ^ 3) * L.class_words;
  const int rn = py ? r : r - 1, rs = py ? r + 1 : r;
  const SvRows rows = {chain + (size_t)cls * L.class_words + (size_t)r * L.P,
                           chain + (size_t)(cls ^ 1) * L.class_words + (size_t)r * L.P, V + (size_t)rn * L.P,
                           V + (size_t)rs * L.P, D + (size_t)rn * L.P, D + (size_t)rs * L.P};
  const uint32_t c2 = (uint32_t)(uint64_t)L.s, c3 = ((uint32_t)((uint64_t)L.s >> 32) & 0xffffu) | (L.stream << 16);
  sv_update_word(rows, w + 1, px, py, imask, (uint32_t)w, (uint32_t)r, L.leaf, L.seed, c2, c3);
}

// Resident engine: the chains in shared memory, a band of class rows per CTA.
//
// Bound: latency.  With one word a thread and a cluster barrier per sub-sweep a word took about 800 dependent
// instructions (Philox, then planes against nine thresholds): n = 512 6.2 us per sweep (four sub-sweeps),
// n = 48 with two chains 2.2 us.  Here
//   * draw warps compute, phases ahead, what does not depend on the state: for every word the
//     bits [u < T] of each distinct threshold T (nine; five where T depends on k1 + k2 only, as
//     for a = b).  16 planes are compared at once, least significant first (one logic operation
//     per plane and threshold for "less", one for "equal"); words with an undecided point, one
//     warp in eight, look at more.  The update warps then select among the words: about 50
//     operations a word;
//   * a phase is the two sub-sweeps of one row parity.  They read rows of the other parity and
//     their own row, so bands meet at most twice a sweep; a band also updates `depth` rows beyond
//     its own on both sides, whose draws it makes itself, and meets its neighbours every `depth`
//     sweeps only (rows as 64-bit words tagged with the period, through L2; every wait bounded).
// Measured (GB300, a = b): n = 512 1.10 us per sweep, n = 101 0.86, n = 1024 1.84 (before, one launch per
// sub-sweep: 8.3), n = 48 with two chains 0.80.  A warp's draws cost about 600 cycles of a scheduler in
// Philox (the high halves of its products) and 360 (five thresholds) or 630 (nine) in the comparison; a
// band's update alone takes about 0.65 us per sweep, an exchange 0.3-0.5 us.
struct SvBandArgs {
  const uint32_t* src;  // chain 0, chain c at + c * chain_words
  uint32_t* dst;        // not src: a band may write back before another has loaded
  size_t chain_words, class_words;
  int P, n, R, words;   // words: data words of a row that can change
  int bands, depth;     // sweeps between exchanges (each band owns at least depth rows)
  int group;            // update threads per chain, a word each (a multiple of 32)
  int batch;            // phases drawn at once
  int items;            // most words of one sub-sweep in a band (a multiple of 4)
  int rows;             // most rows of a band's window
  uint32_t leaf[32][9];  // as SvLaunch::leaf; of the distinct thresholds only, in the order they are drawn
  uint64_t seed;
  uint32_t stream;
  int64_t s0;           // first sub-sweep, a multiple of 4
  int sweeps;
  uint64_t* xbuf;       // [period parity][band][to above, to below][chain][row][class][word], tags cleared
  int* error;
  long max_spin;
  int silent_plus1;     // test hook: this band, less one, publishes nothing
  // Coupling from the past (couple, two chains): blockIdx.y = k runs attempt attempt0 + k, sub-sweeps
  // [-4 first << attempt, 0), into the k-th pair of chains at dst, and leaves once a smaller one has coalesced.
  int couple, attempt0;
  int64_t first;
  size_t xteam;         // words of xbuf a team
  int* best;            // smallest attempt that coalesced
  int2* team;           // [k] {bands whose chains differ, bands done}
};

constexpr int kSvTeams = 4;  // attempts side by side
constexpr int kSvDrawPlanes = 16;
constexpr int kSvBandThreads = 640;

// First row of band b of `bands` over the rows that can change.
__host__ __device__ __forceinline__ int sv_band_row(int b, int bands, int rows) { return (int)((int64_t)b * rows / bands); }

// Rows [lo, hi) that a band owning [r0, r1) updates in a phase of row parity py, `left` sweeps
// before its next exchange (this one included).
__host__ __device__ __forceinline__ void sv_phase_rows(int n, int r0, int r1, int py, int left, int* lo, int* hi) {
  *lo = max(py ? 0 : 1, r0 - (left - 1));
  *hi = min(py ? (n - 2) / 2 + 1 : (n - 1) / 2 + 1, py ? r1 + left - 1 : r1 + left);
  if (*hi < *lo) *hi = *lo;
}

// One plane of the bit-sliced comparison, from the least significant up: less = T ? ~p | less : ~p & less
// and equal &= ~(p ^ T), one operation each (the compiler makes two of the first).
__device__ __forceinline__ uint32_t sv_less(uint32_t less, uint32_t p, uint32_t T) {
  uint32_t d;
  constexpr int a = 0xf0, b = 0xcc, c = 0xaa;
  asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(d) : "r"(T), "r"(p), "r"(less), "n"(((a & (~b | c)) | (~a & ~b & c)) & 0xff));
  return d;
}
__device__ __forceinline__ uint32_t sv_equal(uint32_t equal, uint32_t p, uint32_t T) {
  uint32_t d;
  constexpr int a = 0xf0, b = 0xcc, c = 0xaa;
  asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(d) : "r"(T), "r"(p), "r"(equal), "n"((c & ~(a ^ b)) & 0xff));
  return d;
}

// Bits [u < T[m]] of the 32 points of word w of row r in one sub-sweep, for M thresholds.
template <int M>
__device__ __forceinline__ void sv_draw_word(uint32_t* set, int item, int items, const uint32_t (&leaf)[32][9], uint32_t imask,
                                             uint32_t w, uint32_t r, uint32_t c2, uint32_t c3, uint64_t seed) {
  uint32_t planes[kSvDrawPlanes];
#pragma unroll
  for (int q = 0; q < kSvDrawPlanes / 4; ++q) {
    const uint4 b = sv_block(w, r, q, c2, c3, seed);
    planes[4 * q] = b.x, planes[4 * q + 1] = b.y, planes[4 * q + 2] = b.z, planes[4 * q + 3] = b.w;
  }
  uint32_t lt[M], eq[M], open = 0;
#pragma unroll
  for (int m = 0; m < M; ++m) lt[m] = 0u, eq[m] = imask;
#pragma unroll
  for (int t = kSvDrawPlanes - 1; t >= 0; --t)
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const uint32_t T = leaf[31 - t][m];
      lt[m] = sv_less(lt[m], planes[t], T);
      eq[m] = sv_equal(eq[m], planes[t], T);
    }
#pragma unroll
  for (int m = 0; m < M; ++m) open |= eq[m];
  for (int q = kSvDrawPlanes / 4; open && q < 8; ++q) {
    const uint4 b = sv_block(w, r, q, c2, c3, seed);
    const uint32_t more[4] = {b.x, b.y, b.z, b.w};
    open = 0;
#pragma unroll
    for (int m = 0; m < M; ++m) {
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const uint32_t T = leaf[31 - 4 * q - t][m];
        lt[m] |= eq[m] & ~more[t] & T;
        eq[m] &= ~(more[t] ^ T);
      }
      open |= eq[m];
    }
  }
#pragma unroll
  for (int m = 0; m < M; ++m) set[m * items + item] = lt[m];
}

// The drawn bit of each point's threshold, from the bits of its diagonal points that equal h' + 1: e1a,
// e1b on the a/c diagonal, e2a, e2b on the b/c diagonal.  kSum: T depends on k1 + k2 only.
template <bool kSum>
__device__ __forceinline__ uint32_t sv_pick(const uint32_t (&drawn)[kSum ? 5 : 9], uint32_t e1a, uint32_t e1b,
                                            uint32_t e2a, uint32_t e2b) {
  if constexpr (kSum) {
    const uint32_t x = e1a ^ e1b ^ e2a, y = (e1a & e1b) | (e2a & (e1a | e1b));  // e1a + e1b + e2a
    const uint32_t one = x ^ e2b, z = x & e2b, two = y ^ z, four = y & z;
    const uint32_t l01 = (one & drawn[1]) | (~one & drawn[0]), l23 = (one & drawn[3]) | (~one & drawn[2]);
    const uint32_t low = (two & l23) | (~two & l01);
    return (four & drawn[4]) | (~four & low);
  } else {
    const uint32_t a1 = e1a ^ e1b, a2 = e1a & e1b, b1 = e2a ^ e2b, b2 = e2a & e2b;
    uint32_t k[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const uint32_t low = (b1 & drawn[3 * i + 1]) | (~b1 & drawn[3 * i]);
      k[i] = (b2 & drawn[3 * i + 2]) | (~b2 & low);
    }
    const uint32_t low = (a1 & k[1]) | (~a1 & k[0]);
    return (a2 & k[2]) | (~a2 & low);
  }
}

__device__ __forceinline__ int sv_div(int a, float inv) { return (int)(((float)a + 0.5f) * inv); }  // a < 2^20

template <int NCH, bool kSum>
__global__ void __launch_bounds__(kSvBandThreads, 1) k_sv_bands(const __grid_constant__ SvBandArgs A) {
  constexpr int M = kSum ? 5 : 9;
  // [NCH][4][rows][P] states; [2][batch][2][M][items] drawn bits; [depth + 1][2] rows of a phase
  extern __shared__ __align__(16) uint32_t sm[];
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const int n = A.n, P = A.P, words = A.words, band = blockIdx.x;
  const int movable = (n - 1) / 2 + 1;  // rows that can change
  __shared__ int s_stop[2];  // a smaller attempt coalesced, by parity of the batch
  const bool couple = NCH == 2 && A.couple;
  const int team = couple ? (int)blockIdx.y : 0, attempt = A.attempt0 + team;
  const int all_sweeps = couple ? (int)(A.first << attempt) : A.sweeps;
  const int64_t s0 = couple ? -4 * (int64_t)all_sweeps : A.s0;
  uint64_t* const xbuf = A.xbuf + team * A.xteam;
  const int r0 = sv_band_row(band, A.bands, movable), r1 = sv_band_row(band + 1, A.bands, movable);
  const int w0 = max(r0 - A.depth, 0), w1 = min(r1 + A.depth, A.R);  // the window's rows
  const int cs = A.rows * P;
  uint32_t* const drawn = sm + ((NCH * 4 * cs + 3) & ~3);
  const int sub_words = M * A.items, set_words = A.batch * 2 * sub_words;
  int2* const phase_tab = reinterpret_cast<int2*>(drawn + 2 * set_words);  // [sweeps left][py]: first row, words
  const float inv_words = 1.0f / (float)words;

  for (int i = tid; i < NCH * 4 * (w1 - w0) * P; i += nt) {
    const int p = i % P, lr = (i / P) % (w1 - w0), cc = i / (P * (w1 - w0));  // cc: chain * 4 + class
    sm[cc * cs + lr * P + p] =
        A.src[(size_t)(cc >> 2) * A.chain_words + (size_t)(cc & 3) * A.class_words + (size_t)(w0 + lr) * P + p];
  }

  for (int i = tid; i < 2 * (A.depth + 1); i += nt) {
    int lo, hi;
    sv_phase_rows(n, r0, r1, i & 1, i >> 1, &lo, &hi);
    phase_tab[i] = make_int2(lo, (hi - lo) * words);
  }
  __syncthreads();

  const int updaters = NCH * A.group;
  const bool updates = tid < updaters;
  const int phases = 2 * all_sweeps, batches = (phases + A.batch - 1) / A.batch;
  // Draws of batch b: tasks of 32 words in turn over the draw warps.
  int ahead = 0, drawn_left = min(A.depth, all_sweeps);  // the sweep reached, and sweeps left before the exchange after it
  int2 rows_of[2] = {phase_tab[2 * drawn_left], phase_tab[2 * drawn_left + 1]};
  auto draw_batch = [&](int b) {
    const int dw = warp - (updaters >> 5), ndw = (nt - updaters) >> 5;
    uint32_t* const set = drawn + (b & 1) * set_words;
    int turn = 0;
    for (int q = 0; q < A.batch; ++q) {
      const int f = b * A.batch + q;
      if (f >= phases) break;
      const int py = f & 1;
      const int lo = py ? rows_of[1].x : rows_of[0].x, items = py ? rows_of[1].y : rows_of[0].y;
      if (py && A.depth > 1) {
        ++ahead;
        drawn_left = drawn_left > 1 ? drawn_left - 1 : min(A.depth, all_sweeps - ahead);
        rows_of[0] = phase_tab[2 * drawn_left], rows_of[1] = phase_tab[2 * drawn_left + 1];
      }
      for (int e0 = 0; e0 < 2 * items; e0 += 32, turn = turn + 1 == ndw ? 0 : turn + 1) {
        if (turn != dw) continue;
        const int e = e0 + lane;
        if (e >= 2 * items) continue;
        const int px = e >= items ? 1 : 0, it = e - px * items, rr = sv_div(it, inv_words), w = it - rr * words;
        const uint64_t s = (uint64_t)(s0 + 2 * (int64_t)f + px);
        const uint32_t imask = interior_mask(w, px ? 0 : 1, (n - 1 - px) / 2);
        sv_draw_word<M>(set + (2 * q + px) * sub_words, it, A.items, A.leaf, imask, (uint32_t)w, (uint32_t)(lo + rr),
                        (uint32_t)s, ((uint32_t)(s >> 32) & 0xffffu) | (A.stream << 16), A.seed);
      }
    }
  };

  const int chain = NCH == 2 && tid >= A.group ? 1 : 0, ut = tid - chain * A.group;
  uint32_t* const S = sm + chain * 4 * cs;
  auto group_sync = [&](int group) {
    if (group == 32)
      __syncwarp();
    else
      asm volatile("bar.sync %0, %1;" ::"r"(1 + chain), "r"(group) : "memory");
  };
  const int my_row = sv_div(ut, inv_words), my_word = ut - my_row * words;
  const uint32_t my_mask[2] = {interior_mask(my_word, 1, (n - 1) / 2), interior_mask(my_word, 0, (n - 2) / 2)};
  bool dead = false;  // a wait gave up: no further waits, the launch runs to its end
  // Exchange: what each thread sends (its word, of the last sweep before an exchange) and receives (up to
  // four words) is the same every period; -1: nothing.
  const int per_side = A.depth * 4 * words;
  const uint32_t xparity = (uint32_t)(A.bands * 2 * NCH * per_side);
  auto slot = [&](int b, int dir) { return ((b * 2 + dir) * NCH + chain) * per_side; };
  int send_up[2] = {-1, -1}, send_dn[2] = {-1, -1}, recv_from[4], recv_to[4];
#pragma unroll
  for (int py = 0; py < 2; ++py) {
    const int2 ph = phase_tab[2 + py];
    const int row = ph.x + my_row;
    if (!updates || ut >= ph.y || row < r0 || row >= r1 || band + 1 == A.silent_plus1) continue;
    if (band > 0 && row < r0 + A.depth) send_up[py] = slot(band, 0) + ((row - r0) * 4 + 2 * py) * words + my_word;
    if (band + 1 < A.bands && row >= r1 - A.depth)
      send_dn[py] = slot(band, 1) + ((row - (r1 - A.depth)) * 4 + 2 * py) * words + my_word;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int e = ut + i * A.group;
    const int dir = e >= per_side ? 1 : 0, x = e - dir * per_side, q = sv_div(x, inv_words), w = x - q * words;
    const int row = (dir ? r1 : r0 - A.depth) + (q >> 2), py = (q >> 1) & 1;  // the neighbours' rows next to ours
    const bool on = updates && e < 2 * per_side && (dir ? band + 1 < A.bands : band > 0) && row >= (py ? 0 : 1) &&
                    row <= (n - 1 - py) / 2;
    recv_from[i] = on ? slot(dir ? band + 1 : band - 1, 1 - dir) + x : -1;
    recv_to[i] = (q & 3) * cs + (row - w0) * P + 1 + w;
  }
  auto send = [&](uint32_t per, int at, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(xbuf + (per & 1) * xparity + at),
                 "l"(((uint64_t)(per + 1) << 32) | v)
                 : "memory");
  };
  auto receive = [&](uint32_t per) {
    const uint64_t* const buf = xbuf + (per & 1) * xparity;
    uint64_t v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (recv_from[i] >= 0) asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v[i]) : "l"(buf + recv_from[i]) : "memory");
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (recv_from[i] < 0) continue;
      for (long it = 0; !dead && (uint32_t)(v[i] >> 32) != per + 1; ++it) {
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v[i]) : "l"(buf + recv_from[i]) : "memory");
        if (it >= A.max_spin) {
          dead = true;
          atomicExch(A.error, 1);
        } else if ((it & 255) == 255 && (*static_cast<volatile int*>(A.error) ||
                                         (couple && *static_cast<volatile int*>(A.best) < attempt))) {
          dead = true;
        }
      }
      if (!dead) S[recv_to[i]] = (uint32_t)v[i];
    }
    group_sync(A.group);
  };

  if (!updates) draw_batch(0);
  __syncthreads();
  // Held in registers: a parameter read again in each phase is a constant load on its critical path.
  int depth = A.depth, sweeps = all_sweeps, items = A.items, group = A.group, row_words = P, class_words = cs;
  asm volatile("" : "+r"(depth), "+r"(sweeps), "+r"(items), "+r"(group), "+r"(row_words), "+r"(class_words));
  int in_period = 0;  // sweeps since the last exchange
  uint32_t period = 0;
  int2 ph = phase_tab[2 * min(A.depth, all_sweeps)];  // the phase's first row and its words
  for (int b = 0; b < batches; ++b) {
    if (updates) {
      const uint32_t* bits = drawn + (b & 1) * set_words;
      const int last = min(phases - b * A.batch, A.batch);
      for (int q = 0; q < last; ++q) {
        const int f = b * A.batch + q, py = f & 1;
        const int left = min(depth - in_period, sweeps - (f >> 1));
        // Classes: a, b = (0, py), (1, py), which move; c, d = (0, 1 - py), (1, 1 - py), which do not.  Sub-sweep
        // px = 0 reads points k - 1, k of b and d and k of c; px = 1 points k, k + 1 of a and c and k of d:
        // one set of loads serves both, but for the word of a to the right.
        const bool mine = ut < ph.y;
        const int flip_side = py ? 0 : ~0;  // sigma of h' + 1 is h at odd x + y, ~h at even
        const int at = mine ? (ph.x - w0 + my_row) * row_words + 1 + my_word : row_words + 1;
        uint32_t* const pa = S + 2 * py * class_words + at;
        const uint32_t* const pc = S + 2 * (1 - py) * class_words + at - (py ? 0 : row_words);
        const uint32_t va = pa[0], vb = pa[class_words], vb_w = pa[class_words - 1];
        const uint32_t c_n = pc[0], c_s = pc[row_words], c_ne = pc[1], c_se = pc[row_words + 1];
        const uint32_t d_n = pc[class_words], d_s = pc[class_words + row_words], d_nw = pc[class_words - 1], d_sw = pc[class_words + row_words - 1];
        uint32_t drawn0[M], drawn1[M];
#pragma unroll
        for (int m = 0; m < M; ++m) drawn0[m] = bits[m * items + ut], drawn1[m] = bits[sub_words + m * items + ut];
        bits += 2 * sub_words;
        uint32_t now;
        {
          const uint32_t hw = __funnelshift_l(vb_w, vb, 1);
          const uint32_t flip = ~(vb ^ hw) & ~(vb ^ c_n) & ~(vb ^ c_s) & (mine ? my_mask[0] : 0u);
          const uint32_t sup = vb ^ flip_side;
          const uint32_t lt = sv_pick<kSum>(drawn0, ~(__funnelshift_l(d_nw, d_n, 1) ^ sup), ~(d_s ^ sup), ~(d_n ^ sup),
                                            ~(__funnelshift_l(d_sw, d_s, 1) ^ sup));
          now = (va & ~flip) | (flip & ~(lt ^ sup));
          if (mine) pa[0] = now;
        }
        const int next_left = py ? (left > 1 ? left - 1 : min(depth, sweeps - (f >> 1) - 1)) : left;
        ph = phase_tab[2 * next_left + 1 - py];
        group_sync(group);
        {
          const uint32_t sup = now ^ ~flip_side;
          const uint32_t lt = sv_pick<kSum>(drawn1, ~(c_n ^ sup), ~(__funnelshift_r(c_s, c_se, 1) ^ sup),
                                            ~(__funnelshift_r(c_n, c_ne, 1) ^ sup), ~(c_s ^ sup));
          const uint32_t he = __funnelshift_r(now, pa[1], 1);
          const uint32_t flip = ~(now ^ he) & ~(now ^ d_n) & ~(now ^ d_s) & (mine ? my_mask[1] : 0u);
          const uint32_t moved = (vb & ~flip) | (flip & ~(lt ^ sup));
          if (mine) pa[class_words] = moved;
          // The last sweep before an exchange leaves the boundary rows as the neighbours need them.
          if (left == 1 && A.bands > 1) {
            const int up = py ? send_up[1] : send_up[0], dn = py ? send_dn[1] : send_dn[0];
            if (up >= 0) {
              send(period, up, now);
              send(period, up + words, moved);
            }
            if (dn >= 0) {
              send(period, dn, now);
              send(period, dn + words, moved);
            }
          }
        }
        group_sync(group);
        if (py && ++in_period == depth) {
          in_period = 0;
          if (A.bands > 1 && (f >> 1) + 1 < sweeps) receive(period++);
        }
      }
    } else {
      if (couple && tid == updaters) s_stop[b & 1] = *static_cast<volatile int*>(A.best) < attempt;
      if (b + 1 < batches) draw_batch(b + 1);
    }
    __syncthreads();
    if (couple && *static_cast<volatile int*>(&s_stop[b & 1])) return;
  }
  if (couple) {  // the last band to finish knows whether any differs
    const int mine = (band + 1 == A.bands ? A.R : r1) - r0;
    bool differ = false;
    for (int i = tid; i < 4 * mine * P; i += nt) {
      const int at = (i / (mine * P)) * cs + (r0 - w0) * P + i % (mine * P);
      differ = differ || sm[at] != sm[4 * cs + at];
    }
    const int any = __syncthreads_or(differ || dead ? 1 : 0);
    if (tid == 0) {
      if (any) atomicAdd(&A.team[team].x, 1);
      __threadfence();
      if (atomicAdd(&A.team[team].y, 1) == A.bands - 1 && atomicAdd(&A.team[team].x, 0) == 0) atomicMin(A.best, attempt);
    }
  }
  const int own = (band + 1 == A.bands ? A.R : r1) - r0;  // the last row may be fixed: the last band's
  for (int i = tid; i < NCH * 4 * own * P; i += nt) {
    const int p = i % P, lr = (i / P) % own, cc = i / (P * own);
    A.dst[(size_t)(2 * team + (cc >> 2)) * A.chain_words + (size_t)(cc & 3) * A.class_words + (size_t)(r0 + lr) * P + p] =
        sm[cc * cs + (r0 - w0 + lr) * P + p];
  }
}

// OR of (top ^ bottom) over all words of the two chains.
__global__ void k_sv_diff(const uint32_t* a, const uint32_t* b, size_t words, uint32_t* flag) {
  uint32_t acc = 0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (size_t)gridDim.x * blockDim.x)
    acc |= a[i] ^ b[i];
  acc = __reduce_or_sync(0xffffffffu, acc);
  if ((threadIdx.x & 31) == 0 && acc) atomicOr(flag, 1u);
}

// Heights (n + 1) x (n + 1) to one chain's class words, a warp per row and 64 columns; *bad is set where
// two neighbours do not differ by one.
__global__ void __launch_bounds__(256) k_sv_pack(const int32_t* h, uint32_t* chain, SvGeom G, int* bad) {
  const int lane = threadIdx.x & 31, n = G.n, L = n + 1, words = G.P - 2;
  const int it = blockIdx.x * 8 + (int)(threadIdx.x >> 5);
  if (it >= L * words) return;
  const int y = it / words, w = it - y * words, o = __ldg(h) & 1;
  bool wrong = false;
#pragma unroll
  for (int px = 0; px < 2; ++px) {
    const int x = 2 * (32 * w + lane) + px;
    uint32_t sigma = 0;
    if (x <= n) {
      const int v = h[(size_t)y * L + x];
      wrong = wrong || (x < n && abs(h[(size_t)y * L + x + 1] - v) != 1) || (y < n && abs(h[(size_t)(y + 1) * L + x] - v) != 1);
      sigma = (uint32_t)((v - o - ((x + y) & 1)) >> 1) & 1u;
    }
    const uint32_t bits = __ballot_sync(~0u, sigma);
    if (lane == 0) chain[(size_t)(px | ((y & 1) << 1)) * G.class_words + (size_t)(y >> 1) * G.P + 1 + w] = bits;
  }
  if (__any_sync(~0u, wrong) && lane == 0) *bad = 1;
}

// The heights of a chain's class words, a warp per row: along a row the height moves by the step of
// +-1 between two residues mod 4, from the left column, which never moves (h holds the start heights).
__global__ void __launch_bounds__(256) k_sv_unpack(const uint32_t* chain, SvGeom G, int32_t* h) {
  const int lane = threadIdx.x & 31, n = G.n, L = n + 1, y = blockIdx.x * 8 + (int)(threadIdx.x >> 5);
  if (y > n) return;
  const uint32_t* const even = chain + (size_t)((y & 1) << 1) * G.class_words + (size_t)(y >> 1) * G.P + 1;
  const uint32_t* const odd = even + G.class_words;
  auto residue = [&](int x) -> int {  // without the start's parity, which both ends of a step share
    const int k = x >> 1;
    return ((x + y) & 1) + 2 * (int)(((x & 1 ? odd : even)[k >> 5] >> (k & 31)) & 1u);
  };
  int base = h[(size_t)y * L];
  for (int x0 = 1; x0 <= n; x0 += 32) {
    const int x = x0 + lane;
    const uint32_t ups = __ballot_sync(~0u, x <= n && ((residue(min(x, n)) - residue(min(x, n) - 1)) & 3) == 1);
    if (x <= n) h[(size_t)y * L + x] = base + 2 * __popc(ups & (0xffffffffu >> (31 - lane))) - (lane + 1);
    base += 2 * __popc(ups) - 32;
  }
}

void fill_launch(SvLaunch& L, const SvGeom& G, int64_t s) {
  L.px = (int)(s & 1);
  L.py = (int)((s >> 1) & 1);
  L.s = s;
  const int n = G.n;
  L.r_lo = L.py ? 0 : 1;
  const int r_hi = (n - 1 - L.py) / 2;
  L.rows = r_hi - L.r_lo + 1;
  L.k_lo = L.px ? 0 : 1;
  L.k_hi = (n - 1 - L.px) / 2;
  L.words = L.k_hi / 32 + 1;
}

}  // namespace

// ---- host side ------------------------------------------------------------------------

std::vector<uint32_t> sv_thresholds_host(double a, double b, double c) {
  std::vector<uint32_t> T(9);
  for (int k1 = 0; k1 < 3; ++k1)
    for (int k2 = 0; k2 < 3; ++k2) {
      double wp = 1.0, wm = 1.0;
      for (int i = 0; i < 2; ++i) wp *= i < k1 ? c : a, wm *= i < 2 - k1 ? c : a;
      for (int i = 0; i < 2; ++i) wp *= i < k2 ? c : b, wm *= i < 2 - k2 ? c : b;
      const double scaled = std::floor(wp / (wp + wm) * 4294967296.0);
      T[3 * k1 + k2] = scaled >= 4294967295.0 ? 0xffffffffu : (uint32_t)scaled;
    }
  return T;
}

// Checks |dh| = 1 across every edge; returns false otherwise.
bool sv_valid_heights(const int32_t* h, int n) {
  const int L = n + 1;
  for (int y = 0; y <= n; ++y)
    for (int x = 0; x <= n; ++x) {
      const int v = h[(size_t)y * L + x];
      if (x < n && std::abs(h[(size_t)y * L + x + 1] - v) != 1) return false;
      if (y < n && std::abs(h[(size_t)(y + 1) * L + x] - v) != 1) return false;
    }
  return true;
}

void sv_pack(const int32_t* h, const SvGeom& G, uint32_t* out) {
  const int n = G.n, L = n + 1, o = h[0] & 1;
  std::fill(out, out + G.chain_words, 0u);
  for (int y = 0; y <= n; ++y)
    for (int x = 0; x <= n; ++x) {
      const int v = h[(size_t)y * L + x] - o, p = (x + y) & 1;
      const uint32_t sigma = (uint32_t)(((v - p) >> 1) & 1);
      const int cls = (x & 1) | ((y & 1) << 1), r = y >> 1, k = x >> 1;
      out[(size_t)cls * G.class_words + (size_t)r * G.P + 1 + (k >> 5)] |= sigma << (k & 31);
    }
}

// Heights from the bits, anchored on the left column of the start heights (the boundary is
// never updated): along each row h moves by the step of +-1 that lands on the stored residue.
void sv_unpack(const uint32_t* bits, const SvGeom& G, const int32_t* start, int32_t* out) {
  const int n = G.n, L = n + 1, o = start[0] & 1;
  for (int y = 0; y <= n; ++y) {
    int prev = start[(size_t)y * L];
    out[(size_t)y * L] = prev;
    for (int x = 1; x <= n; ++x) {
      const int cls = (x & 1) | ((y & 1) << 1), r = y >> 1, k = x >> 1;
      const uint32_t sigma = (bits[(size_t)cls * G.class_words + (size_t)r * G.P + 1 + (k >> 5)] >> (k & 31)) & 1u;
      const int residue = (((x + y) & 1) + 2 * (int)sigma + o) & 3;
      const int up = prev + 1;
      prev = ((up & 3) == residue) ? up : prev - 1;
      out[(size_t)y * L + x] = prev;
    }
  }
}

namespace {

struct SvDevice {
  uint32_t* chains = nullptr;  // the state of the per-sub-sweep kernels; the resident engine's start
  uint32_t* other = nullptr;   // resident engine: two more states, written in turn, or one of each attempt side by side
  uint64_t* xbuf = nullptr;
  int32_t* heights = nullptr;
  int* flag = nullptr;  // {chains differ or heights not valid, a wait gave up, SvBandArgs::best, unused, SvBandArgs::team}
  cudaStream_t stream = nullptr;
  ~SvDevice() {
    for (void* p : {(void*)chains, (void*)other, (void*)xbuf, (void*)heights, (void*)flag}) dev_free(p, stream);
  }
};

rt_status sv_check_common(int32_t n, const double* abc, double* a, double* b, double* c) {
  if (n < 2 || n > 65534) return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex: n must be in [2, 65534]");
  *a = abc ? abc[0] : 1.0;
  *b = abc ? abc[1] : 1.0;
  *c = abc ? abc[2] : 1.0;
  for (double v : {*a, *b, *c})
    if (!(v > 0.0) || !std::isfinite(v)) return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex: weights must be finite and > 0");
  return RT_OK;
}

rt_status sv_check_device() {
  int devs = 0;
  if (cudaGetDeviceCount(&devs) != cudaSuccess || devs == 0) {
    cudaGetLastError();
    return fail(RT_ERR_CUDA, "no CUDA device: the sweep has no CPU fallback");
  }
  return RT_OK;
}

struct SvBandPlan {
  bool ok = false;
  bool sum = false;  // thresholds depend on k1 + k2 only
  int bands = 0, depth = 0, group = 0, batch = 0, items = 0, rows = 0, threads = 0, sms = 0;
  size_t smem = 0, xbuf_words = 0;
  void* kernel = nullptr;
};

bool sv_sum_thresholds(const std::vector<uint32_t>& T) {
  return T[1] == T[3] && T[2] == T[4] && T[4] == T[6] && T[5] == T[7];
}

SvBandPlan sv_band_plan(const SvGeom& G, int chains, const std::vector<uint32_t>& T) {
  SvBandPlan p;
  const int n = G.n, movable = (n - 1) / 2 + 1, words = (n - 1) / 2 / 32 + 1;
  int dev = 0, sms = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess) {
    cudaGetLastError();
    return p;
  }
  p.sms = sms;
  p.sum = sv_sum_thresholds(T);
  const int M = p.sum ? 5 : 9;
  // One band where half a warp holds a sub-sweep (n = 30: 0.84 us a sweep, two bands 0.95-1.0; n = 40: 1.08 and
  // 0.88).  Else bands of `depth` rows, so that a band's words with its 2 depth - 1 spare rows fill one or two
  // warps: depth 4, 3, 2 at 2, 3, 4 or more words a row (n = 101: depth 3 and 4 0.86-0.88 us, 2 0.96; n = 190: 3
  // 1.16, 4 1.23; n = 256: 2 1.10, 3 1.23; n = 512: 2 1.10, 1 1.50); depth 1 once every band has more than two
  // rows (n = 600: depth 2 1.23, 1 1.83; n = 700: 2.03 and 1.96; n = 1024: 2.5 and 1.9).
  p.depth = words <= 2 ? 4 : words == 3 ? 3 : movable <= 2 * sms ? 2 : 1;
  p.bands = std::min(sms, movable / p.depth);
  if (movable * words <= 16 || p.bands < 2) p.bands = 1, p.depth = 1;
  int most = 0;
  for (int b = 0; b < p.bands; ++b) {
    const int r0 = sv_band_row(b, p.bands, movable), r1 = sv_band_row(b + 1, p.bands, movable);
    if (p.bands > 1 && r1 - r0 < p.depth) return p;
    int lo, hi;
    for (int py = 0; py < 2; ++py) {
      sv_phase_rows(n, r0, r1, py, p.depth, &lo, &hi);
      most = std::max(most, hi - lo);
    }
    p.rows = std::max(p.rows, std::min(r1 + p.depth, G.R) - std::max(r0 - p.depth, 0));
  }
  p.items = std::max(4, (most * words + 3) / 4 * 4);
  // a word of a phase each; in an exchange up to four words of the neighbours' rows
  p.group = (std::max(p.items, p.bands > 1 ? 2 * p.depth * words : 0) + 31) / 32 * 32;
  // Draw warps share the schedulers with the update warps, which they slow: no more of them than keep ahead
  // (n = 512, 40 words: 4, 6, 8, 12 draw warps 1.14, 1.10, 1.17, 1.25 us; n = 1024, 80 words: 8, 12, 16 1.93,
  // 1.84, 1.88 us).  Batches long enough that the barrier at their end does not count (n = 512: 4 and 8
  // phases 1.14 and 1.10 us).
  const int draw_warps = p.items <= 20 ? 4 : p.items <= 56 ? 6 : 12;
  p.batch = p.items <= 56 ? 8 : p.items <= 96 ? 4 : p.items <= 256 ? 2 : 1;
  auto bytes = [&]() {
    return (((size_t)chains * 4 * p.rows * G.P + 3) / 4 * 4 + (size_t)2 * p.batch * 2 * M * p.items +
            4 * (size_t)(p.depth + 1) + p.group) * sizeof(uint32_t);  // idle lanes read past the drawn bits
  };
  p.smem = bytes();
  if (chains * p.group > 512 || p.smem > 220 * 1024 || (p.bands > 1 && !coop) || p.bands > sms) return p;
  p.threads = chains * p.group + 32 * std::min(draw_warps, (kSvBandThreads - chains * p.group) / 32);
  p.xbuf_words = (size_t)2 * p.bands * 2 * chains * p.depth * 4 * words;
  p.kernel = chains == 1 ? (p.sum ? (void*)k_sv_bands<1, true> : (void*)k_sv_bands<1, false>)
                         : (p.sum ? (void*)k_sv_bands<2, true> : (void*)k_sv_bands<2, false>);
  int per_sm = 0;
  if (dev_allow_smem(p.kernel, p.smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, p.kernel, p.threads, p.smem) != cudaSuccess) {
    cudaGetLastError();
    return p;
  }
  p.ok = per_sm >= 1;
  return p;
}

// Allocates and runs: `chains` (1 or 2) chains start back to back in dev.chains.
struct SvRun {
  SvGeom G;
  int chains;
  std::vector<uint32_t> T;
  SvBandPlan plan;
  SvDevice dev;
  cudaStream_t st;
  bool bands = false;
  int teams = 1;  // attempts side by side

  // keep: run() is called again, from the same start.
  rt_status prepare(int engine, bool keep) {
    dev.stream = st;
    // Engine 2 is refused where 16 CTAs cannot hold the chains.
    if (engine == 2 && (size_t)chains * 4 * ((G.R + 15) / 16) * G.P * sizeof(uint32_t) > 200 * 1024)
      return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex: no thread-block cluster holds this size (engine 2)");
    if (engine != 1) plan = sv_band_plan(G, chains, T);
    // 256 words a band (n = 2048): 5.4 us a sweep, per-sub-sweep kernels 8.9; 484 (n = 2800): 13-15 and 11.
    bands = plan.ok && (engine == 2 || plan.items <= 320);
    if (bands && keep) teams = std::max(1, std::min(kSvTeams, plan.sms / plan.bands));
    const size_t bytes = chains * G.chain_words * sizeof(uint32_t);
    if (rt_status e = dev_alloc(&dev.chains, bytes, st)) return e;
    if (bands || keep)
      if (rt_status e = dev_alloc(&dev.other, (bands ? std::max(2, teams) : 1) * bytes, st)) return e;
    if (rt_status e = dev_alloc(&dev.flag, kFlagBytes, st)) return e;
    if (bands && plan.bands > 1)
      if (rt_status e = dev_alloc(&dev.xbuf, teams * plan.xbuf_words * sizeof(uint64_t), st)) return e;
    cudaMemsetAsync(dev.flag, 0, kFlagBytes, st);
    return RT_OK;
  }

  static constexpr size_t kFlagBytes = (4 + 2 * kSvTeams) * sizeof(int);

  SvBandArgs band_args(uint64_t seed, uint32_t stream) const {
    SvBandArgs A{};
    A.chain_words = G.chain_words;
    A.class_words = G.class_words;
    A.P = G.P;
    A.n = G.n;
    A.R = G.R;
    A.words = (G.n - 1) / 2 / 32 + 1;
    A.bands = plan.bands;
    A.depth = plan.depth;
    A.group = plan.group;
    A.batch = plan.batch;
    A.items = plan.items;
    A.rows = plan.rows;
    uint32_t order[9];
    const int by_sum[9] = {0, 1, 2, 5, 8, 0, 0, 0, 0};  // a threshold of each k1 + k2
    for (int m = 0; m < 9; ++m) order[m] = T[plan.sum ? by_sum[m] : m];
    sv_leaves(order, A.leaf);
    A.seed = seed;
    A.stream = stream;
    A.xbuf = dev.xbuf;
    A.error = dev.flag + 1;
    A.max_spin = test_silence().spin(1L << 22);
    A.silent_plus1 = test_silence().next_plus1();
    return A;
  }

  // Attempts [attempt0, attempt0 + n) of a coupling from the past side by side (n <= teams), attempt k from sweep
  // -(first << k); dev.flag's best tells the smallest that coalesced.
  void couple(uint64_t seed, uint32_t stream, int64_t first, int attempt0, int n) {
    SvBandArgs A = band_args(seed, stream);
    A.src = dev.chains;
    A.dst = dev.other;
    A.couple = 1;
    A.attempt0 = attempt0;
    A.first = first;
    A.xteam = plan.xbuf_words;
    A.best = dev.flag + 2;
    A.team = reinterpret_cast<int2*>(dev.flag + 4);
    cudaMemsetAsync(dev.flag, 0, kFlagBytes, st);
    cudaMemsetAsync(A.best, 0x7f, sizeof(int), st);
    void* args[] = {&A};
    if (plan.bands > 1) {
      cudaMemsetAsync(dev.xbuf, 0, n * plan.xbuf_words * sizeof(uint64_t), st);  // no stale tags
      cudaLaunchCooperativeKernel(plan.kernel, dim3(plan.bands, n), dim3(plan.threads), args, plan.smem, st);
    } else {
      cudaLaunchKernel(plan.kernel, dim3(1, n), dim3(plan.threads), args, plan.smem, st);
    }
  }

  // Sub-sweeps [s0, s0 + count), whole sweeps, from the start states; returns where the states are.
  uint32_t* run(uint64_t seed, uint32_t stream, int64_t s0, int64_t count) {
    const size_t words = chains * G.chain_words;
    if (count == 0) return dev.chains;
    if (!bands) {
      SvLaunch L{};
      L.base = dev.chains;
      if (dev.other) {
        L.base = dev.other;
        cudaMemcpyAsync(dev.other, dev.chains, words * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st);
      }
      L.chain_words = G.chain_words;
      L.class_words = G.class_words;
      L.P = G.P;
      L.n = G.n;
      sv_leaves(T.data(), L.leaf);
      L.seed = seed;
      L.stream = stream;
      for (int64_t s = s0; s < s0 + count; ++s) {
        fill_launch(L, G, s);
        const int threads = L.words * L.rows;
        if (threads <= 0) continue;
        pdl_launch(k_sv_sub, dim3((threads + 127) / 128, chains), dim3(128), st, L);
      }
      return L.base;
    }
    SvBandArgs A = band_args(seed, stream);
    A.src = dev.chains;
    constexpr int64_t kChunk = 1 << 14;  // sweeps per launch: bounds one launch to a fraction of a second
    for (int64_t done = 0; done < count / 4; done += kChunk) {
      A.dst = A.src == dev.other ? dev.other + words : dev.other;
      A.s0 = s0 + 4 * done;
      A.sweeps = (int)std::min(kChunk, count / 4 - done);
      void* args[] = {&A};
      if (plan.bands > 1) {
        cudaMemsetAsync(dev.xbuf, 0, plan.xbuf_words * sizeof(uint64_t), st);  // no stale tags
        cudaLaunchCooperativeKernel(plan.kernel, dim3(plan.bands), dim3(plan.threads), args, plan.smem, st);
      } else {
        cudaLaunchKernel(plan.kernel, dim3(1), dim3(plan.threads), args, plan.smem, st);
      }
      A.src = A.dst;
    }
    return const_cast<uint32_t*>(A.src);
  }
};

int64_t sv_interior_points(int n) { return (int64_t)(n - 1) * (n - 1); }

}  // namespace
}  // namespace rt

using namespace rt;

extern "C" {

RT_API rt_status rt_sv_thresholds(double a, double b, double c, uint32_t* out9) {
  clear_error();
  if (!out9) return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex thresholds: NULL output");
  if (!(a > 0 && b > 0 && c > 0) || !std::isfinite(a) || !std::isfinite(b) || !std::isfinite(c))
    return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex: weights must be finite and > 0");
  const std::vector<uint32_t> T = sv_thresholds_host(a, b, c);
  std::memcpy(out9, T.data(), 9 * sizeof(uint32_t));
  return RT_OK;
}

RT_API rt_status rt_sv_dwbc_height(int32_t n, int32_t top, int32_t* out) {
  clear_error();
  if (n < 1 || !out) return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex dwbc: n >= 1 and an output of (n+1)^2");
  const int L = n + 1;
  for (int y = 0; y <= n; ++y)
    for (int x = 0; x <= n; ++x) out[(size_t)y * L + x] = top ? std::min(x + y, 2 * n - x - y) : std::abs(x - y);
  return RT_OK;
}

RT_API rt_status rt_sv_height_to_asm(const int32_t* h, int32_t n, int32_t* out) {
  clear_error();
  if (n < 1 || !h || !out) return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex height_to_asm: bad arguments");
  if (!sv_valid_heights(h, n)) return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex: not a height function (|dh| != 1)");
  const int L = n + 1;
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) {
      const int nw = h[(size_t)i * L + j], ne = h[(size_t)i * L + j + 1];
      const int sw = h[(size_t)(i + 1) * L + j], se = h[(size_t)(i + 1) * L + j + 1];
      out[(size_t)i * n + j] = (ne + sw - nw - se) / 2;
    }
  return RT_OK;
}

RT_API rt_status rt_sv_asm_to_height(const int32_t* a, int32_t n, int32_t* out) {
  clear_error();
  if (n < 1 || !a || !out) return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex asm_to_height: bad arguments");
  const int L = n + 1;
  // h(y, x) = x + y - 2 * sum_{i < y, j < x} a(i, j)
  std::vector<int64_t> S((size_t)L * L, 0);
  for (int y = 1; y <= n; ++y)
    for (int x = 1; x <= n; ++x)
      S[(size_t)y * L + x] = a[(size_t)(y - 1) * n + x - 1] + S[(size_t)(y - 1) * L + x] + S[(size_t)y * L + x - 1] -
                             S[(size_t)(y - 1) * L + x - 1];
  for (int y = 0; y <= n; ++y)
    for (int x = 0; x <= n; ++x) out[(size_t)y * L + x] = (int32_t)(x + y - 2 * S[(size_t)y * L + x]);
  if (!sv_valid_heights(out, n)) return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex: not an alternating sign matrix");
  for (int k = 0; k <= n; ++k)
    if (out[(size_t)n * L + k] != n - k || out[(size_t)k * L + n] != n - k)
      return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex: not an alternating sign matrix (row or column sums)");
  return RT_OK;
}

RT_API rt_status rt_sv_walk(int32_t* h, int32_t n, int64_t sweeps, int64_t seed, const double* abc,
                            const rt_walk_opts* opts, rt_cftp_stats* stats) {
  clear_error();
  rt_walk_opts o;
  rt_walk_opts_default(&o);
  o.rng_mode = RT_RNG_FAST;
  if (opts) o = *opts;
  if (!h || sweeps < 0) return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex walk: NULL heights or negative sweeps");
  if (o.rng_mode != RT_RNG_FAST)
    return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex walk: only the fast (Philox) random mode exists for this model");
  if (o.fast_stream >= 65536u) return fail(RT_ERR_INVALID_ARGUMENT, "fast_stream must be < 65536");
  double a, b, c;
  if (rt_status st = sv_check_common(n, abc, &a, &b, &c)) return st;
  const SvGeom G = sv_geom(n);
  const size_t points = (size_t)(n + 1) * (n + 1);
  // Packed, checked and unpacked on the device from n = 96 up, where the host's 5 ns a point pass the device's two
  // launches and one wait (walk of 4 sweeps without them: n = 95 on the host 81 us, n = 96 on the device 67, n = 512
  // 1.4 ms and 92 us); the heights on the device take four bytes a point, 1 GB at most.
  bool on_device = n >= 96 && n <= 16384;
  const rt_status no_device = sv_check_device();
  if (no_device) on_device = false;
  const char* const invalid = "six-vertex: not a height function (|dh| != 1)";
  if (!on_device && !sv_valid_heights(h, n)) return fail(RT_ERR_INVALID_ARGUMENT, invalid);
  if (no_device) return sv_check_device();
  const std::vector<uint32_t> T = sv_thresholds_host(a, b, c);
  cudaStream_t st = (cudaStream_t)o.cuda_stream;
  SvRun R{G, 1, T};
  R.st = st;
  if (rt_status e = R.prepare(o.engine, false)) {
    if (on_device && !sv_valid_heights(h, n)) return fail(RT_ERR_INVALID_ARGUMENT, invalid);
    return e;
  }
  if (on_device && dev_alloc(&R.dev.heights, points * sizeof(int32_t), st)) {  // no room for them: on the host
    clear_error();
    on_device = false;
    if (!sv_valid_heights(h, n)) return fail(RT_ERR_INVALID_ARGUMENT, invalid);
  }
  std::vector<uint32_t> bits;
  if (on_device) {
    int bad = 0;
    cudaMemcpyAsync(R.dev.heights, h, points * sizeof(int32_t), cudaMemcpyHostToDevice, st);
    cudaMemsetAsync(R.dev.chains, 0, G.chain_words * sizeof(uint32_t), st);  // the guard words
    k_sv_pack<<<((n + 1) * (G.P - 2) + 7) / 8, 256, 0, st>>>(R.dev.heights, R.dev.chains, G, R.dev.flag);
    cudaMemcpyAsync(&bad, R.dev.flag, sizeof bad, cudaMemcpyDeviceToHost, st);
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail(RT_ERR_CUDA, std::string("six-vertex walk: ") + cudaGetErrorString(e));
    if (bad) return fail(RT_ERR_INVALID_ARGUMENT, invalid);
  } else {
    bits.resize(G.chain_words);
    sv_pack(h, G, bits.data());
    cudaMemcpyAsync(R.dev.chains, bits.data(), bits.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, st);
  }
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, st);
  const uint32_t* at = R.run((uint64_t)seed, o.fast_stream, 0, 4 * sweeps);
  cudaError_t err = cudaGetLastError();
  cudaEventRecord(e1, st);
  int flag[2] = {0, 0};
  cudaMemcpyAsync(flag, R.dev.flag, sizeof flag, cudaMemcpyDeviceToHost, st);
  if (on_device)
    k_sv_unpack<<<(n + 1 + 7) / 8, 256, 0, st>>>(at, G, R.dev.heights);
  else
    cudaMemcpyAsync(bits.data(), at, bits.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
  cudaError_t waited = cudaStreamSynchronize(st);
  if (err == cudaSuccess) err = waited;
  float ms = 0.f;
  if (err == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (err != cudaSuccess) return fail(RT_ERR_CUDA, std::string("six-vertex walk: ") + cudaGetErrorString(err));
  if (flag[1]) return fail(RT_ERR_TIMEOUT, "six-vertex walk: a band gave up waiting for a neighbour's rows");
  if (on_device) {
    if (cudaMemcpyAsync(h, R.dev.heights, points * sizeof(int32_t), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        (waited = cudaStreamSynchronize(st)) != cudaSuccess) {
      cudaGetLastError();
      return fail(RT_ERR_CUDA, "six-vertex walk: copying the heights back failed");
    }
  } else {
    std::vector<int32_t> start(h, h + points);
    sv_unpack(bits.data(), G, start.data(), h);
  }
  if (stats) {
    std::memset(stats, 0, sizeof *stats);
    stats->attempts = 1;
    stats->total_steps = 4 * sweeps;
    stats->final_steps = 4 * sweeps;
    stats->flip_attempts = sv_interior_points(n) * sweeps;
    stats->seconds = ms * 1e-3;
  }
  return RT_OK;
}

RT_API rt_status rt_sv_cftp(const int32_t* hmax, const int32_t* hmin, int32_t n, int64_t seed, int64_t first_sweeps,
                            int32_t max_attempts, const double* abc, const rt_walk_opts* opts, int32_t* out,
                            rt_cftp_stats* stats) {
  clear_error();
  rt_walk_opts o;
  rt_walk_opts_default(&o);
  o.rng_mode = RT_RNG_FAST;
  if (opts) o = *opts;
  if (!hmax || !hmin || !out || first_sweeps < 1 || max_attempts < 1)
    return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex cftp: bad arguments");
  if (o.rng_mode != RT_RNG_FAST)
    return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex cftp: only the fast (Philox) random mode exists for this model");
  if (o.fast_stream >= 65536u) return fail(RT_ERR_INVALID_ARGUMENT, "fast_stream must be < 65536");
  double a, b, c;
  if (rt_status st = sv_check_common(n, abc, &a, &b, &c)) return st;
  if (c < a || c < b)
    return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex cftp: the heat-bath coupling is monotone only for c >= max(a, b)");
  if (!sv_valid_heights(hmax, n) || !sv_valid_heights(hmin, n))
    return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex: not a height function (|dh| != 1)");
  const int L = n + 1;
  for (int y = 0; y <= n; ++y)
    for (int x = 0; x <= n; ++x) {
      const bool edge = y == 0 || x == 0 || y == n || x == n;
      const int32_t u = hmax[(size_t)y * L + x], v = hmin[(size_t)y * L + x];
      if ((edge && u != v) || u < v)
        return fail(RT_ERR_INVALID_ARGUMENT, "six-vertex cftp: hmax must dominate hmin with the same boundary");
    }
  if (rt_status st = sv_check_device()) return st;
  const SvGeom G = sv_geom(n);
  const std::vector<uint32_t> T = sv_thresholds_host(a, b, c);
  cudaStream_t st = (cudaStream_t)o.cuda_stream;
  SvRun R{G, 2, T};
  R.st = st;
  if (rt_status e = R.prepare(o.engine, true)) return e;
  std::vector<uint32_t> start(2 * G.chain_words);
  sv_pack(hmax, G, start.data());
  sv_pack(hmin, G, start.data() + G.chain_words);
  cudaMemcpyAsync(R.dev.chains, start.data(), start.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, st);
  if (stats) std::memset(stats, 0, sizeof *stats);
  const uint32_t* at = R.dev.chains;
  float total_ms = 0.f;
  int64_t total_sub = 0;
  // Attempts in groups of up to four, side by side (n = 48, first 64 sweeps: 3.9 -> 2.4 ms), up to 2^17 sweeps each
  // (about 0.1 s); longer ones alone, in several launches.
  for (int attempt = 0; attempt < max_attempts;) {
    if (attempt > 44 || first_sweeps > ((int64_t)1 << 44) >> attempt) break;
    int n = 0;
    while (R.bands && n < R.teams && attempt + n < max_attempts && attempt + n < 44 &&
           first_sweeps <= ((int64_t)1 << 17) >> (attempt + n))
      ++n;
    const int64_t Tsw = first_sweeps << attempt;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, st);
    if (n > 0) {
      R.couple((uint64_t)seed, o.fast_stream, first_sweeps, attempt, n);
      cudaEventRecord(e1, st);
    } else {
      cudaMemsetAsync(R.dev.flag, 0, 2 * sizeof(int), st);
      at = R.run((uint64_t)seed, o.fast_stream, -4 * Tsw, 4 * Tsw);
      cudaEventRecord(e1, st);
      k_sv_diff<<<64, 256, 0, st>>>(at, at + G.chain_words, G.chain_words, (uint32_t*)R.dev.flag);
    }
    cudaError_t err = cudaGetLastError();
    int flag[3] = {1, 0, 0};
    cudaMemcpyAsync(flag, R.dev.flag, sizeof flag, cudaMemcpyDeviceToHost, st);
    const cudaError_t waited = cudaStreamSynchronize(st);
    if (err == cudaSuccess) err = waited;
    float ms = 0.f;
    if (err == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (err != cudaSuccess) return fail(RT_ERR_CUDA, std::string("six-vertex cftp: ") + cudaGetErrorString(err));
    if (flag[1]) return fail(RT_ERR_TIMEOUT, "six-vertex cftp: a band gave up waiting for a neighbour's rows");
    total_ms += ms;
    int ran = 1;
    bool differ = flag[0] != 0;
    if (n > 0) {
      differ = flag[2] >= attempt + n;
      ran = differ ? n : flag[2] - attempt + 1;
      at = R.dev.other + (size_t)(ran - 1) * 2 * G.chain_words;
    }
    for (int k = 0; k < ran; ++k, ++attempt) {
      total_sub += 4 * (first_sweeps << attempt);
      if (stats) {
        stats->attempts = attempt + 1;
        stats->total_steps = total_sub;
        stats->flip_attempts += 2 * sv_interior_points(G.n) * (first_sweeps << attempt);
        stats->seconds = total_ms * 1e-3;
      }
    }
    if (!differ) {
      std::vector<uint32_t> bits(G.chain_words);
      cudaMemcpy(bits.data(), at, bits.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost);
      sv_unpack(bits.data(), G, hmax, out);
      if (stats) stats->final_steps = 4 * (first_sweeps << (attempt - 1));
      return RT_OK;
    }
  }
  // not coalesced: out holds the top chain of the last attempt
  std::vector<uint32_t> bits(G.chain_words);
  if (cudaMemcpy(bits.data(), at, bits.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost) == cudaSuccess)
    sv_unpack(bits.data(), G, hmax, out);
  return fail(RT_ERR_NOT_COALESCED, "six-vertex cftp: chains did not coalesce within max_attempts");
}

}  // extern "C"
