// Grid engine of the domino sweep: the bit planes of domino_cluster.cu on every SM.
//
// A band of colour-array rows per SM (one cooperative launch), planes, flips and draws as in the
// cluster kernel: draw warps compose a run's half-sweeps into move words, a run ahead of the update
// warps, which apply them.  The two overlap, so a run takes the longer of its draws and of its
// exchange.
//
// Exchange: a word of a band's first (last) row shares its up (down) edges with the band above
// (below).  After each run it stores the plane word that the run changed as a 64-bit word tagged with
// the run (single-copy atomic: who sees the tag sees the data), one slot per run parity; the facing
// word polls for the run before, takes the new plane word from it and goes on.  A band is at most
// one run ahead of a facing neighbour, so a slot is rewritten only after it was read.  Runs of a
// launch alternate in colour, so the two parities' slots hold the last changes of both planes when
// the launch ends.  Every wait is bounded.
//
// Bound: mid-size domains by the exchange, 0.85 us a run through L2 (k_deep below makes one exchange serve
// several runs); from order 700 up by the issue of the draws (order 1024: 237 words a band, about 24
// instructions a word and half-sweep).  Measured (us per half-sweep, before: the band kernel with polled
// deltas, domino_bits.cu, which draws, exchanges and writes back in turn): TinyMT order 400 0.62 (1.05), 512
// 0.71 (1.2), 1024 with two chains 1.36 (1.95); fast mode order 1024 1.35 (3.2).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <string>
#include <vector>

#include "domino_grid.h"
#include "domino_planes.cuh"
#include "domino_runs.h"
#include "domino_sweep.h"
#include "rng.cuh"

namespace rt {

namespace {

// Threads a CTA: 64 registers a thread, 80 where the generators of 8 words need them.  16 words: 16 draw
// warps and 4 update warps launched with 96 registers a thread, of which the update warps give
// up 32 each to the draw warps' 104 (the sum stays the launch's).
constexpr int gr_max_threads(bool fast, int slots) { return fast || slots <= 4 ? 1024 : (slots <= 8 ? 768 : 640); }
constexpr bool gr_splits(bool fast, int slots) { return !fast && slots == 16; }

struct GrArgs {
  uint8_t* base;
  int N, P, cols, bands, draw_warps;
  size_t chain_stride, colour_stride;
  uint4* tmt;
  const uint4* tmt_params;
  const int* cand;  // [2][N]
  const int* row_start;
  const int* windows;  // [band]{first word, words}
  int xlo, xn;         // the exchange rows' first word and words
  DmRule rule;
  const uint32_t* runs;  // TinyMT: (colour << 31) | length
  int nruns;             // fast mode: half-sweeps
  uint64_t seed;
  uint32_t stream;
  int64_t h0;
  uint64_t* xbuf;  // [run parity][band][to above, to below][xn][chain]
  int* error;
  long max_spin;
  int silent_band_plus1;
  int depth, first, last;  // k_deep: runs between exchanges; the first and last row of any band
  // Coupling from the past (k_deep, couple, two chains): blockIdx.y = k runs attempt attempt0 + k from the chains
  // at start into the k-th pair at base, and leaves once a smaller one has coalesced.
  int couple, attempt0;
  int64_t first_sweeps;  // fast mode: half-sweeps [-2 first_sweeps << attempt, 0)
  const uint8_t* start;
  size_t team_stride, xteam;
  int* best;                    // smallest attempt that coalesced
  int2* team;                   // [k] {bands whose chains differ, bands done}
  const int4* attempt_desc;     // TinyMT, [k]: {first run, runs, first epoch seed, 0}
  const uint32_t* epoch_seeds;  // a run that starts an epoch (bit 30) seeds the generators from the next
};

// Bounded wait for the element's tag; false (and the error word set) when it gave up, or another band did.
__device__ __forceinline__ bool gr_recv(const uint64_t* g, uint32_t tag, uint32_t& v, long max_spin, int* error,
                                        const int* best = nullptr, int attempt = 0) {
  for (long it = 0; it <= max_spin; ++it) {
    uint64_t x;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(x) : "l"(g) : "memory");
    v = (uint32_t)x;
    if ((uint32_t)(x >> 32) == tag) return true;
    if ((it & 255) == 255 && (*static_cast<volatile int*>(error) || (best && *static_cast<const volatile int*>(best) < attempt)))
      return false;
  }
  atomicExch(error, 1);
  return false;
}
__device__ __forceinline__ void gr_send(uint64_t* g, uint32_t tag, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(g), "l"(((uint64_t)tag << 32) | v) : "memory");
}

// KS: words per draw warp; UI: words and chains per update lane.
template <int NCH, int kMode, int KS, int UI>
__global__ void __launch_bounds__(gr_max_threads(kMode == kClFast, KS), 1) k_grid(const __grid_constant__ GrArgs a) {
  extern __shared__ __align__(16) uint32_t sm[];
  __shared__ uint4 srule[4];
  __shared__ int s_cnt[2];
  __shared__ uint32_t s_colour[2];
  __shared__ int s_failed;
  constexpr bool kFast = kMode == kClFast, kParams = kMode == kClTmtParams;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = (int)(blockDim.x >> 5);
  const int ndraw = a.draw_warps, nslots = ndraw * KS, band = blockIdx.x;
  const int r0 = a.row_start[band], r1 = a.row_start[band + 1], R = r1 - r0 + 1;
  const int wlo = a.windows[2 * band], wn = a.windows[2 * band + 1];  // this band's window words
  const bool has_up = band > 0, has_dn = band + 1 < a.bands;
  if (tid < 4)
    srule[tid] = kFast ? make_uint4(a.rule.w_up[tid], a.rule.lo_dn[tid], a.rule.w_dn[tid], 0u)
                       : make_uint4(a.rule.w_up[tid] << 9, a.rule.lo_dn[tid] << 9, a.rule.w_dn[tid] << 9, 0u);
  // Shared memory: planes [R rows from r0 - 1][wn][NCH][4]; a scratch word; the slots (row << 16) |
  // word, valid cells (0: none); the moves [run parity][slot]; the slot of each item.
  uint32_t* const pad = sm + R * 4 * wn * NCH;
  uint2* const sslot = reinterpret_cast<uint2*>(pad + kClPad);
  uint2* const smove = sslot + nslots;
  uint16_t* const sitem = reinterpret_cast<uint16_t*>(smove + 2 * nslots);
  for (int k = tid; k < nslots; k += (int)blockDim.x) sslot[k] = make_uint2(0u, 0u);
  if (tid < 2) s_cnt[tid] = 0;
  if (tid == 0) s_failed = 0;
  __syncthreads();
  auto row_words = [&](int i, int* w0) -> int {
    const int lo = a.cand[i], hi = a.cand[a.N + i];
    if (i < 1 || i > a.N - 2 || lo == INT_MAX) return 0;
    *w0 = lo >> 5;
    return (hi >> 5) - (lo >> 5) + 1;
  };
  for (int i = r0 + tid; i < r1; i += (int)blockDim.x) {
    int w0 = 0;
    const int c = row_words(i, &w0);
    if (c) atomicAdd(&s_cnt[i & 1], c);
  }
  __syncthreads();
  // Slots as in the cluster kernel: each parity's words in equal blocks over its share of the warps.
  // Items: the last row's words, the first row's, then the others in row order.
  const int c0 = s_cnt[0], c1 = s_cnt[1], nwords = c0 + c1;
  const int need0 = (c0 + KS - 1) / KS, need1 = (c1 + KS - 1) / KS;
  int cw0 = nwords > 0 ? (ndraw * c0 + nwords / 2) / nwords : ndraw;
  cw0 = min(max(cw0, need0), ndraw - need1);
  const int cw1 = ndraw - cw0;
  const int per0 = cw0 ? (c0 + cw0 - 1) / cw0 : 1, per1 = cw1 ? (c1 + cw1 - 1) / cw1 : 1;
  int first_w0 = 0;
  const int n_first = row_words(r0, &first_w0), n_last = r1 - 1 > r0 ? row_words(r1 - 1, &first_w0) : 0;
  for (int i = r0 + tid; i < r1; i += (int)blockDim.x) {
    int w0 = 0, before = 0, inner = 0;
    const int c = row_words(i, &w0);
    for (int q = r0; q < i; ++q) {
      int x;
      const int n = row_words(q, &x);
      if (((q ^ i) & 1) == 0) before += n;
      if (q > r0) inner += n;
    }
    const int per = (i & 1) ? per1 : per0, first = (i & 1) ? cw0 : 0;
    const int item = i == r0 ? n_last : (i == r1 - 1 ? 0 : n_last + n_first + inner);
    const int lo = a.cand[i], hi = a.cand[a.N + i];
    for (int k = 0; k < c; ++k) {
      const int w = w0 + k, at = before + k, slot = (first + at / per) * KS + at % per;
      const int blo = max(lo - 32 * w, 0), bhi = min(hi - 32 * w, 31);
      const uint32_t valid = (0xffffffffu << blo) & (0xffffffffu >> (31 - bhi));
      sslot[slot] = make_uint2(((uint32_t)i << 16) | (uint32_t)w, valid);
      sitem[item + k] = (uint16_t)slot;
    }
  }
  cl_load_window<NCH>(sm, a.base, a.chain_stride, a.colour_stride, a.P, r0 - 1, R, wlo, wn);
  __syncthreads();
  auto xel = [&](uint32_t par, int b, int to_below, int xi) -> uint64_t* {
    return a.xbuf + (((size_t)par * a.bands + b) * 2 + to_below) * (size_t)(a.xn * NCH) + xi;
  };
  auto run_at = [&](int j) -> uint32_t {
    if (kFast) return ((a.h0 + j) & 1) ? 1u : 0x80000001u;  // even half-sweeps black (colour 1)
    return j < a.nruns ? __ldg(&a.runs[j]) : 0u;
  };
  const int nruns = a.nruns;
  bool failed = false;
  if (warp >= ndraw) {
    // ---- update warps
    if constexpr (gr_splits(kFast, KS)) asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    enum : uint32_t { kPubUp = 1, kPubDn = 2, kLinkUp = 4, kLinkDn = 8, kOdd = 16 };
    const uint32_t pitch = (uint32_t)(wn * NCH * 16), move_bytes = (uint32_t)(nslots * sizeof(uint2));
    uint32_t above[UI], valid[UI], move_at[UI], flags[UI];  // flags: the exchange index << 8 as well
    bool edge[UI];
    auto word_at = [&](int i, int w) -> bool {
      int w0 = 0;
      const int c = row_words(i, &w0);
      return w >= w0 && w < w0 + c;
    };
#pragma unroll
    for (int u = 0; u < UI; ++u) {
      const int idx = tid - 32 * ndraw + u * 32 * (nwarps - ndraw), k = idx / NCH, c = idx % NCH;
      const int slot = k < nwords ? (int)sitem[k] : 0;
      const uint2 e = k < nwords ? sslot[slot] : make_uint2(0u, 0u);
      const bool mine = e.y != 0u;
      const int i = (int)(e.x >> 16), w = (int)(e.x & 0xffffu), xi = (w - a.xlo) * NCH + c;
      valid[u] = e.y;
      move_at[u] = (uint32_t)__cvta_generic_to_shared(smove + slot);
      // (a lane without a word works on the scratch words, whose row below is `pitch` on)
      above[u] = (uint32_t)__cvta_generic_to_shared(mine ? sm + (((i - r0) * wn + w - wlo) * NCH + c) * 4 : pad + 8);
      uint32_t f = 0u;
      if (mine) {
        f = (uint32_t)xi << 8 | ((i & 1) ? kOdd : 0u);
        if (has_up && i == r0) f |= kPubUp | (word_at(i - 1, w) ? kLinkUp : 0u);
        if (has_dn && i == r1 - 1) f |= kPubDn | (word_at(i + 1, w) ? kLinkDn : 0u);
      }
      flags[u] = f;
      edge[u] = __any_sync(~0u, f & (kPubUp | kPubDn));
    }
    const bool silent = band + 1 == a.silent_band_plus1;  // test hook: publishes nothing
    __syncthreads();  // the first run's moves are drawn
    for (int j = 0; j < nruns; ++j) {
      const uint32_t b = (uint32_t)j & 1u, t = s_colour[b];
      bool live = !*static_cast<volatile int*>(&s_failed);
      const uint32_t off_u = t ? 0u : 4u, off_d = 4u - off_u;
#pragma unroll
      for (int u = 0; u < UI; ++u) {
        const uint32_t here = valid[u] ? above[u] + pitch : above[u];
        const uint2 move = cl_lds2(move_at[u] + b * move_bytes);
        const uint2 ab = cl_lds2(above[u]);
        const uint4 me = cl_lds4(here);
        const uint32_t west = cl_lds(here - 16u * NCH + 12u);
        const bool aligned = ((flags[u] & kOdd) != 0u) == (t != 0u);  // left HE, right HO of the same word
        uint32_t U = t ? ab.x : ab.y, D = t ? me.y : me.x;
        if (edge[u] && j > 0) {
          // the neighbours' words of the run before, which changed these planes (the vote wants all the warp's lanes,
          // whatever each has read of s_failed)
          const int xi = (int)(flags[u] >> 8);
          bool ok = live;
          if (ok && (flags[u] & kLinkUp)) ok = gr_recv(xel(b ^ 1u, band - 1, 1, xi), (uint32_t)j, U, a.max_spin, a.error);
          if (ok && (flags[u] & kLinkDn)) ok = gr_recv(xel(b ^ 1u, band + 1, 0, xi), (uint32_t)j, D, a.max_spin, a.error);
          if (!__all_sync(~0u, ok)) {
            live = false;
            failed = true;
            s_failed = 1;
          }
        }
        const uint32_t lft = aligned ? me.z : __funnelshift_l(west, me.w, 1), rgt = aligned ? me.w : me.z;
        // Flippable: up = down, left = right, up != left (states 3 and 12); T: cells whose state at
        // the end of the run differs.
        const uint32_t flip = ~(U ^ D) & ~(lft ^ rgt) & (U ^ lft) & valid[u];
        const uint32_t T = flip & ((U & ~move.x) | (~U & move.y));
        const uint32_t new_u = U ^ T, new_d = D ^ T;
        if (edge[u] && live && !silent) {
          const int xi = (int)(flags[u] >> 8);
          if (flags[u] & kPubUp) gr_send(xel(b, band, 0, xi), (uint32_t)j + 1u, new_u);
          if (flags[u] & kPubDn) gr_send(xel(b, band, 1, xi), (uint32_t)j + 1u, new_d);
        }
        if (valid[u]) {
          cl_sts(above[u] + off_u, new_u);
          cl_sts(here + off_d, new_d);
          cl_sts(here + 8u, me.z ^ T);
          // HO: the word itself, or (left edges of an unaligned row) bit k - 1 of this word and bit
          // 31 of the word to the left, whose other bits belong to that word's cells.
          cl_xor(here + 12u, aligned ? T : T >> 1);
          cl_xor_if(here - 16u * NCH + 12u, aligned ? 0u : T << 31);
        }
      }
      if ((j & 63) != 63) {
        cl_cta_sync();
      } else if (__syncthreads_or(failed ? 1 : 0)) {  // a band that gave up leaves within 64 runs
        failed = true;
        break;
      }
    }
  } else {
    // ---- draw warps
    if constexpr (gr_splits(kFast, KS)) asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    const int par = (int)((sslot[warp * KS].x >> 16) & 1u);
    auto gen_index = [&](int s, bool* v) -> int64_t {
      const uint2 e = sslot[warp * KS + s];
      *v = (e.y >> lane) & 1u;
      return (int64_t)((int)(e.x >> 16) - 1) * a.cols + (32 * (int)(e.x & 0xffffu) + lane - 1);
    };
    auto params_of = [&](int s, uint32_t& m1, uint32_t& m2, uint32_t& tm) {
      m1 = kTmtMat1;
      m2 = kTmtMat2;
      tm = kTmtTmat;
      if (kParams) {
        // (lanes without a cell read the first entry)
        bool v;
        const int64_t g = gen_index(s, &v);
        const uint4 p = __ldg(&a.tmt_params[v ? g : 0]);
        m1 = p.x;
        m2 = p.y;
        tm = p.z;
      }
    };
    uint4 gen[kFast ? 1 : KS];
    uint32_t f_row[kFast ? KS / 4 : 1], f_quad[kFast ? KS / 4 : 1];
    int groups = 0;
    if constexpr (!kFast) {
#pragma unroll
      for (int s = 0; s < KS; ++s) {
        bool v;
        const int64_t g = gen_index(s, &v);
        gen[s] = make_uint4(0u, 0u, 0u, 0u);
        if (v) gen[s] = a.tmt[g];
      }
    } else {
#pragma unroll
      for (int g = 0; g < KS / 4; ++g) {
        const uint2 e = sslot[warp * KS + 4 * g + (lane >> 3)];
        f_row[g] = e.x >> 16;
        f_quad[g] = (e.x & 0xffffu) * 8u + (uint32_t)(lane & 7);
        if (__any_sync(~0u, e.y)) groups = g + 1;
      }
    }
    auto draw_run = [&](uint32_t run, int64_t h, uint2* out) {
      const uint4 rl = srule[par | ((int)(run >> 31) << 1)];
      if constexpr (!kFast) {
        cl_moves_tmt<KS>(gen, rl, (int)(run & 0x3fffffffu), out + warp * KS, params_of);
      } else {
#pragma unroll
        for (int g = 0; g < KS / 4; ++g) {
          if (g > 0 && g >= groups) break;
          cl_moves_fast(a.seed, a.stream, h, f_row[g], f_quad[g], rl, out + warp * KS + 4 * g);
        }
      }
    };
    uint32_t next = run_at(1);
    if (nruns > 0) {
      const uint32_t run = run_at(0);
      draw_run(run, a.h0, smove);
      if (tid == 0) s_colour[0] = run >> 31;
    }
    __syncthreads();
    for (int j = 0; j < nruns; ++j) {
      const uint32_t after = run_at(j + 2);
      if (j + 1 < nruns) {
        if (tid == 0) s_colour[(j + 1) & 1] = next >> 31;
        draw_run(next, a.h0 + j + 1, smove + ((j + 1) & 1) * nslots);
      }
      next = after;
      if ((j & 63) != 63) {
        cl_cta_sync();
      } else if (__syncthreads_or(0)) {
        failed = true;
        break;
      }
    }
    if constexpr (!kFast) {
#pragma unroll
      for (int s = 0; s < KS; ++s) {
        bool v;
        const int64_t g = gen_index(s, &v);
        if (v) a.tmt[g] = gen[s];
      }
    }
  }
  __syncthreads();
  // The neighbours' last words into this band's copies of the shared planes: of the last run, all;
  // of the run before, those of words that have no word of this band facing them (the others were
  // taken, and changed since by this band's last run).
  if (nruns > 0 && !failed && !s_failed) {
    const uint32_t last = (uint32_t)nruns - 1u, t = s_colour[last & 1u];
    int up_w0 = 0, dn_w0 = 0, w0 = 0;
    const int n_up = has_up ? row_words(r0 - 1, &up_w0) * NCH : 0, n_dn = has_dn ? row_words(r1, &dn_w0) * NCH : 0;
    for (int k = tid; k < n_up + n_dn; k += (int)blockDim.x) {
      const bool up = k < n_up;
      const int q = up ? k : k - n_up, w = (up ? up_w0 : dn_w0) + q / NCH, c = q % NCH, xi = (w - a.xlo) * NCH + c;
      uint32_t* const pl = sm + (((up ? 0 : R - 1) * wn + w - wlo) * NCH + c) * 4;
      const int nb = up ? band - 1 : band + 1, dir = up ? 1 : 0;
      const int n_mine = row_words(up ? r0 : r1 - 1, &w0);
      const bool faced = w >= w0 && w < w0 + n_mine;
      uint32_t v = 0u;
      if (!gr_recv(xel(last & 1u, nb, dir, xi), last + 1u, v, a.max_spin, a.error)) {
        failed = true;
        break;
      }
      pl[up ? t : 1u - t] = v;
      if (faced || last == 0u) continue;
      if (!gr_recv(xel((last & 1u) ^ 1u, nb, dir, xi), last, v, a.max_spin, a.error)) {
        failed = true;
        break;
      }
      pl[up ? 1u - t : t] = v;
    }
  }
  if (__syncthreads_or(failed || s_failed ? 1 : 0) && tid == 0) atomicExch(a.error, 1);
  cl_store_window<NCH>(sm, a.base, a.chain_stride, a.colour_stride, a.P, a.cols, r0 - 1, R, wlo, wn);
}

// The same sweep with an exchange every `depth` runs: a band also updates rows beyond its own, whose draws it
// repeats, one row fewer on each side with every run, and takes the rows around its own anew (all four planes,
// from the bands that own them) before the next `depth` runs.  One word or chain per update lane.  The draw
// warps are a period of `depth` runs ahead, and only the update warps meet after every run.
// Bound: a run's dependent instructions, 0.13 us, the exchange of a period, 0.7 us, and the issue of the draws,
// the spare rows' included.  Measured (us per half-sweep, before: one cluster, domino_cluster.cu): TinyMT order
// 16 0.17 (0.22), 40 0.23 (0.30), 100 0.30 (0.37), 200 0.38 (0.50 in k_grid); fast mode order 16 0.22 (0.31),
// 40 0.27 (0.51), 100 0.34 (0.54), 300 0.56 (1.08 in k_grid).
//
// Coupling from the past: four attempts side by side on a quarter of the SMs each; a band leaves an attempt once
// a smaller one has coalesced, and the last band to finish tells whether its chains met.  Exact samples (before:
// domino_cluster.cu, also four side by side): fast mode order 8 0.28 ms (0.57), 40 6.3 (9.6), 48 11.3 (20.0); TinyMT
// order 15 0.74 (1.25), 32 4.0 (7.3), 48 17.9 (21.1).
constexpr int kGrMove = 4;  // words of an exchange a lane sends, and takes
constexpr int kGrMaxDepth = 12;

template <int NCH, int kMode, int KS>
__global__ void __launch_bounds__(gr_max_threads(kMode == kClFast, KS), 1) k_deep(const __grid_constant__ GrArgs a) {
  extern __shared__ __align__(16) uint32_t sm[];
  __shared__ uint4 srule[4];
  __shared__ int s_cnt[2];
  __shared__ uint32_t s_colour[2][kGrMaxDepth];
  __shared__ int s_stop[2];  // a smaller attempt coalesced, by parity of the period
  constexpr bool kFast = kMode == kClFast, kParams = kMode == kClTmtParams;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = (int)(blockDim.x >> 5);
  const int ndraw = a.draw_warps, nslots = ndraw * KS, band = blockIdx.x, depth = a.depth;
  const int r0 = a.row_start[band], r1 = a.row_start[band + 1];
  const int u0 = max(r0 - (depth - 1), a.first), u1 = min(r1 + depth, a.last + 1);  // rows updated in some run
  const int i0 = u0 - 1, R = u1 - i0;                                              // window rows
  const int wlo = a.windows[2 * band], wn = a.windows[2 * band + 1];
  if (tid < 4)
    srule[tid] = kFast ? make_uint4(a.rule.w_up[tid], a.rule.lo_dn[tid], a.rule.w_dn[tid], 0u)
                       : make_uint4(a.rule.w_up[tid] << 9, a.rule.lo_dn[tid] << 9, a.rule.w_dn[tid] << 9, 0u);
  // Shared memory as in k_grid: planes, a scratch word, slots, moves [period parity][run of the period][slot], the
  // slot of each item.
  uint32_t* const pad = sm + R * 4 * wn * NCH;
  uint2* const sslot = reinterpret_cast<uint2*>(pad + kClPad);
  uint2* const smove = sslot + nslots;
  uint16_t* const sitem = reinterpret_cast<uint16_t*>(smove + 2 * depth * nslots);
  for (int k = tid; k < nslots; k += (int)blockDim.x) sslot[k] = make_uint2(0u, 0u);
  if (tid < 2) s_cnt[tid] = 0;
  __syncthreads();
  auto row_words = [&](int i, int* w0) -> int {
    const int lo = i >= 1 && i <= a.N - 2 ? a.cand[i] : INT_MAX, hi = i >= 1 && i <= a.N - 2 ? a.cand[a.N + i] : 0;
    if (lo == INT_MAX) return 0;
    *w0 = lo >> 5;
    return (hi >> 5) - (lo >> 5) + 1;
  };
  for (int i = u0 + tid; i < u1; i += (int)blockDim.x) {
    int w0 = 0;
    const int c = row_words(i, &w0);
    if (c) atomicAdd(&s_cnt[i & 1], c);
  }
  __syncthreads();
  const int c0 = s_cnt[0], c1 = s_cnt[1], nwords = c0 + c1;
  const int need0 = (c0 + KS - 1) / KS, need1 = (c1 + KS - 1) / KS;
  int cw0 = nwords > 0 ? (ndraw * c0 + nwords / 2) / nwords : ndraw;
  cw0 = min(max(cw0, need0), ndraw - need1);
  const int cw1 = ndraw - cw0;
  const int per0 = cw0 ? (c0 + cw0 - 1) / cw0 : 1, per1 = cw1 ? (c1 + cw1 - 1) / cw1 : 1;
  for (int i = u0 + tid; i < u1; i += (int)blockDim.x) {
    int w0 = 0, before = 0, item = 0;
    const int c = row_words(i, &w0);
    for (int q = u0; q < i; ++q) {
      int x;
      const int n = row_words(q, &x);
      if (((q ^ i) & 1) == 0) before += n;
      item += n;
    }
    const int per = (i & 1) ? per1 : per0, first = (i & 1) ? cw0 : 0;
    for (int k = 0; k < c; ++k) {
      const int w = w0 + k, at = before + k, slot = (first + at / per) * KS + at % per;
      const int blo = max(a.cand[i] - 32 * w, 0), bhi = min(a.cand[a.N + i] - 32 * w, 31);
      sslot[slot] = make_uint2(((uint32_t)i << 16) | (uint32_t)w, (0xffffffffu << blo) & (0xffffffffu >> (31 - bhi)));
      sitem[item + k] = (uint16_t)slot;
    }
  }
  const bool couple = NCH == 2 && a.couple;
  const int team = couple ? (int)blockIdx.y : 0, attempt = a.attempt0 + team;
  cl_load_window<NCH>(sm, couple ? a.start : a.base, a.chain_stride, a.colour_stride, a.P, i0, R, wlo, wn);
  __syncthreads();
  int nruns = a.nruns, epoch = 0;
  const uint32_t* runs = a.runs;
  int64_t h0 = a.h0;
  if (couple) {
    if (kFast) {
      nruns = (int)(2 * (a.first_sweeps << attempt));
      h0 = -(int64_t)nruns;
    } else {
      const int4 d = a.attempt_desc[team];
      runs += d.x;
      nruns = d.y;
      epoch = d.z;
    }
  }
  uint64_t* const xbuf = a.xbuf + team * a.xteam;
  auto run_at = [&](int j) -> uint32_t {
    if (kFast) return ((h0 + j) & 1) ? 1u : 0x80000001u;  // even half-sweeps black (colour 1)
    return j < nruns ? __ldg(&runs[j]) : 0u;
  };
  // Runs left before the next exchange at which row i is first needed.
  auto needed = [&](int i) { return i < r0 ? r0 - i + 1 : (i >= r1 ? i - r1 + 1 : 1); };
  const int periods = (nruns + depth - 1) / depth;
  bool dead = false;  // a wait gave up: no more waits, the launch runs to its end
  if (warp >= ndraw) {
    // ---- update warps
    const int ut = tid - 32 * ndraw, nupd = 32 * (nwarps - ndraw);
    const uint32_t pitch = (uint32_t)(wn * NCH * 16), move_bytes = (uint32_t)(nslots * sizeof(uint2));
    const int k = ut / NCH, c = ut % NCH, slot = k < nwords ? (int)sitem[k] : 0;
    const uint2 e = k < nwords ? sslot[slot] : make_uint2(0u, 0u);
    const uint32_t valid = e.y;
    const int i = (int)(e.x >> 16), w = (int)(e.x & 0xffffu), need = valid ? needed(i) : INT_MAX;
    const bool odd = i & 1;
    const uint32_t move_at = (uint32_t)__cvta_generic_to_shared(smove + slot);
    const uint32_t above = (uint32_t)__cvta_generic_to_shared(valid ? sm + (((i - 1 - i0) * wn + w - wlo) * NCH + c) * 4 : pad + 8);
    const uint32_t here = valid ? above + pitch : above;
    // Exchange words: of row i those that its own, the row above's or the row below's candidates change, and the
    // word to the left (its last HO bit); and of every row its first element, whatever it holds (a scratch word
    // outside the window), so that two bands wait for each other or not at all, also where a gap in the domain leaves
    // one of them nothing to change.  Per lane, the same every time; ~0: none.
    const bool silent = band + 1 == a.silent_band_plus1;  // test hook: publishes nothing
    const uint32_t parity = (uint32_t)((a.last - a.first + 1) * a.xn * NCH * 4);
    uint32_t send_at[kGrMove], send_to[kGrMove], take_at[kGrMove], take_to[kGrMove];
    auto element = [&](int row, int q, uint32_t* local, uint32_t* global) {
      const int p = q & 3, cc = (q >> 2) % NCH, ww = a.xlo + (q >> 2) / NCH;
      int lo = INT_MAX, hi = -1;
      for (int r = row - 1; r <= row + 1; ++r) {
        int first = 0;
        const int n = row_words(r, &first);
        if (n) lo = min(lo, first - 1), hi = max(hi, first + n - 1);
      }
      if (row < a.first || row > a.last || row < i0 || row >= u1) return;
      const bool held = ww >= lo && ww <= hi && ww >= wlo && ww < wlo + wn;
      if (!held && q != 0) return;
      *local = (uint32_t)__cvta_generic_to_shared(held ? sm + (((row - i0) * wn + ww - wlo) * NCH + cc) * 4 + p : pad);
      *global = (uint32_t)((row - a.first) * a.xn * NCH * 4 + q);
    };
    const int per_row = a.xn * NCH * 4, own = r1 - r0, edge_rows = min(own, 2 * depth);
#pragma unroll
    for (int m = 0; m < kGrMove; ++m) {
      send_at[m] = take_at[m] = ~0u;
      send_to[m] = take_to[m] = 0u;
      const int x = ut + m * nupd, y = x / per_row, q = x - y * per_row;
      if (y < edge_rows && !silent) element(own <= 2 * depth || y < depth ? r0 + y : r1 - 2 * depth + y, q, &send_at[m], &send_to[m]);
      if (y < 2 * depth) element(y < depth ? r0 - depth + y : r1 + y - depth, q, &take_at[m], &take_to[m]);
    }
    auto exchange = [&](uint32_t period) {
      uint64_t* const buf = xbuf + (period & 1u) * parity;
      uint64_t v[kGrMove];
#pragma unroll
      for (int m = 0; m < kGrMove; ++m)
        if (send_at[m] != ~0u) gr_send(buf + send_to[m], period + 1u, cl_lds(send_at[m]));
#pragma unroll
      for (int m = 0; m < kGrMove; ++m)
        if (take_at[m] != ~0u) asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v[m]) : "l"(buf + take_to[m]) : "memory");
#pragma unroll
      for (int m = 0; m < kGrMove; ++m) {
        if (take_at[m] == ~0u) continue;
        uint32_t got = (uint32_t)v[m];
        if ((uint32_t)(v[m] >> 32) != period + 1u && !dead && !gr_recv(buf + take_to[m], period + 1u, got, a.max_spin, a.error, couple ? a.best : nullptr, attempt))
          dead = true;
        if (!dead) cl_sts(take_at[m], got);
      }
      asm volatile("bar.sync 1, %0;" ::"r"(nupd) : "memory");
    };
    __syncthreads();  // the first period's moves are drawn
    for (int q = 0; q < periods; ++q) {
      if (q > 0) exchange((uint32_t)q - 1u);
      const int len = min(depth, nruns - q * depth);
      uint32_t at = move_at + (uint32_t)((q & 1) * depth) * move_bytes;
      for (int r = 0; r < len; ++r, at += move_bytes) {
        const uint32_t t = s_colour[q & 1][r];
        if (need <= len - r) {
          const uint32_t off_u = t ? 0u : 4u, off_d = 4u - off_u;
          const uint2 move = cl_lds2(at);
          const uint2 ab = cl_lds2(above);
          const uint4 me = cl_lds4(here);
          const uint32_t west = cl_lds(here - 16u * NCH + 12u);
          const bool aligned = odd == (t != 0u);  // left HE, right HO of the same word
          const uint32_t U = t ? ab.x : ab.y, D = t ? me.y : me.x;
          const uint32_t lft = aligned ? me.z : __funnelshift_l(west, me.w, 1), rgt = aligned ? me.w : me.z;
          const uint32_t flip = ~(U ^ D) & ~(lft ^ rgt) & (U ^ lft) & valid;
          const uint32_t T = flip & ((U & ~move.x) | (~U & move.y));
          cl_sts(above + off_u, U ^ T);
          cl_sts(here + off_d, D ^ T);
          cl_sts(here + 8u, me.z ^ T);
          cl_xor(here + 12u, aligned ? T : T >> 1);
          cl_xor_if(here - 16u * NCH + 12u, aligned ? 0u : T << 31);
        }
        asm volatile("bar.sync 1, %0;" ::"r"(nupd) : "memory");
      }
      cl_cta_sync();
      if (couple && *static_cast<volatile int*>(&s_stop[q & 1])) return;
    }
    // The rows around its own as the other bands leave them; and no band writes back before the bands around it
    // have loaded.
    if (periods > 0) exchange((uint32_t)periods - 1u);
  } else {
    // ---- draw warps
    const int par = (int)((sslot[warp * KS].x >> 16) & 1u);
    auto gen_index = [&](int s, bool* v) -> int64_t {
      const uint2 e = sslot[warp * KS + s];
      *v = (e.y >> lane) & 1u;
      return (int64_t)((int)(e.x >> 16) - 1) * a.cols + (32 * (int)(e.x & 0xffffu) + lane - 1);
    };
    auto params_of = [&](int s, uint32_t& m1, uint32_t& m2, uint32_t& tm) {
      m1 = kTmtMat1;
      m2 = kTmtMat2;
      tm = kTmtTmat;
      if (kParams) {
        bool v;
        const int64_t g = gen_index(s, &v);
        const uint4 p = __ldg(&a.tmt_params[v ? g : 0]);
        m1 = p.x;
        m2 = p.y;
        tm = p.z;
      }
    };
    uint4 gen[kFast ? 1 : KS];
    uint32_t f_row[kFast ? KS / 4 : 1], f_quad[kFast ? KS / 4 : 1];
    int f_need[kFast ? KS / 4 : 1];  // runs left at which the group is first needed
    if constexpr (!kFast) {
#pragma unroll
      for (int s = 0; s < KS; ++s) {
        bool v;
        const int64_t g = gen_index(s, &v);
        gen[s] = make_uint4(0u, 0u, 0u, 0u);
        if (v && !couple) gen[s] = a.tmt[g];
      }
    } else {
#pragma unroll
      for (int g = 0; g < KS / 4; ++g) {
        const uint2 e = sslot[warp * KS + 4 * g + (lane >> 3)];
        f_row[g] = e.x >> 16;
        f_quad[g] = (e.x & 0xffffu) * 8u + (uint32_t)(lane & 7);
        f_need[g] = __reduce_min_sync(~0u, e.y ? needed((int)f_row[g]) : INT_MAX);
      }
    }
    // A period's runs, from run j0 on.
    auto draw_period = [&](int q) {
      const int j0 = q * depth, len = min(depth, nruns - j0);
      uint2* const out = smove + (q & 1) * depth * nslots;
      if constexpr (!kFast) {
        for (int r = 0; r < len; ++r) {
          const uint32_t run = run_at(j0 + r);
          if (tid == 0) s_colour[q & 1][r] = run >> 31;
          if (NCH == 2 && ((run >> 30) & 1u)) {  // InitTinyMT for an epoch (tinymt.clh:183-203, as k_tmt_seed)
            const uint32_t seed = __ldg(&a.epoch_seeds[epoch++]);
#pragma unroll
            for (int s = 0; s < KS; ++s) {
              bool v;
              const int64_t g = gen_index(s, &v);
              uint32_t m1, m2, tm;
              params_of(s, m1, m2, tm);
              if (v) gen[s] = tmt_seed(seed + (uint32_t)g, m1, m2, tm);
            }
          }
          cl_moves_tmt<KS>(gen, srule[par | ((int)(run >> 31) << 1)], (int)(run & 0x3fffffffu),
                           out + r * nslots + warp * KS, params_of);
        }
      } else {
        // two runs at a time: a Philox block is a chain of its own
        for (int r = 0; r < len; r += 2) {
          const uint32_t c0 = run_at(j0 + r) >> 31, c1 = c0 ^ 1u;
          if (tid == 0) {
            s_colour[q & 1][r] = c0;
            if (r + 1 < len) s_colour[q & 1][r + 1] = c1;
          }
          const uint4 rl0 = srule[par | (int)(c0 << 1)], rl1 = srule[par | (int)(c1 << 1)];
#pragma unroll
          for (int g = 0; g < KS / 4; ++g) {
            if (f_need[g] > len - r) continue;
            uint2* const to = out + r * nslots + warp * KS + 4 * g;
            if (f_need[g] <= len - r - 1) {
              cl_moves_fast2(a.seed, a.stream, h0 + j0 + r, f_row[g], f_quad[g], rl0, rl1, to, to + nslots);
            } else {
              cl_moves_fast(a.seed, a.stream, h0 + j0 + r, f_row[g], f_quad[g], rl0, to);
            }
          }
        }
      }
    };
    if (periods > 0) draw_period(0);
    __syncthreads();
    for (int q = 0; q < periods; ++q) {
      if (couple && tid == 0) s_stop[q & 1] = *static_cast<volatile int*>(a.best) < attempt;
      if (q + 1 < periods) draw_period(q + 1);
      cl_cta_sync();
      if (couple && *static_cast<volatile int*>(&s_stop[q & 1])) return;
    }
    __syncthreads();  // the bands around have loaded (the last exchange)
    if constexpr (!kFast) {
#pragma unroll
      for (int s = 0; s < KS; ++s) {
        bool v;
        const int64_t g = gen_index(s, &v);
        const int i = (int)(sslot[warp * KS + s].x >> 16);
        if (v && !couple && i >= r0 && i < r1) a.tmt[g] = gen[s];
      }
    }
  }
  if (warp >= ndraw) __syncthreads();
  const bool any_dead = __syncthreads_or(dead ? 1 : 0);
  if (couple) {  // the last band to finish knows whether any differs (a band that left for a smaller attempt never counts)
    uint32_t differ = 0u;
    for (int x = tid; x < (r1 - r0) * wn; x += (int)blockDim.x) {
      const uint4* w = reinterpret_cast<const uint4*>(sm) + ((r0 - i0) * wn + x) * 2;
      differ |= (w[0].x ^ w[1].x) | (w[0].y ^ w[1].y) | (w[0].z ^ w[1].z) | (w[0].w ^ w[1].w);
    }
    const int any = __syncthreads_or(differ != 0u || any_dead ? 1 : 0);
    if (tid == 0) {
      if (any) atomicAdd(&a.team[team].x, 1);
      __threadfence();
      if (atomicAdd(&a.team[team].y, 1) == a.bands - 1 && atomicAdd(&a.team[team].x, 0) == 0) atomicMin(a.best, attempt);
    }
  } else if (any_dead && tid == 0) {
    atomicExch(a.error, 1);
  }
  cl_store_window<NCH>(sm + (r0 - 1 - i0) * 4 * wn * NCH, a.base + team * a.team_stride, a.chain_stride, a.colour_stride, a.P, a.cols, r0 - 1, r1 - r0 + 1,
                       wlo, wn);
}

template <int NCH, int kMode, int UI>
void* gr_kernel_ks(int ks) {
  if constexpr (kMode == kClFast) {
    switch (ks) {
      case 4: return (void*)k_grid<NCH, kMode, 4, UI>;
      case 8: return (void*)k_grid<NCH, kMode, 8, UI>;
      case 12: return (void*)k_grid<NCH, kMode, 12, UI>;
      default: return (void*)k_grid<NCH, kMode, 16, UI>;
    }
  } else {
    switch (ks) {
      case 1: return (void*)k_grid<NCH, kMode, 1, UI>;
      case 2: return (void*)k_grid<NCH, kMode, 2, UI>;
      case 4: return (void*)k_grid<NCH, kMode, 4, UI>;
      case 8: return (void*)k_grid<NCH, kMode, 8, UI>;
      default: return (void*)k_grid<NCH, kMode, 16, UI>;
    }
  }
}
template <int NCH, int UI>
void* gr_kernel_mode(int mode, int ks) {
  return mode == kClFast ? gr_kernel_ks<NCH, kClFast, UI>(ks)
                         : (mode == kClTmt ? gr_kernel_ks<NCH, kClTmt, UI>(ks) : gr_kernel_ks<NCH, kClTmtParams, UI>(ks));
}
void* gr_kernel(int nch, int mode, int ks, int ui) {
  if (nch == 1) return ui == 1 ? gr_kernel_mode<1, 1>(mode, ks) : gr_kernel_mode<1, 4>(mode, ks);
  return ui == 1 ? gr_kernel_mode<2, 1>(mode, ks) : gr_kernel_mode<2, 4>(mode, ks);
}

template <int NCH>
void* gr_deep_kernel(int mode, int ks) {
  if (mode == kClFast) return ks == 4 ? (void*)k_deep<NCH, kClFast, 4> : (void*)k_deep<NCH, kClFast, 8>;
  if (mode == kClTmt)
    return ks == 1 ? (void*)k_deep<NCH, kClTmt, 1> : (ks == 2 ? (void*)k_deep<NCH, kClTmt, 2> : (void*)k_deep<NCH, kClTmt, 4>);
  return ks == 1 ? (void*)k_deep<NCH, kClTmtParams, 1>
                 : (ks == 2 ? (void*)k_deep<NCH, kClTmtParams, 2> : (void*)k_deep<NCH, kClTmtParams, 4>);
}

#define RT_CUDA_G(expr)                                                                 \
  do {                                                                                  \
    cudaError_t _e = (expr);                                                            \
    if (_e != cudaSuccess)                                                              \
      return fail(RT_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(_e));     \
  } while (0)

}  // namespace

void GrPlan::build(const std::vector<int>& lo, const std::vector<int>& hi, int N, int nch, bool fast, int bands_max) {
  ok = false;
  why.clear();
  words = draw_cells = 0;
  const int rows = N - 2;
  std::vector<int> cnt(N + 1, 0);
  int w0 = INT_MAX, w1 = -1, first = -1, last = -1;
  for (int i = 1; i <= rows; ++i) {
    if (lo[i] < 0) continue;
    cnt[i] = hi[i] / 32 - lo[i] / 32 + 1;
    words += cnt[i];
    draw_cells += hi[i] - lo[i] + 1;
    w0 = std::min(w0, lo[i] / 32);
    w1 = std::max(w1, hi[i] / 32);
    if (first < 0) first = i;
    last = i;
  }
  if (words == 0) {
    why = "no flip candidates";
    return;
  }
  if (N > 0xffff) {
    why = "tiling too large for the slot descriptors";
    return;
  }
  // The vertices around the candidates change too: a row above and below, a word left and right
  // (and one more word of margin for the edges of those).
  first = std::max(1, first - 1);
  last = std::min(rows, last + 1);
  xlo = w0;
  xn = w1 - w0 + 1;
  bands = std::min(std::min(bands_max, kGrMaxBands), last - first + 1);
  // Contiguous bands, the largest (in words) as small as possible.
  auto pack = [&](int64_t cap) -> bool {
    int k = 0;
    int64_t in = 0;
    row_start[0] = first;
    for (int i = first; i <= last; ++i) {
      if (in > 0 && in + cnt[i] > cap) {
        if (++k >= bands) return false;
        row_start[k] = i;
        in = 0;
      }
      in += cnt[i];
    }
    for (int q = k + 1; q <= bands; ++q) row_start[q] = last + 1;
    return true;
  };
  int64_t a = 1, b = words;
  for (int i = first; i <= last; ++i) a = std::max<int64_t>(a, cnt[i]);
  while (a < b) {
    const int64_t mid = (a + b) / 2;
    if (pack(mid)) b = mid;
    else a = mid + 1;
  }
  pack(a);
  while (bands > 1 && row_start[bands - 1] > last) --bands;
  // A band's window: the words of its rows and of the neighbours' facing rows, with the margins of
  // the vertices around the candidates.
  size_t window_max = 0;
  int64_t words_max = 0;
  std::vector<int64_t> par((size_t)bands * 2, 0);
  for (int k = 0; k < bands; ++k) {
    int a0 = INT_MAX, a1 = -1;
    for (int i = row_start[k] - 1; i <= row_start[k + 1]; ++i)
      if (i >= 1 && i <= rows && lo[i] >= 0) {
        a0 = std::min(a0, lo[i] / 32);
        a1 = std::max(a1, hi[i] / 32);
      }
    if (a1 < 0) a0 = a1 = w0;
    windows[2 * k] = a0 - 2;
    windows[2 * k + 1] = a1 - a0 + 5;
    window_max = std::max(window_max, (size_t)(row_start[k + 1] - row_start[k] + 1) * windows[2 * k + 1]);
    for (int i = row_start[k]; i < row_start[k + 1]; ++i) par[2 * k + (i & 1)] += cnt[i];
    words_max = std::max(words_max, par[2 * k] + par[2 * k + 1]);
  }
  // Words per draw warp and items per update lane: the fewest whose warps fit.
  const int64_t items = words_max * nch;
  slots = 0;
  for (int ks : {1, 2, 4, 8, 12, 16}) {
    if (fast ? ks < 4 : ks == 12) continue;
    int64_t draw = 1;
    for (int k = 0; k < bands; ++k) draw = std::max<int64_t>(draw, (par[2 * k] + ks - 1) / ks + (par[2 * k + 1] + ks - 1) / ks);
    for (int ui : {1, 4}) {
      const int64_t update = std::max<int64_t>(1, (items + 32 * ui - 1) / (32 * ui));
      if (draw + update > gr_max_threads(fast, ks) / 32) continue;
      if (gr_splits(fast, ks)) {  // whole warpgroups
        if (draw > 16 || update > 4 || ui != 4) continue;
        draw = 16;
      }
      slots = ks;
      per_lane = ui;
      draw_warps = (int)draw;
      update_warps = gr_splits(fast, ks) ? 4 : (int)update;
      break;
    }
    if (slots) break;
  }
  if (!slots) {
    why = "too many words per band for register-resident generators";
    return;
  }
  smem_bytes = (window_max * 4 * nch + kClPad) * sizeof(uint32_t) +
               3 * (size_t)draw_warps * slots * sizeof(uint2) + (size_t)words_max * sizeof(uint16_t) + 16;
  if (smem_bytes > 200 * 1024) {
    why = "band window exceeds shared memory";
    return;
  }
  ok = true;
}

// The same domain with an exchange every `runs` runs; false where no form of k_deep holds it.
bool GrPlan::build_deep(const std::vector<int>& lo, const std::vector<int>& hi, int N, int nch, bool fast, int bands_max, int runs) {
  const int rows = N - 2;
  std::vector<int> cnt(N + 1, 0);
  int w0 = INT_MAX, w1 = -1;
  first = last = -1;
  for (int i = 1; i <= rows; ++i) {
    if (lo[i] < 0) continue;
    cnt[i] = hi[i] / 32 - lo[i] / 32 + 1;
    w0 = std::min(w0, lo[i] / 32);
    w1 = std::max(w1, hi[i] / 32);
    if (first < 0) first = i;
    last = i;
  }
  first = std::max(1, first - 1);
  last = std::min(rows, last + 1);
  xlo = w0 - 1;
  xn = w1 - w0 + 2;
  const int total = last - first + 1;
  bands = std::min(std::min(bands_max, kGrMaxBands), total);
  for (int k = 0; k <= bands; ++k) row_start[k] = first + (int)((int64_t)total * k / bands);
  size_t window_max = 0;
  int64_t words_max = 0, send_max = 0;
  std::vector<int64_t> par((size_t)bands * 2, 0);
  for (int k = 0; k < bands; ++k) {
    const int r0 = row_start[k], r1 = row_start[k + 1], u0 = std::max(r0 - (runs - 1), first), u1 = std::min(r1 + runs, last + 1);
    int a0 = INT_MAX, a1 = -1;
    for (int i = u0 - 1; i <= u1; ++i)
      if (i >= 1 && i <= rows && lo[i] >= 0) {
        a0 = std::min(a0, lo[i] / 32);
        a1 = std::max(a1, hi[i] / 32);
      }
    if (a1 < 0) a0 = a1 = w0;
    windows[2 * k] = a0 - 2;
    windows[2 * k + 1] = a1 - a0 + 5;
    window_max = std::max(window_max, (size_t)(u1 - u0 + 1) * windows[2 * k + 1]);
    for (int i = u0; i < u1; ++i) par[2 * k + (i & 1)] += cnt[i];
    words_max = std::max(words_max, par[2 * k] + par[2 * k + 1]);
    send_max = std::max<int64_t>(send_max, std::max(std::min(r1 - r0, 2 * runs), 2 * runs) * (int64_t)xn * nch * 4);
  }
  if (words_max * nch > 320) return false;
  update_warps = (int)std::max<int64_t>(1, (std::max(words_max * nch, (send_max + kGrMove - 1) / kGrMove) + 31) / 32);
  per_lane = 1;
  slots = 0;
  for (int ks : {1, 2, 4, 8}) {
    if (fast ? ks < 4 : ks > 4) continue;
    int64_t draw = 1;
    for (int k = 0; k < bands; ++k) draw = std::max<int64_t>(draw, (par[2 * k] + ks - 1) / ks + (par[2 * k + 1] + ks - 1) / ks);
    if (draw + update_warps > gr_max_threads(fast, ks) / 32) continue;
    slots = ks;
    draw_warps = (int)draw;
    break;
  }
  if (!slots) return false;
  smem_bytes = (window_max * 4 * nch + kClPad) * sizeof(uint32_t) +
               (1 + 2 * (size_t)runs) * (size_t)draw_warps * slots * sizeof(uint2) + (size_t)words_max * sizeof(uint16_t) + 16;
  if (smem_bytes > 200 * 1024) return false;
  depth = runs;
  return true;
}

GridEngine::~GridEngine() {
  for (void* p : {(void*)d_rows, (void*)d_xbuf, (void*)d_runs, (void*)d_team, (void*)d_teams, (void*)d_xteams}) dev_free(p, stream);
}

// Runs between exchanges: more of them share one exchange, but a band of rho rows draws for rho + 2 d - 1.
// Measured (us per half-sweep, diamonds, one chain; d = 1 is k_grid):
//   TinyMT  order 16: d = 4 0.19, 6 0.17, 8 0.19    40: 4 0.22, 6 0.23, 8 0.25    64: 4 0.25, 6 0.24, 8 0.28
//           100: 1 0.51, 2 0.41, 3 0.35, 4 0.30, 6 0.37    200: 1 0.50, 2 0.38, 3 0.41    250: 1 0.54, 2 0.47, 3 0.57
//           300: 1 0.57, 2 0.60
//   fast    order 24: d = 4 0.35, 8 0.29, 12 0.22    64: 4 0.45, 8 0.31, 12 0.29    100: 1 0.99, 4 0.42, 8 0.35
//           150: 4 0.45, 6 0.37, 8 0.37, 12 0.48    200: 1 1.06, 3 0.52, 4 0.45, 6 0.44, 8 0.50
//           300: 1 1.08, 3 0.57, 4 0.56, 6 0.60    400: 2 0.72, 3 0.76    512: 2 0.95, 3 1.23
// (rows of 1, 2, 3, 4, 5, 7, 8, 10, 13 and 17 words).  Wider rows than the last ones: d = 1.
// The same lines serve two chains on a quarter of the SMs (couplings; ms of a call whose longest attempt is 8192
// half-sweeps):
//   TinyMT  order 16: d = 5 4.10, 6 3.91, 7 3.77    40: 4 5.18, 6 5.42, 8 6.37    64: 3 6.42, 4 5.89, 5 5.81
//           100: 2 7.92, 3 7.50, 4 7.96    128: 1 12.40, 2 8.70, 3 9.05    160: 1 12.84, 2 11.86
//   fast    order 24: d = 8 4.52, 12 4.26    64: 8 5.37, 11 5.13, 12 5.19    100: 6 6.86, 8 6.60, 10 7.11
//           128: 7 7.33, 8 7.69    160: 4 8.84, 5 9.05, 6 10.10    200: 2 13.98, 4 12.63
// within a tenth of the best for diamonds.  Few rows of many words are further off: 20 x 400 in TinyMT mode 2 8.65 and
// one cluster 6.25, in fast mode 6 7.26 and 7, the choice, 9.63.
static int gr_depth(const GrPlan& p, bool fast, int bands) {
  const int rows = p.row_start[p.bands] - p.row_start[0], used = std::min(bands, rows), rho = (rows + used - 1) / used;
  const auto words = [&](int d) { return (rho + 2 * d - 1) * p.xn; };
  if (fast) {
    for (int d = 12; d > 2; --d)
      if (words(d) <= (d > 8 ? 75 : 110)) return d;
    return words(2) <= 175 ? 2 : 1;
  }
  for (int d = 6; d > 2; --d)
    if (words(d) <= 36) return d;
  return words(2) <= 56 ? 2 : 1;
}

rt_status GridEngine::prepare(DmSampler& s) {
  ready = false;
  plan.ok = false;
  nch = s.active;
  stream = s.stream;
  int dev = 0, coop = 0;
  RT_CUDA_G(cudaGetDevice(&dev));
  RT_CUDA_G(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  RT_CUDA_G(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  bands_max = s.eff_bands > 0 ? std::min(s.eff_bands, sms) : sms;
  const bool fast = s.opts.rng_mode == RT_RNG_FAST;
  if (s.opts.rng_mode == RT_RNG_MTGP || (nch != 1 && nch != 2)) {
    plan.why = "TinyMT or fast mode with 1 or 2 swept chains";
    return RT_OK;
  }
  if (s.border_candidates) {
    plan.why = "a flip candidate borders the cells the reference never rebuilds";
    return RT_OK;
  }
  for (int c = 0; c < 4; ++c) {  // the kernel tests the tempered word against interval ends x 2^9
    const uint64_t lo_dn = s.rule.lo_dn[c], w_dn = s.rule.w_dn[c];
    if (fast ? s.rule.lo_up[c] != 0
             : s.rule.lo_up[c] != 0 || s.rule.w_up[c] >= (1u << 23) || w_dn >= (1u << 23) || lo_dn + w_dn > (1u << 23)) {
      plan.why = "rule intervals outside the kernel's compare range";
      return RT_OK;
    }
  }
  if (!coop) {
    plan.why = "device lacks cooperative launch";
    return RT_OK;
  }
  const int deep_bands = s.couple ? std::max(1, sms / kGrTeams) : bands_max;
  plan.depth = 1;
  plan.build(s.cand_lo, s.cand_hi, s.N, nch, fast, bands_max);
  if (!plan.ok) return RT_OK;
  const int mode = fast ? kClFast : (s.tmt_params ? kClTmtParams : kClTmt);
  if (const int runs = gr_depth(plan, fast, deep_bands); runs > 1) {
    GrPlan deep = plan;
    if (deep.build_deep(s.cand_lo, s.cand_hi, s.N, nch, fast, deep_bands, runs)) plan = deep;
  }
  kernel = plan.depth > 1 ? (nch == 1 ? gr_deep_kernel<1>(mode, plan.slots) : gr_deep_kernel<2>(mode, plan.slots))
                          : gr_kernel(nch, mode, plan.slots, plan.per_lane);
  RT_CUDA_G(dev_allow_smem(kernel, plan.smem_bytes));
  int per_sm = 0;
  RT_CUDA_G(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, plan.threads(), plan.smem_bytes));
  if ((int64_t)per_sm * sms < plan.bands * (s.couple && plan.depth > 1 ? kGrTeams : 1)) {
    plan.ok = false;
    plan.why = "bands cannot all be resident";
    return RT_OK;
  }
  if (!d_rows) {
    if (rt_status st = dev_alloc(&d_rows, (3 * kGrMaxBands + 2) * sizeof(int), stream)) return st;
    xbuf_bytes = plan.depth > 1 ? (size_t)2 * (plan.last - plan.first + 1) * plan.xn * nch * 4 * sizeof(uint64_t)
                                : (size_t)2 * plan.bands * 2 * plan.xn * nch * sizeof(uint64_t);
    if (rt_status st = dev_alloc(&d_xbuf, xbuf_bytes, stream)) return st;
  }
  RT_CUDA_G(cudaMemcpyAsync(d_rows, plan.row_start, sizeof plan.row_start, cudaMemcpyHostToDevice, stream));
  RT_CUDA_G(cudaMemcpyAsync(d_rows + kGrMaxBands + 1, plan.windows, sizeof plan.windows, cudaMemcpyHostToDevice, stream));
  ready = true;
  return RT_OK;
}

namespace {

GrArgs gr_args(const GridEngine& e, DmSampler& s) {
  GrArgs a{};
  a.base = s.base;
  a.N = s.N;
  a.P = s.P;
  a.cols = s.N / 2 - 2;
  a.bands = e.plan.bands;
  a.draw_warps = e.plan.draw_warps;
  a.chain_stride = s.chain_stride;
  a.colour_stride = s.colour_stride;
  a.tmt = s.tmt;
  a.tmt_params = s.tmt_params;
  a.cand = s.d_cand;
  a.row_start = e.d_rows;
  a.windows = e.d_rows + kGrMaxBands + 1;
  a.xlo = e.plan.xlo;
  a.xn = e.plan.xn;
  a.depth = e.plan.depth;
  a.first = e.plan.first;
  a.last = e.plan.last;
  a.rule = s.rule;
  a.stream = s.opts.fast_stream;
  a.xbuf = e.d_xbuf;
  a.error = e.d_rows + 3 * kGrMaxBands + 1;
  a.max_spin = s.test_max_spin > 0 ? s.test_max_spin : test_silence().spin(1L << 22);
  a.silent_band_plus1 = s.test_silent_band >= 0 ? s.test_silent_band + 1 : test_silence().next_plus1();
  return a;
}

}  // namespace

rt_status GridEngine::cftp(DmSampler& s, int a0, int n, const std::vector<std::vector<RunEngine::Epoch>>& epochs,
                           int64_t first_sweeps, uint64_t fast_seed, int* attempts_run, bool* coalesced) {
  const bool fast = s.opts.rng_mode == RT_RNG_FAST;
  if (plan.depth < 2 || n < 1 || n > kGrTeams || nch != 2) return fail(RT_ERR_INVALID_ARGUMENT, "grid cftp: 1..4 attempts, 2 chains");
  if (rt_status st = check_error(s)) return st;
  GrArgs a = gr_args(*this, s);
  a.couple = 1;
  a.attempt0 = a0;
  a.first_sweeps = first_sweeps;
  a.seed = fast_seed;
  a.start = s.base + 2 * s.chain_stride;
  a.team_stride = 2 * s.chain_stride;
  a.xteam = xbuf_bytes / sizeof(uint64_t);
  constexpr size_t kWords = 4 + 2 * kGrTeams;  // {best, error, -, -, team}
  if (!d_team) {
    if (rt_status st = dev_alloc(&d_team, kWords * sizeof(int), stream)) return st;
    if (rt_status st = dev_alloc(&d_teams, kGrTeams * a.team_stride, stream)) return st;
    if (rt_status st = dev_alloc(&d_xteams, kGrTeams * xbuf_bytes, stream)) return st;
  }
  a.base = d_teams;
  a.xbuf = d_xteams;
  a.best = d_team;
  a.error = d_team + 1;
  a.team = reinterpret_cast<int2*>(d_team + 4);
  std::vector<uint32_t> runs, seeds;
  std::vector<int4> desc;
  if (!fast) {
    for (int k = 0; k < n; ++k) {
      int4 d = make_int4((int)runs.size(), 0, (int)seeds.size(), 0);
      for (const RunEngine::Epoch& e : epochs[(size_t)k]) {
        if (!e.colours || e.colours->empty()) continue;
        seeds.push_back(e.seed);
        append_runs(e.colours->data(), (int64_t)e.colours->size(), true, &runs);
      }
      d.y = (int)runs.size() - d.x;
      desc.push_back(d);
    }
    // one block: the descriptors, the epoch seeds, the runs
    const size_t at_seeds = desc.size() * sizeof(int4), at_runs = at_seeds + seeds.size() * sizeof(uint32_t);
    const int64_t words = (int64_t)(at_runs / sizeof(uint32_t) + runs.size());
    if (runs_cap < words) {
      dev_free(d_runs, s.stream);
      d_runs = nullptr;
      runs_cap = 0;
      if (rt_status st = dev_alloc(&d_runs, (size_t)words * sizeof(uint32_t), s.stream)) return st;
      runs_cap = words;
    }
    std::vector<uint32_t> block((size_t)words);
    std::memcpy(block.data(), desc.data(), at_seeds);
    std::copy(seeds.begin(), seeds.end(), block.begin() + (long)(at_seeds / sizeof(uint32_t)));
    std::copy(runs.begin(), runs.end(), block.begin() + (long)(at_runs / sizeof(uint32_t)));
    RT_CUDA_G(cudaMemcpyAsync(d_runs, block.data(), block.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, s.stream));
    a.attempt_desc = reinterpret_cast<const int4*>(d_runs);
    a.epoch_seeds = d_runs + at_seeds / sizeof(uint32_t);
    a.runs = d_runs + at_runs / sizeof(uint32_t);
  }
  for (int k = 0; k < n; ++k)  // the cells that no attempt writes
    RT_CUDA_G(cudaMemcpyAsync(d_teams + k * a.team_stride, a.start, a.team_stride, cudaMemcpyDeviceToDevice, s.stream));
  RT_CUDA_G(cudaMemsetAsync(d_team, 0, kWords * sizeof(int), s.stream));
  RT_CUDA_G(cudaMemsetAsync(d_team, 0x7f, sizeof(int), s.stream));  // no attempt yet
  RT_CUDA_G(cudaMemsetAsync(d_xteams, 0, n * xbuf_bytes, s.stream));  // no stale tags
  void* args[] = {&a};
  RT_CUDA_G(cudaLaunchCooperativeKernel(kernel, dim3((unsigned)plan.bands, (unsigned)n), dim3((unsigned)plan.threads()), args,
                                        plan.smem_bytes, s.stream));
  s.launches++;
  int res[2] = {0, 0};
  RT_CUDA_G(cudaMemcpyAsync(res, d_team, sizeof res, cudaMemcpyDeviceToHost, s.stream));
  RT_CUDA_G(cudaStreamSynchronize(s.stream));
  if (res[1]) return fail(RT_ERR_TIMEOUT, "grid sweep: a band gave up waiting (a neighbour's boundary words never came)");
  *coalesced = res[0] < a0 + n;
  *attempts_run = *coalesced ? res[0] - a0 + 1 : n;
  RT_CUDA_G(cudaMemcpyAsync(s.base, d_teams + (*attempts_run - 1) * a.team_stride, a.team_stride, cudaMemcpyDeviceToDevice,
                            s.stream));
  return RT_OK;
}

rt_status GridEngine::launch(DmSampler& s, const uint8_t* colours_host, int64_t steps, uint64_t fast_seed, int64_t h0) {
  const int64_t chunk_max = 65536;  // bounds one launch to a fraction of a second
  std::vector<uint32_t> runs;
  for (int64_t done = 0; done < steps;) {
    const int64_t n = std::min(chunk_max, steps - done);
    GrArgs a = gr_args(*this, s);
    a.seed = fast_seed;
    a.h0 = h0 + done;
    a.nruns = (int)n;
    if (s.opts.rng_mode != RT_RNG_FAST) {
      runs.clear();
      append_runs(colours_host + done, n, false, &runs);
      if (runs_cap < (int64_t)runs.size()) {
        dev_free(d_runs, s.stream);
        d_runs = nullptr;
        runs_cap = 0;
        if (rt_status st = dev_alloc(&d_runs, runs.size() * sizeof(uint32_t), s.stream)) return st;
        runs_cap = (int64_t)runs.size();
      }
      RT_CUDA_G(cudaMemcpyAsync(d_runs, runs.data(), runs.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, s.stream));
      a.runs = d_runs;
      a.nruns = (int)runs.size();
    }
    if (!pending_error_check) RT_CUDA_G(cudaMemsetAsync(a.error, 0, sizeof(int), s.stream));
    RT_CUDA_G(cudaMemsetAsync(d_xbuf, 0, xbuf_bytes, s.stream));  // no stale tags
    void* args[] = {&a};
    RT_CUDA_G(cudaLaunchCooperativeKernel(kernel, dim3((unsigned)plan.bands), dim3((unsigned)plan.threads()), args,
                                          plan.smem_bytes, s.stream));
    s.launches++;
    pending_error_check = true;
    done += n;
  }
  return RT_OK;
}

rt_status GridEngine::check_error(DmSampler& s) {
  if (!pending_error_check) return RT_OK;
  int err = 0;
  RT_CUDA_G(cudaMemcpyAsync(&err, d_rows + 3 * kGrMaxBands + 1, sizeof(int), cudaMemcpyDeviceToHost, s.stream));
  RT_CUDA_G(cudaStreamSynchronize(s.stream));
  pending_error_check = false;
  if (err) return fail(RT_ERR_TIMEOUT, "grid sweep: a band gave up waiting (a neighbour's boundary words never came)");
  return RT_OK;
}

}  // namespace rt
