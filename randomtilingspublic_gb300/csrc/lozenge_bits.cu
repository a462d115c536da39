// Bit-plane engine of the lozenge sweep: one bit per lattice edge in shared memory.
//
// The reference keeps one byte per vertex (its six edge bits), rotates one colour per step
// (25 <-> 38, lozengekernel.cl:74-105) and rebuilds three bits of each vertex of the two others
// (:107-125).  Every edge joins vertices of two colours, so the edges alone are the state: vertex
// (i, j) owns E (to (i, j+1)), NE (to (i-1, j+1)) and N (to (i-1, j)); its six bits are 8 = E(i, j),
// 2 = NE(i, j), 1 = N(i, j), 4 = E(i, j-1), 16 = NE(i+1, j-1), 32 = N(i+1, j).  It can flip when
// {E, N, NE(i+1, j-1)} are equal, the other three their complement; a flip toggles all six, and no
// two vertices of a colour share an edge: there is no colour to rebuild.
//
// Planes: row i, column residue q = j mod 3, bit k of word w for slot m = 32 w + k (j = 3 m + q): nine
// words a row and word.  Colour r sits at q = (i + r) mod 3 in row i, so a vertex's planes are words
// of its own row and the next, shifted by one slot only where q = 0 looks at column j - 1.
//
// A band (CTA) owns rows [r0, r1) and also holds NE and N of row r1.  After each run (consecutive
// steps of one colour) the first and last rows' toggles go to the neighbour as one word per 32 slots
// and chain, and the facing row's lanes apply them before they read.  Bands are one CTA, the CTAs of
// one cluster (st.async into the neighbour's shared memory, counted by an mbarrier) or one CTA per
// SM (64-bit words tagged with the run through L2; cooperative launch).  Every wait is bounded.
//
// Draws do not depend on the state: warps of their own make them, a run ahead, and compose a run's
// steps into one pair of move words per 32 slots (as domino_cluster.cu).
//
// Coupling from the past where one CTA holds the chains: four CTAs run attempts side by side, as in
// domino_cluster.cu (exact sample of the hexagon of side 20 in fast mode: 7.3 -> 5.9 ms, and 4.0 with draws a period ahead).
//
// What bounds it: the exchange of each run, 0.5 us in a cluster and 0.85 us through L2.  The byte kernel
// (lozenge_resident.cu) spent its step on the rotation and rebuild of bytes: hexagon 512 0.73 us a step
// (TinyMT; before 2.20) and 0.91 us (fast mode; 2.14), hexagon 20 0.36 (1.39) and 0.27 (1.36).  It
// stays for inputs whose edges disagree or whose candidates
// border vertices that the reference never rebuilds, and for sizes without a plan here.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <string>
#include <vector>

#include "lozenge_bits.h"
#include "rng.cuh"

namespace rt {

namespace {

enum : int { kLbTmt = 0, kLbTmtParams = 1, kLbFast = 2 };
constexpr int lb_max_threads(int ks, bool fast) { return !fast && ks > 4 ? 640 : 1024; }

struct LbArgs {
  uint8_t* base;
  size_t colour_stride, chain_stride;
  int N, M, P, bands, draw_warps;
  const int* row_start;
  const int* cand;
  int wlo, wn, w0, words;
  uint32_t lo_up, w_up, lo_dn, w_dn;  // TinyMT: times 2^9, tested on the tempered word
  uint4* tmt;
  const uint4* tmt_params;
  const uint32_t* runs;  // TinyMT: (colour << 30) | (epoch start << 29) | length
  int nruns;             // fast mode: steps
  uint64_t seed;
  uint32_t stream;
  int64_t h0;
  uint64_t* xbuf;  // [2 parities][band][to above, to below][word][chain]
  int* error;
  long max_spin;
  int silent_plus1;  // test hook: this band, less one, publishes nothing
  // Coupling from the past (attempts > 0, two chains, kLbOne): CTA `team` runs attempts team, team + teams, ...
  // from the chains at start, into chains of its own at base + team * team_stride.
  int attempts;
  int64_t first_sweeps;  // fast mode: attempt k runs 3 first_sweeps << k steps up to step 0
  const uint8_t* start;
  size_t team_stride;
  int* best;                    // smallest attempt that coalesced
  const int4* attempt_desc;     // TinyMT: {first run, runs, first epoch seed, 0}
  const uint32_t* epoch_seeds;  // a run that starts an epoch (bit 29) seeds the generators from the next
};

__device__ __forceinline__ uint32_t lb_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t lb_remote(const void* local, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(lb_addr(local)), "r"(rank));
  return r;
}
__device__ __forceinline__ void lb_send_if(bool on, uint32_t addr, uint32_t v, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t"
      "@p st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.u32 [%0], %1, [%2];\n\t}" ::"r"(addr),
      "r"(v), "r"(bar), "r"((uint32_t)on)
      : "memory");
}
__device__ __forceinline__ void lb_expect_if(bool on, uint32_t bar, uint32_t bytes) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t"
      "@p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(bar),
      "r"(bytes), "r"((uint32_t)on)
      : "memory");
}
__device__ __forceinline__ bool lb_bar_wait(uint32_t addr, uint32_t parity, long max_spin) {
  for (long it = 0; it <= max_spin; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ uint32_t lb_lds(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lb_lds2(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void lb_sts(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void lb_xor_if(uint32_t a, uint32_t v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p red.shared.xor.b32 [%0], %1;\n\t}" ::"r"(a), "r"(v)
               : "memory");
}
__device__ __forceinline__ void lb_cta_sync() { asm volatile("barrier.sync 0;" ::: "memory"); }

constexpr int kLbWord = 12;  // words per (row, word, chain): E0-2, NE0-2, N0-2, three of padding
constexpr int kLbPad = 3 * kLbWord * 2;
// Runs that the draw warps are ahead: one, but a period in one CTA in fast mode, where a run is one step of one Philox
// block's latency: there two blocks go side by side, and only the update warps meet after every step (hexagon 20:
// 0.35 -> 0.27 us a step, exact sample 5.9 -> 4.0 ms; hexagon 8: 0.15).
constexpr int lb_ahead(bool fast, int form) { return fast && form == kLbOne ? 8 : 1; }

// KS: words per draw warp.
template <int NCH, int kMode, int KS, int kForm>
__global__ void __launch_bounds__(lb_max_threads(KS, kMode == kLbFast), 1) k_lz_bits(const __grid_constant__ LbArgs a) {
  extern __shared__ __align__(16) uint32_t lsm[];
  __shared__ __align__(8) uint64_t s_bar[2][2];  // [from above, from below][run parity]
  __shared__ uint32_t s_colour[2];
  __shared__ int s_failed;
  __shared__ int s_stop;  // a smaller attempt coalesced
  constexpr bool kFast = kMode == kLbFast, kParams = kMode == kLbTmtParams;
  constexpr int kAhead = lb_ahead(kFast, kForm);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = (int)(blockDim.x >> 5);
  const int ndraw = a.draw_warps, nslots = ndraw * KS, band = kForm == kLbOne ? 0 : (int)blockIdx.x;
  const bool cftp = kForm == kLbOne && NCH == 2 && a.attempts > 0;
  uint8_t* const base = a.base + (cftp ? blockIdx.x * a.team_stride : 0);
  const int r0 = a.row_start[band], r1 = a.row_start[band + 1], R = r1 - r0, wn = a.wn, wlo = a.wlo, W = a.words;
  const bool has_up = band > 0, has_dn = band + 1 < a.bands;
  // Shared memory: planes [rows r0 .. r1][wn][NCH][12]; a scratch word; received toggles [from above,
  // from below][run parity][W][NCH]; slots (row - r0) << 16 | word (~0: none); moves [parity][slot].
  uint32_t* const pad = lsm + (size_t)(R + 1) * wn * NCH * kLbWord;
  uint32_t* const recv = pad + kLbPad;
  uint32_t* const sslot = recv + 4 * W * NCH;
  uint2* const smove = reinterpret_cast<uint2*>(sslot + ((nslots + 1) & ~1) + ((4 * W * NCH) & 1));
  auto PL = [&](int y, int x, int c) -> uint32_t* { return lsm + ((size_t)(y * wn + x) * NCH + c) * kLbWord; };
  for (int k = tid; k < nslots; k += (int)blockDim.x) sslot[k] = ~0u;
  for (int k = tid; k < kLbPad; k += (int)blockDim.x) pad[k] = 0u;
  if (tid < 4 && kForm == kLbCluster)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(lb_addr(&s_bar[tid >> 1][tid & 1])) : "memory");
  if (kForm == kLbCluster) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  if (tid == 0) s_failed = 0;
  __syncthreads();
  auto row_words = [&](int i, int* first) -> int {
    const int lo = a.cand[i], hi = a.cand[a.N + i];
    if (lo == INT_MAX) return 0;
    *first = lo >> 5;
    return (hi >> 5) - (lo >> 5) + 1;
  };
  for (int y = tid; y < R; y += (int)blockDim.x) {
    int at = 0, f = 0;
    for (int q = 0; q < y; ++q) at += row_words(r0 + q, &f);
    const int n = row_words(r0 + y, &f);
    for (int k = 0; k < n; ++k) sslot[at + k] = (uint32_t)y << 16 | (uint32_t)(f + k);
  }
  // planes of rows r0 .. r1: a warp per row and word, lane l reads slot 32 w + l of the three residues
  auto load_planes = [&](const uint8_t* src) {
    for (int it = warp; it < (R + 1) * wn; it += nwarps) {
      const int y = it / wn, x = it - y * wn, i = r0 + y, m = 32 * (wlo + x) + lane;
      const bool in = i < a.N && m >= 0 && m < a.P;
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        uint32_t bits[9];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const int col = (q + 3 - i % 3) % 3;  // colour of residue q in row i
          const uint32_t v =
              in ? src[(size_t)c * a.chain_stride + (size_t)col * a.colour_stride + (size_t)i * a.P + m] : 0u;
          bits[q] = __ballot_sync(~0u, v & 8u);
          bits[3 + q] = __ballot_sync(~0u, v & 2u);
          bits[6 + q] = __ballot_sync(~0u, v & 1u);
        }
        uint32_t mine = 0u;
#pragma unroll
        for (int k = 0; k < 9; ++k) mine = lane == k ? bits[k] : mine;
        if (lane < kLbWord) PL(y, x, c)[lane] = mine;
      }
    }
  };
  if (!cftp) load_planes(base);
  __syncthreads();

  // Update warps: the first holds the last row, the second the first row (all W words, so that the
  // neighbour's toggles of words without candidates here are applied too), the rest the others.
  const bool updates = warp >= ndraw;
  const int uw = warp - ndraw;
  int my_y = -1, my_x = 0, my_c = 0;  // row, window word, chain
  if (updates) {
    const int k = lane / NCH;
    my_c = lane % NCH;
    if (uw < 2) {
      if (k < W && (uw == 0 || R > 1)) {
        my_y = uw == 0 ? R - 1 : 0;
        my_x = a.w0 + k - wlo;
      }
    } else {
      const int item = (tid - 32 * (ndraw + 2)) / NCH;  // of the slots in rows 1 .. R - 2
      int f = 0;
      const int skip = R > 1 ? row_words(r0, &f) : 0;
      int inner = 0;
      for (int y = 1; y + 1 < R; ++y) inner += row_words(r0 + y, &f);
      if (item < inner) {
        my_y = (int)(sslot[skip + item] >> 16);
        my_x = (int)(sslot[skip + item] & 0xffffu) - wlo;
      }
    }
  }
  uint32_t valid = 0u;
  int my_slot = 0;
  if (my_y >= 0) {
    const int i = r0 + my_y, w = wlo + my_x, lo = a.cand[i], hi = a.cand[a.N + i];
    if (lo != INT_MAX && w >= (lo >> 5) && w <= (hi >> 5)) {
      const int blo = max(lo - 32 * w, 0), bhi = min(hi - 32 * w, 31);
      valid = (0xffffffffu << blo) & (0xffffffffu >> (31 - bhi));
      int f = 0, at = 0;
      for (int y = 0; y < my_y; ++y) at += row_words(r0 + y, &f);
      my_slot = at + w - (lo >> 5);
    }
  }
  const bool is_last = updates && uw == 0 && my_y >= 0 && has_dn;                      // faces the band below
  const bool is_first = updates && my_y == 0 && has_up && (uw == 1 || (uw == 0 && R == 1));  // the band above
  const bool tells_dn = is_last && band + 1 != a.silent_plus1, tells_up = is_first && band + 1 != a.silent_plus1;
  const uint32_t here = lb_addr(my_y >= 0 ? PL(my_y, my_x, my_c) : pad + kLbWord * NCH);
  const uint32_t below = lb_addr(my_y >= 0 ? PL(my_y + 1, my_x, my_c) : pad + 2 * kLbWord * NCH);
  const uint32_t left = (uint32_t)(NCH * kLbWord * 4);  // bytes to the word on the left
  const int i3 = my_y >= 0 ? (r0 + my_y) % 3 : 0;
  const uint32_t move_at = lb_addr(smove + my_slot), move_bytes = (uint32_t)(nslots * sizeof(uint2));
  const int xw = my_y >= 0 ? (my_x - (a.w0 - wlo)) * NCH + my_c : 0;  // this lane's exchange word
  const uint32_t recv_up = lb_addr(recv + xw), recv_dn = lb_addr(recv + 2 * W * NCH + xw);
  const uint32_t recv_bytes = (uint32_t)(W * NCH * 4);
  const uint32_t bar_up = lb_addr(&s_bar[0][0]), bar_dn = lb_addr(&s_bar[1][0]);
  uint32_t send_up = 0u, send_dn = 0u, rbar_up = 0u, rbar_dn = 0u;
  if constexpr (kForm == kLbCluster) {
    auto remote_recv = [&](int k, int side) -> uint32_t {  // band k's element for this lane's word
      const int Rk = a.row_start[k + 1] - a.row_start[k];
      const uint32_t off = (uint32_t)(((Rk + 1) * wn * NCH * kLbWord + kLbPad + 2 * side * W * NCH + xw) * 4);
      return lb_remote(lsm, k) + off;
    };
    if (is_first) send_up = remote_recv(band - 1, 1), rbar_up = lb_remote(&s_bar[1][0], band - 1);
    if (is_last) send_dn = remote_recv(band + 1, 0), rbar_dn = lb_remote(&s_bar[0][0], band + 1);
  }
  auto xel = [&](uint32_t par, int b, int to_below) -> uint64_t* {
    return a.xbuf + (((size_t)par * a.bands + b) * 2 + to_below) * (W * NCH) + xw;
  };

  // Draw warps.
  auto gen_index = [&](int s, bool* v) -> int64_t {
    const uint32_t e = updates ? ~0u : sslot[warp * KS + s];
    const int i = r0 + (int)(e >> 16), m = 32 * (int)(e & 0xffffu) + lane;
    *v = e != ~0u && m >= a.cand[i] && m <= a.cand[a.N + i];
    return (int64_t)i * a.M + m;
  };
  uint4 gen[kFast ? 1 : KS];
  uint32_t f_row[kFast ? KS / 4 : 1], f_quad[kFast ? KS / 4 : 1];
  int n_mine = 0;  // slots (fast mode: groups of four) of this warp
  if constexpr (!kFast) {
#pragma unroll
    for (int s = 0; s < KS; ++s) {
      gen[s] = make_uint4(0u, 0u, 0u, 0u);
      if (updates) continue;
      if (sslot[warp * KS + s] != ~0u) n_mine = s + 1;
      bool v;
      const int64_t g = gen_index(s, &v);
      if (v && !cftp) gen[s] = a.tmt[g];
    }
  } else {
#pragma unroll
    for (int g = 0; g < KS / 4; ++g) {
      const uint32_t e = updates ? ~0u : sslot[warp * KS + 4 * g + (lane >> 3)];
      f_row[g] = e == ~0u ? 0u : (uint32_t)r0 + (e >> 16);
      f_quad[g] = e == ~0u ? 0u : (e & 0xffffu) * 8u + (uint32_t)(lane & 7);
      if (__any_sync(~0u, e != ~0u)) n_mine = g + 1;
    }
  }
  // Fast mode: the moves of four words from their Philox blocks.
  auto put = [&](const uint4& d, uint2* out) {
    auto nib = [](bool p, bool q, bool r, bool s) { return (p ? 1u : 0u) | (q ? 2u : 0u) | (r ? 4u : 0u) | (s ? 8u : 0u); };
    const uint32_t u = nib(d.x - a.lo_up < a.w_up, d.y - a.lo_up < a.w_up, d.z - a.lo_up < a.w_up, d.w - a.lo_up < a.w_up);
    const uint32_t v = nib(d.x - a.lo_dn < a.w_dn, d.y - a.lo_dn < a.w_dn, d.z - a.lo_dn < a.w_dn, d.w - a.lo_dn < a.w_dn);
    const uint32_t mine = (u ^ 15u) | (v << 16);
    const uint32_t pair = mine | (__shfl_down_sync(~0u, mine, 1) << 4);
    if (!(lane & 1)) {
      uint8_t* to = reinterpret_cast<uint8_t*>(out + (lane >> 3)) + ((lane & 7) >> 1);
      to[0] = (uint8_t)pair;
      to[4] = (uint8_t)(pair >> 16);
    }
  };
  auto draw_run = [&](uint32_t run, int64_t h, uint32_t reseed_to, uint2* out) {
    if constexpr (!kFast) {
      const int L = (int)(run & 0x1fffffffu);
      if ((run >> 29) & 1u) {  // an epoch's generators (as k_lz_seed)
#pragma unroll
        for (int s = 0; s < KS; ++s) {
          bool v;
          const int64_t g = gen_index(s, &v);
          uint32_t m1 = kTmtMat1, m2 = kTmtMat2, tm = kTmtTmat;
          if (kParams) {
            const uint4 p = __ldg(&a.tmt_params[v ? g : 0]);
            m1 = p.x, m2 = p.y, tm = p.z;
          }
          if (v) gen[s] = tmt_seed(reseed_to + (uint32_t)g, m1, m2, tm);
        }
      }
      // Every lane composes the moves of all its warp's words where registers allow it, else lane s
      // those of slot s.
      constexpr bool kAll = KS <= 4;
      uint32_t x[kAll ? KS : 1], y[kAll ? KS : 1];
#pragma unroll
      for (int s = 0; s < (kAll ? KS : 1); ++s) x[s] = 0xffffffffu, y[s] = 0u;
      for (int hh = 0; hh < L; ++hh) {
        uint32_t um = 0u, dm = 0u;
#pragma unroll
        for (int s = 0; s < KS; ++s) {
          if (s > 0 && s >= n_mine) break;
          uint32_t m1 = kTmtMat1, m2 = kTmtMat2, tm = kTmtTmat;
          if (kParams) {
            bool v;
            const int64_t g = gen_index(s, &v);
            const uint4 p = __ldg(&a.tmt_params[v ? g : 0]);
            m1 = p.x, m2 = p.y, tm = p.z;
          }
          const uint32_t t0 = tmt_next_t0_mad(gen[s], m1, m2, tm);
          const uint32_t bu = __ballot_sync(~0u, t0 - a.lo_up < a.w_up);
          const uint32_t bd = __ballot_sync(~0u, t0 - a.lo_dn < a.w_dn);
          if constexpr (kAll) {
            x[s] ^= (x[s] & bu) | (~x[s] & bd);
            y[s] ^= (y[s] & bu) | (~y[s] & bd);
          } else {
            um = lane == s ? bu : um;
            dm = lane == s ? bd : dm;
          }
        }
        if constexpr (!kAll) {
          x[0] ^= (x[0] & um) | (~x[0] & dm);
          y[0] ^= (y[0] & um) | (~y[0] & dm);
        }
      }
      if constexpr (kAll) {
#pragma unroll
        for (int s = 0; s < KS; ++s)
          if (lane == s) out[warp * KS + s] = make_uint2(x[s], y[s]);
      } else {
        if (lane < KS) out[warp * KS + lane] = make_uint2(x[0], y[0]);
      }
    } else {
#pragma unroll
      for (int g = 0; g < KS / 4; ++g) {
        if (g > 0 && g >= n_mine) break;
        put(fast_quad(a.seed, a.stream, h, f_row[g], f_quad[g]), out + warp * KS + 4 * g);
      }
    }
  };
  const int n_att = cftp ? a.attempts : 1, teams = (int)gridDim.x;
  bool stopped = false;
  for (int att = cftp ? (int)blockIdx.x : 0; att < n_att; att += teams) {
    int nruns = a.nruns, epoch = 0;
    const uint32_t* runs = a.runs;
    int64_t h0 = a.h0;
    if (cftp) {
      if (kFast) {
        nruns = (int)(3 * (a.first_sweeps << att));
        h0 = -(int64_t)nruns;
      } else {
        const int4 d = a.attempt_desc[att];
        runs += d.x;
        nruns = d.y;
        epoch = d.z;
      }
      load_planes(a.start);
    }
    const int c0 = kFast ? (int)(((h0 % 3) + 3) % 3) : 0;
    auto run_at = [&](int j) -> uint32_t {
      if (kFast) return (uint32_t)((c0 + j) % 3) << 30 | 1u;
      return j < nruns ? __ldg(&runs[j]) : 0u;
    };
    auto seed_of = [&](uint32_t run) -> uint32_t {
      return !kFast && ((run >> 29) & 1u) ? __ldg(&a.epoch_seeds[epoch++]) : 0u;
    };
    // A period's steps, two at a time (those past the end are not used).
    auto draw_period = [&](int q) {
      if constexpr (kAhead > 1) {
        uint2* const out = smove + (q & 1) * kAhead * nslots + warp * KS;
  #pragma unroll
        for (int g = 0; g < KS / 4; ++g) {
          if (g > 0 && g >= n_mine) break;
          for (int r = 0; r < kAhead; r += 2) {
            const int64_t h = h0 + q * kAhead + r;
            const uint4 d0 = fast_quad(a.seed, a.stream, h, f_row[g], f_quad[g]);
            const uint4 d1 = fast_quad(a.seed, a.stream, h + 1, f_row[g], f_quad[g]);
            put(d0, out + r * nslots + 4 * g);
            put(d1, out + (r + 1) * nslots + 4 * g);
          }
        }
      }
    };
    uint32_t next = run_at(1);
    if (kAhead > 1) {
      if (!updates) draw_period(0);
    } else if (!updates && nruns > 0) {
      const uint32_t run = run_at(0);
      draw_run(run, h0, seed_of(run), smove);
      if (tid == 0) s_colour[0] = run >> 30;
    }
    // Every 256 runs: has a smaller attempt coalesced?
    auto told_stop = [&](int j) {
      if (!cftp || (j & 255) != 255) return false;
      if (tid == 0) s_stop = *static_cast<volatile int*>(a.best) < att;
      __syncthreads();
      return *static_cast<volatile int*>(&s_stop) != 0;
    };
    if constexpr (kForm == kLbCluster) cooperative_groups::this_cluster().sync();
    else __syncthreads();

    bool failed = false;
    uint32_t r_last = 0u;  // colour of the run before
    // The neighbours' toggles of run `last` (colour r_last) into this CTA's copies of the planes.
    // Each boundary row is one warp, so a word of its left neighbour is patched after the __syncwarp.  All its lanes come
    // here whatever they read of s_failed (another warp may just be setting it): the votes want them all.
    auto patch = [&](uint32_t last, bool& live) {
      const uint32_t par = last & 1u;
      uint32_t tu = 0u, td = 0u;
      if constexpr (kForm == kLbCluster) {
        const uint32_t phase = (last >> 1) & 1u;
        if (__any_sync(~0u, is_first)) live = live && lb_bar_wait(bar_up + 8u * par, phase, a.max_spin);
        if (__any_sync(~0u, is_last)) live = live && lb_bar_wait(bar_dn + 8u * par, phase, a.max_spin);
        if (is_first && live) tu = lb_lds(recv_up + par * recv_bytes);
        if (is_last && live) td = lb_lds(recv_dn + par * recv_bytes);
      } else if constexpr (kForm == kLbGrid) {
        auto poll = [&](const uint64_t* g) -> uint32_t {
          uint64_t v = 0;
          for (long it = 0;; ++it) {
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(g) : "memory");
            if ((uint32_t)(v >> 32) == last + 1u) break;
            if (it > a.max_spin) {
              live = false;
              break;
            }
          }
          return (uint32_t)v;
        };
        if (is_first && live) tu = poll(xel(par, band - 1, 1));
        if (is_last && live) td = poll(xel(par, band + 1, 0));
      }
      if (!__all_sync(~0u, live)) {
        live = false;
        return;
      }
      const int q = (i3 + (int)r_last) % 3;  // this row's residue in that run
      // from above: row r0 - 1 (residue q - 1) toggled N(r0, q - 1) and NE(r0, q - 2), one slot to the
      // left where its residue is 0
      const uint32_t tu_right = __shfl_down_sync(~0u, tu, NCH);  // the word on the right's
      if (is_first) {
        const int qa = q == 0 ? 2 : q - 1, qb = qa == 0 ? 2 : qa - 1;
        const uint32_t right = my_x - (a.w0 - wlo) + 1 < W ? tu_right : 0u;
        const uint32_t n_at = here + 4u * (6 + qa), ne_at = here + 4u * (3 + qb);
        lb_sts(n_at, lb_lds(n_at) ^ tu);
        lb_sts(ne_at, lb_lds(ne_at) ^ (qa == 0 ? __funnelshift_r(tu, right, 1) : tu));
        if (qa == 0 && my_x == a.w0 - wlo) lb_xor_if(ne_at - left, tu << 31);  // into the word left of all
      }
      // from below: row r1 (residue q + 1) toggled NE and N of its own vertices
      if (is_last) {
        const int qc = q == 2 ? 0 : q + 1;
        const uint32_t n_at = below + 4u * (6 + qc), ne_at = below + 4u * (3 + qc);
        lb_sts(n_at, lb_lds(n_at) ^ td);
        lb_sts(ne_at, lb_lds(ne_at) ^ td);
      }
      __syncwarp();
    };
    if constexpr (kAhead > 1) {
      const int periods = (nruns + kAhead - 1) / kAhead;
      int r = c0;  // the step's colour
      for (int p = 0; p < periods; ++p) {
        if (updates) {
          uint32_t at = move_at + (uint32_t)((p & 1) * kAhead) * move_bytes;
          const int len = min(kAhead, nruns - p * kAhead);
          for (int k = 0; k < len; ++k, at += move_bytes) {
            const uint2 move = lb_lds2(at);
            const int q = i3 + r >= 3 ? i3 + r - 3 : i3 + r, qw = q == 0 ? 2 : q - 1;
            const uint32_t own = here + 4u * q, west = here + 4u * qw, south = below + 4u * (6 + q), sw = below + 4u * (3 + qw);
            const uint32_t e = lb_lds(own), ne = lb_lds(own + 12u), n = lb_lds(own + 24u);
            uint32_t w = lb_lds(west), ws = lb_lds(sw);
            const uint32_t s = lb_lds(south), w_l = lb_lds(west - left), ws_l = lb_lds(sw - left);
            if (q == 0) {
              w = __funnelshift_l(w_l, w, 1);
              ws = __funnelshift_l(ws_l, ws, 1);
            }
            const uint32_t flip = ~(n ^ e) & ~(n ^ ws) & (n ^ ne) & (n ^ w) & (n ^ s) & valid;
            const uint32_t T = flip & ((n & ~move.x) | (~n & move.y));
            lb_sts(own, e ^ T);
            lb_sts(own + 12u, ne ^ T);
            lb_sts(own + 24u, n ^ T);
            lb_sts(south, s ^ T);
            const uint32_t tw = q == 0 ? T >> 1 : T, tl = q == 0 ? T << 31 : 0u;
            lb_xor_if(west, tw);
            lb_xor_if(sw, tw);
            lb_xor_if(west - left, tl);
            lb_xor_if(sw - left, tl);
            r = r == 2 ? 0 : r + 1;
            asm volatile("bar.sync 1, %0;" ::"r"(32 * (nwarps - ndraw)) : "memory");
          }
        } else if (p + 1 < periods) {
          draw_period(p + 1);
        }
        lb_cta_sync();
        if (told_stop(p * kAhead + kAhead - 1)) {
          stopped = true;
          break;
        }
      }
    } else if (updates) {
      const bool edge_warp = __any_sync(~0u, is_first || is_last);
      const bool arms = kForm == kLbCluster && warp == ndraw && lane == 0;
      for (int j = 0; j < nruns; ++j) {
        const uint32_t b = (uint32_t)j & 1u;
        bool live = true;
        if constexpr (kForm != kLbOne) live = !*static_cast<volatile int*>(&s_failed);
        if constexpr (kForm == kLbCluster) {
          lb_expect_if(arms && has_up && live, bar_up + 8u * b, recv_bytes);
          lb_expect_if(arms && has_dn && live, bar_dn + 8u * b, recv_bytes);
        }
        const uint32_t r = s_colour[b];
        const uint2 move = lb_lds2(move_at + b * move_bytes);
        if (kForm != kLbOne && edge_warp && j > 0) {
          patch((uint32_t)j - 1u, live);
          if (!live) {
            failed = true;
            s_failed = 1;
          }
        }
        const int q = i3 + (int)r >= 3 ? i3 + (int)r - 3 : i3 + (int)r, qw = q == 0 ? 2 : q - 1;
        const uint32_t own = here + 4u * q, west = here + 4u * qw, south = below + 4u * (6 + q), sw = below + 4u * (3 + qw);
        const uint32_t e = lb_lds(own), ne = lb_lds(own + 12u), n = lb_lds(own + 24u);
        uint32_t w = lb_lds(west), ws = lb_lds(sw);
        const uint32_t s = lb_lds(south), w_l = lb_lds(west - left), ws_l = lb_lds(sw - left);
        if (q == 0) {
          w = __funnelshift_l(w_l, w, 1);
          ws = __funnelshift_l(ws_l, ws, 1);
        }
        // Flippable: E, N, SW equal, NE, W, S their complement; T: slots whose state differs at the
        // end of the run (x: what becomes of 25, y: of 38).
        const uint32_t flip = ~(n ^ e) & ~(n ^ ws) & (n ^ ne) & (n ^ w) & (n ^ s) & valid;
        const uint32_t T = flip & ((n & ~move.x) | (~n & move.y));
        if constexpr (kForm == kLbCluster) {
          lb_send_if(tells_up && live, send_up + b * recv_bytes, T, rbar_up + 8u * b);
          lb_send_if(tells_dn && live, send_dn + b * recv_bytes, T, rbar_dn + 8u * b);
        } else if constexpr (kForm == kLbGrid) {
          const uint64_t tagged = ((uint64_t)((uint32_t)j + 1u) << 32) | T;
          if (tells_up && live) asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(xel(b, band, 0)), "l"(tagged) : "memory");
          if (tells_dn && live) asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(xel(b, band, 1)), "l"(tagged) : "memory");
        }
        lb_sts(own, e ^ T);
        lb_sts(own + 12u, ne ^ T);
        lb_sts(own + 24u, n ^ T);
        lb_sts(south, s ^ T);
        const uint32_t tw = q == 0 ? T >> 1 : T, tl = q == 0 ? T << 31 : 0u;
        lb_xor_if(west, tw);
        lb_xor_if(sw, tw);
        lb_xor_if(west - left, tl);
        lb_xor_if(sw - left, tl);
        r_last = r;
        if (kForm == kLbOne || (j & 63) != 63) {
          lb_cta_sync();
          if (told_stop(j)) {
            stopped = true;
            break;
          }
        } else if (__syncthreads_or(failed ? 1 : 0)) {  // a band that gave up leaves within 64 runs
          failed = true;
          break;
        }
      }
    } else {
      for (int j = 0; j < nruns; ++j) {
        const uint32_t after = run_at(j + 2);
        if (j + 1 < nruns) {
          if (tid == 0) s_colour[(j + 1) & 1] = next >> 30;
          draw_run(next, h0 + j + 1, seed_of(next), smove + ((j + 1) & 1) * nslots);
        }
        next = after;
        if (kForm == kLbOne || (j & 63) != 63) {
          lb_cta_sync();
          if (told_stop(j)) {
            stopped = true;
            break;
          }
        } else if (__syncthreads_or(0)) {
          failed = true;
          break;
        }
      }
    }
    if constexpr (kForm != kLbOne) {
      // the neighbours' last toggles
      if (nruns > 0 && updates) {
        bool live = !failed && !*static_cast<volatile int*>(&s_failed);
        if (__any_sync(~0u, is_first || is_last)) patch((uint32_t)nruns - 1u, live);
        failed = failed || !live;
      }
      if (__syncthreads_or(failed ? 1 : 0) && tid == 0) {
        *static_cast<volatile int*>(a.error) = 1;
        if (kForm == kLbCluster)
          for (int k = 0; k < 64; ++k) __nanosleep(1000);  // what is in flight to this CTA lands
      }
      if constexpr (kForm == kLbCluster) cooperative_groups::this_cluster().sync();
    }
    __syncthreads();
    if (!cftp) break;
    if (stopped) return;
    uint32_t differ = 0u;
    if (NCH == 2)
      for (int k = tid; k < (R + 1) * wn * kLbWord; k += (int)blockDim.x) {
        const uint32_t* p = lsm + (size_t)(k / kLbWord) * 2 * kLbWord + k % kLbWord;
        differ |= p[0] ^ p[kLbWord];
      }
    if (!__syncthreads_or(differ != 0u)) {
      if (tid == 0) atomicMin(a.best, att);
      break;
    }
  }
  __syncthreads();
  // Rows r0 .. r1 - 1 back to the chains: slots [1, M - 2] of the window's inner words.
  for (int it = warp; it < R * (wn - 2); it += nwarps) {
    const int y = it / (wn - 2), x = 1 + it - y * (wn - 2), i = r0 + y, m = 32 * (wlo + x) + lane;
    if (i < 1 || i > a.N - 2 || m < 1 || m > a.M - 2) continue;
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const uint32_t *p = PL(y, x, c), *d = PL(y + 1, x, c), *pl = PL(y, x - 1, c), *dl = PL(y + 1, x - 1, c);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const int qw = q == 0 ? 2 : q - 1;
        auto bit = [&](uint32_t v) { return (v >> lane) & 1u; };
        const uint32_t w = q == 0 ? __funnelshift_l(pl[qw], p[qw], 1) : p[qw];
        const uint32_t sw = q == 0 ? __funnelshift_l(dl[3 + qw], d[3 + qw], 1) : d[3 + qw];
        const uint32_t v = bit(p[q]) * 8u + bit(p[3 + q]) * 2u + bit(p[6 + q]) + bit(w) * 4u + bit(sw) * 16u + bit(d[6 + q]) * 32u;
        const int col = (q + 3 - i % 3) % 3;
        base[(size_t)c * a.chain_stride + (size_t)col * a.colour_stride + (size_t)i * a.P + m] = (uint8_t)v;
      }
    }
  }
  if constexpr (!kFast) {
    if (cftp) return;  // every epoch seeds its generators
#pragma unroll
    for (int s = 0; s < KS; ++s) {
      if (updates) continue;
      bool v;
      const int64_t g = gen_index(s, &v);
      if (v) a.tmt[g] = gen[s];
    }
  }
}

template <int NCH, int kMode, int kForm>
void* lb_kernel_ks(int ks) {
  if constexpr (kMode == kLbFast) {
    return ks == 4 ? (void*)k_lz_bits<NCH, kMode, 4, kForm>
                   : (ks == 8 ? (void*)k_lz_bits<NCH, kMode, 8, kForm> : (void*)k_lz_bits<NCH, kMode, 16, kForm>);
  } else {
    switch (ks) {
      case 1: return (void*)k_lz_bits<NCH, kMode, 1, kForm>;
      case 2: return (void*)k_lz_bits<NCH, kMode, 2, kForm>;
      case 4: return (void*)k_lz_bits<NCH, kMode, 4, kForm>;
      default: return (void*)k_lz_bits<NCH, kMode, 8, kForm>;
    }
  }
}
template <int NCH, int kForm>
void* lb_kernel_mode(int mode, int ks) {
  return mode == kLbFast ? lb_kernel_ks<NCH, kLbFast, kForm>(ks)
                         : (mode == kLbTmt ? lb_kernel_ks<NCH, kLbTmt, kForm>(ks) : lb_kernel_ks<NCH, kLbTmtParams, kForm>(ks));
}
template <int NCH>
void* lb_kernel(LbForm form, int mode, int ks) {
  return form == kLbOne ? lb_kernel_mode<NCH, kLbOne>(mode, ks)
                        : (form == kLbCluster ? lb_kernel_mode<NCH, kLbCluster>(mode, ks) : lb_kernel_mode<NCH, kLbGrid>(mode, ks));
}

// Words drawn per step up to which one CTA, and up to which one cluster, is the fastest form.  Measured
// (us per step, hexagon of side s, one CTA / cluster / one band per SM; the byte kernel):
//   TinyMT  s = 12 (23 words) 0.28 / 0.34 / 0.42; 1.39    s = 20 (39) 0.41 / 0.36 / 0.53; 1.39
//           s = 100 (500) - / 0.45 / 0.57; 1.51           s = 150 (964) - / 0.68 / 0.56; 1.53
//   fast    s = 28 (55) 0.34 / 0.53 / 0.82; 1.51          s = 56 (120) 0.93 / 0.56 / 0.86; 1.51
//           s = 150 (964) - / 0.67 / 0.84; 1.47           s = 256 (2300) - / 0.99 / 0.86; 1.56
// (TinyMT runs of one colour last 1.5 steps, fast-mode runs one.)
constexpr int lb_one_words(bool tinymt) { return tinymt ? 28 : 79; }
constexpr int lb_cluster_words(bool tinymt) { return tinymt ? 650 : 1650; }

}  // namespace

LbPlan lb_plan(const LzResidentGeom& g, const LzResidentRule& rule, const std::vector<int>& lo, const std::vector<int>& hi,
               bool tinymt, bool params) {
  LbPlan p;
  if (g.nch < 1 || g.nch > 2) return p;
  if (tinymt) {
    const uint64_t top = 1u << 23;
    if ((uint64_t)rule.lo_up + rule.w_up > top || (uint64_t)rule.lo_dn + rule.w_dn > top || rule.w_up >= top || rule.w_dn >= top)
      return p;
  }
  const int N = g.N;
  std::vector<int> cnt(N, 0);
  int first = -1, last = -1, w0 = INT_MAX, w1 = -1;
  int64_t total = 0;
  for (int i = 0; i < N; ++i) {
    if (lo[i] < 0) continue;
    cnt[i] = hi[i] / 32 - lo[i] / 32 + 1;
    total += cnt[i];
    w0 = std::min(w0, lo[i] / 32);
    w1 = std::max(w1, hi[i] / 32);
    if (first < 0) first = i;
    last = i;
  }
  if (total == 0 || N > 0xffff) return p;
  p.w0 = w0;
  p.words = w1 - w0 + 1;
  if (p.words * g.nch > 32) return p;  // a boundary row is one warp
  p.wlo = w0 - 2;
  p.wn = p.words + 4;
  // the vertices around the candidates change too
  first = std::max(1, first - 1);
  last = std::min(N - 2, last + 1);
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return p;
  }
  p.form = total <= lb_one_words(tinymt) ? kLbOne : (total <= lb_cluster_words(tinymt) ? kLbCluster : kLbGrid);
  const int rows = last - first + 1;
  const int want = p.form == kLbOne ? 1 : std::min(p.form == kLbCluster ? kLbClusterCtas : std::min(sms, kLbMaxCtas), rows / 2);
  p.bands = std::max(1, want);
  // contiguous bands of at least two rows, the largest (in words) as small as possible
  auto pack = [&](int64_t cap) -> bool {
    int k = 0;
    int64_t in = 0;
    p.row_start[0] = first;
    for (int i = first; i <= last; ++i) {
      if (i - p.row_start[k] >= 2 && in + cnt[i] > cap && last - i + 1 >= 2) {
        if (++k >= p.bands) return false;
        p.row_start[k] = i;
        in = 0;
      }
      in += cnt[i];
    }
    if (in > cap && k > 0 && last + 1 - p.row_start[k] > 3) return false;
    for (int q = k + 1; q <= p.bands; ++q) p.row_start[q] = last + 1;
    return true;
  };
  int64_t a = 1, b = total + 1;
  while (a < b) {
    const int64_t mid = (a + b) / 2;
    if (pack(mid)) b = mid;
    else a = mid + 1;
  }
  if (!pack(a)) return p;
  while (p.bands > 1 && p.row_start[p.bands - 1] > last) --p.bands;
  if (p.bands == 1) p.form = kLbOne;
  int rows_max = 0;
  int64_t words = 0, inner = 0;
  for (int k = 0; k < p.bands; ++k) {
    const int s = p.row_start[k], e = p.row_start[k + 1];
    rows_max = std::max(rows_max, e - s);
    int64_t w = 0, in = 0;
    for (int i = s; i < e; ++i) {
      w += cnt[i];
      if (i > s && i < e - 1) in += cnt[i];
    }
    words = std::max(words, w);
    inner = std::max(inner, in);
  }
  p.update_warps = 2 + (int)((inner * g.nch + 31) / 32);
  p.slots = 0;
  for (int ks : {1, 2, 4, 8, 16}) {
    if (tinymt ? ks > 8 : ks < 4) continue;
    const int64_t warps = (words + ks - 1) / ks;
    if (warps + p.update_warps <= lb_max_threads(ks, !tinymt) / 32) {
      p.slots = ks;
      p.draw_warps = (int)std::max<int64_t>(1, warps);
      break;
    }
  }
  if (!p.slots) return p;
  const int nslots = p.draw_warps * p.slots;
  p.smem = ((size_t)(rows_max + 1) * p.wn * g.nch * kLbWord + kLbPad + 4 * p.words * g.nch + nslots + 4) * sizeof(uint32_t) +
           2 * (size_t)lb_ahead(!tinymt, p.form) * nslots * sizeof(uint2);
  const int mode = tinymt ? (params ? kLbTmtParams : kLbTmt) : kLbFast;
  p.kernel = g.nch == 1 ? lb_kernel<1>(p.form, mode, p.slots) : lb_kernel<2>(p.form, mode, p.slots);
  if (p.smem > 200 * 1024 ||
      dev_allow_smem(p.kernel, p.smem) != cudaSuccess ||
      (p.form == kLbCluster &&
       cudaFuncSetAttribute(p.kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)) {
    cudaGetLastError();
    return p;
  }
  if (p.form == kLbGrid) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, p.kernel, p.threads(), p.smem) != cudaSuccess ||
        (int64_t)per_sm * sms < p.bands) {
      cudaGetLastError();
      return p;
    }
  } else if (p.form == kLbCluster) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)p.bands;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)p.bands);
    cfg.blockDim = dim3((unsigned)p.threads());
    cfg.dynamicSmemBytes = p.smem;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, p.kernel, &cfg) != cudaSuccess || clusters < 1) {
      cudaGetLastError();
      return p;
    }
  }
  p.ok = true;
  return p;
}

LbState::~LbState() {
  for (void* p : {(void*)d_rows, (void*)d_runs, (void*)d_xbuf, (void*)d_error, (void*)d_epoch, (void*)d_teams}) dev_free(p, stream);
}

#define LB_CUDA(expr)                                                                   \
  do {                                                                                  \
    cudaError_t _e = (expr);                                                            \
    if (_e != cudaSuccess)                                                              \
      return fail(RT_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(_e));     \
  } while (0)

namespace {

rt_status lb_prepare(LbState& st, const LzResidentGeom& g, cudaStream_t s) {
  const LbPlan& p = st.plan;
  st.stream = s;
  if (!st.d_rows) {
    if (rt_status e = dev_alloc(&st.d_rows, sizeof p.row_start, s)) return e;
    if (rt_status e = dev_alloc(&st.d_error, 2 * sizeof(int), s)) return e;
    LB_CUDA(cudaMemcpyAsync(st.d_rows, p.row_start, sizeof p.row_start, cudaMemcpyHostToDevice, s));
    if (p.form == kLbGrid) {
      st.xbuf_bytes = (size_t)2 * p.bands * 2 * p.words * g.nch * sizeof(uint64_t);
      if (rt_status e = dev_alloc(&st.d_xbuf, st.xbuf_bytes, s)) return e;
    }
  }
  return RT_OK;
}

LbArgs lb_args(const LbState& st, const LzResidentGeom& g, uint8_t* base, const LzResidentRule& rule, bool tinymt,
               uint4* tmt, const uint4* params, const int* d_cand, uint64_t fast_seed, uint32_t fast_stream) {
  const LbPlan& p = st.plan;
  LbArgs a{};
  a.base = base;
  a.colour_stride = g.colour_stride;
  a.chain_stride = g.chain_stride;
  a.N = g.N;
  a.M = g.M;
  a.P = g.P;
  a.bands = p.bands;
  a.draw_warps = p.draw_warps;
  a.row_start = st.d_rows;
  a.cand = d_cand;
  a.wlo = p.wlo;
  a.wn = p.wn;
  a.w0 = p.w0;
  a.words = p.words;
  const int sh = tinymt ? 9 : 0;
  a.lo_up = rule.lo_up << sh;
  a.w_up = rule.w_up << sh;
  a.lo_dn = rule.lo_dn << sh;
  a.w_dn = rule.w_dn << sh;
  a.tmt = tmt;
  a.tmt_params = params;
  a.seed = fast_seed;
  a.stream = fast_stream;
  a.xbuf = st.d_xbuf;
  a.error = st.d_error;
  a.max_spin = test_silence().spin(1L << 22);
  return a;
}

// Appends the runs of equal colour of a sequence of steps.
void lb_runs(const uint8_t* colours, int64_t n, bool epoch, std::vector<uint32_t>* runs) {
  const size_t from = runs->size();
  for (int64_t k = 0; k < n; ++k) {
    const uint32_t c = colours[k];
    if (runs->size() > from && (runs->back() >> 30) == c) ++runs->back();
    else runs->push_back(c << 30 | (epoch && k == 0 ? 1u << 29 : 0u) | 1u);
  }
}

rt_status lb_upload_runs(LbState& st, const std::vector<uint32_t>& runs, cudaStream_t s) {
  if (st.runs_cap < (int64_t)runs.size()) {
    dev_free(st.d_runs, s);
    st.d_runs = nullptr;
    st.runs_cap = 0;
    if (rt_status e = dev_alloc(&st.d_runs, runs.size() * sizeof(uint32_t), s)) return e;
    st.runs_cap = (int64_t)runs.size();
  }
  LB_CUDA(cudaMemcpyAsync(st.d_runs, runs.data(), runs.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, s));
  return RT_OK;
}

}  // namespace

rt_status lb_cftp(LbState& st, const LzResidentGeom& g, uint8_t* base, const uint8_t* start, const LzResidentRule& rule,
                  bool tinymt, const uint4* params, const int* d_cand, int n,
                  const std::vector<std::vector<LbEpoch>>& epochs, int64_t first_sweeps, uint64_t fast_seed,
                  uint32_t fast_stream, int* attempts_run, bool* coalesced, cudaStream_t s) {
  const LbPlan& p = st.plan;
  if (p.form != kLbOne || g.nch != 2 || n < 1) return fail(RT_ERR_INVALID_ARGUMENT, "lozenge cftp: one CTA, two chains");
  if (rt_status e = lb_prepare(st, g, s)) return e;
  LbArgs a = lb_args(st, g, base, rule, tinymt, nullptr, params, d_cand, fast_seed, fast_stream);
  std::vector<uint32_t> runs, seeds;
  std::vector<int4> desc;
  if (tinymt) {
    for (int k = 0; k < n; ++k) {
      int4 d = make_int4((int)runs.size(), 0, (int)seeds.size(), 0);
      for (const LbEpoch& e : epochs[(size_t)k]) {
        seeds.push_back(e.seed);
        lb_runs(e.colours->data(), (int64_t)e.colours->size(), true, &runs);
      }
      d.y = (int)runs.size() - d.x;
      desc.push_back(d);
    }
    if (rt_status e = lb_upload_runs(st, runs, s)) return e;
    const size_t desc_off = (seeds.size() * sizeof(uint32_t) + 15) / 16 * 16, bytes = desc_off + desc.size() * sizeof(int4);
    if (st.epoch_cap < bytes) {
      dev_free(st.d_epoch, s);
      st.d_epoch = nullptr;
      st.epoch_cap = 0;
      if (rt_status e = dev_alloc(&st.d_epoch, bytes, s)) return e;
      st.epoch_cap = bytes;
    }
    LB_CUDA(cudaMemcpyAsync(st.d_epoch, seeds.data(), seeds.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, s));
    LB_CUDA(cudaMemcpyAsync(st.d_epoch + desc_off, desc.data(), desc.size() * sizeof(int4), cudaMemcpyHostToDevice, s));
    a.runs = st.d_runs;
    a.epoch_seeds = reinterpret_cast<const uint32_t*>(st.d_epoch);
    a.attempt_desc = reinterpret_cast<const int4*>(st.d_epoch + desc_off);
  }
  const int teams = std::min(n, kLbTeams);
  a.attempts = n;
  a.first_sweeps = first_sweeps;
  a.start = start;
  a.team_stride = 2 * g.chain_stride;
  if (!st.d_teams)
    if (rt_status e = dev_alloc(&st.d_teams, kLbTeams * a.team_stride, s)) return e;
  a.base = st.d_teams;
  for (int k = 0; k < teams; ++k)  // the cells that no attempt writes
    LB_CUDA(cudaMemcpyAsync(st.d_teams + k * a.team_stride, start, a.team_stride, cudaMemcpyDeviceToDevice, s));
  a.best = st.d_error + 1;
  LB_CUDA(cudaMemsetAsync(a.best, 0x7f, sizeof(int), s));  // no attempt yet
  void* args[] = {&a};
  LB_CUDA(cudaLaunchKernel(p.kernel, dim3((unsigned)teams), dim3((unsigned)p.threads()), args, p.smem, s));
  int best = 0;
  LB_CUDA(cudaMemcpyAsync(&best, a.best, sizeof best, cudaMemcpyDeviceToHost, s));
  LB_CUDA(cudaStreamSynchronize(s));
  *coalesced = best < n;
  *attempts_run = *coalesced ? best + 1 : n;
  LB_CUDA(cudaMemcpyAsync(base, st.d_teams + (*attempts_run - 1) % teams * a.team_stride, a.team_stride,
                          cudaMemcpyDeviceToDevice, s));
  return RT_OK;
}

rt_status lb_run(LbState& st, const LzResidentGeom& g, uint8_t* base, const LzResidentRule& rule, bool tinymt, uint4* tmt,
                 const uint4* params, const int* d_cand, const uint8_t* colours_host, int64_t steps, uint64_t fast_seed,
                 uint32_t fast_stream, int64_t h0, cudaStream_t s) {
  const LbPlan& p = st.plan;
  if (rt_status e = lb_prepare(st, g, s)) return e;
  constexpr int64_t kChunk = 1 << 16;  // steps per launch
  std::vector<uint32_t> runs;
  for (int64_t done = 0; done < steps; done += kChunk) {
    const int64_t n = std::min(kChunk, steps - done);
    LbArgs a = lb_args(st, g, base, rule, tinymt, tmt, params, d_cand, fast_seed, fast_stream);
    a.h0 = h0 + done;
    a.nruns = (int)n;
    a.silent_plus1 = test_silence().next_plus1();
    if (tinymt) {
      runs.clear();
      lb_runs(colours_host + done, n, false, &runs);
      if (rt_status e = lb_upload_runs(st, runs, s)) return e;
      a.runs = st.d_runs;
      a.nruns = (int)runs.size();
    }
    if (!st.pending) LB_CUDA(cudaMemsetAsync(st.d_error, 0, sizeof(int), s));
    if (st.d_xbuf) LB_CUDA(cudaMemsetAsync(st.d_xbuf, 0, st.xbuf_bytes, s));  // no stale tags
    void* args[] = {&a};
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    if (p.form == kLbGrid) {
      at[0].id = cudaLaunchAttributeCooperative;
      at[0].val.cooperative = 1;
    } else {
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = (unsigned)p.bands;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
    }
    cfg.gridDim = dim3((unsigned)p.bands);
    cfg.blockDim = dim3((unsigned)p.threads());
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    LB_CUDA(cudaLaunchKernelExC(&cfg, p.kernel, args));
    st.pending = p.form != kLbOne;
  }
  return RT_OK;
}

rt_status lb_error(LbState& st, cudaStream_t s) {
  if (!st.pending) return RT_OK;
  int err = 0;
  LB_CUDA(cudaMemcpyAsync(&err, st.d_error, sizeof err, cudaMemcpyDeviceToHost, s));
  LB_CUDA(cudaStreamSynchronize(s));
  st.pending = false;
  if (err) return fail(RT_ERR_TIMEOUT, "lozenge bit-plane engine: a band gave up waiting for a neighbour's toggles");
  return RT_OK;
}

}  // namespace rt
