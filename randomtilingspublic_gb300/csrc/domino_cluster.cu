// Cluster engine of the domino sweep: the whole tiling in the shared memory of one
// thread-block cluster (1-16 CTAs), one bit per lattice edge.
//
// State, flips and draws are the bit-plane engine's (domino_bits.cu): each colour-array row i
// holds four planes of 32-bit words, bit k of word w for cell m = 32 w + k - VD_t(i) the down
// edge of cell (i, m) of colour t, HE(i) and HO(i) the horizontal edges at lattice columns
// (2m, 2m+1) and (2m+1, 2m+2).  A flip of a colour-t cell toggles its four edges and no two
// cells of colour t share one, so there is no passive colour to rebuild, and consecutive
// half-sweeps of one colour (a run) iterate in registers.
//
// What bounds it: a small domain has little to draw (order 100: 0.1 us of the chip's issue per
// half-sweep), so its time is the chain of dependent exchanges, one per colour run.  The
// band-per-SM engines exchange boundary words through L2 (0.9-1.8 us per run); here the bands
// are the CTAs of one cluster, which store the boundary words of a run straight into the
// neighbour's shared memory (st.async), counted by an mbarrier there: 0.43 us per run with the
// update (a cluster barrier per run instead: 0.8 us, its release waits for every outstanding
// access; tagged words polled in shared memory: 0.57 us).  The draws do not depend on the state,
// so warps of their own make them, a run ahead: they compose a run's half-sweeps into one pair of
// move words per 32 cells, and the update warps apply those in a dozen logic operations.
// It serves launches that ask for 1..16 bands, and couplings from the past of regions that k_deep
// (domino_grid.cu), whose exchange every few runs is faster, does not hold on a quarter of the SMs.
// Measured (us per half-sweep, before: the best band shape): order 16 0.22 (before 0.66), order 100
// 0.36 (0.82), order 200 0.88 (1.07) in TinyMT mode; order 16 0.35 (1.27), order 100 0.53 (1.58),
// order 250 1.03 (1.48) in fast mode, where the draws of 16 SMs take over from the exchange.
//
// A boundary word changes two planes that a neighbour holds too: the first row's flips of
// colour t change VD_{1-t}(r0 - 1), the last row's VD_t(r1 - 1).  In a run of colour t the
// neighbour reads and writes only the other colour's plane of those rows, so the owner sends
// its new words in place.
//
// Coupling from the past: attempts are independent until one coalesces, and one cluster leaves most of the
// chip idle, so four clusters run them side by side, attempt k in cluster k mod 4; look-backs double, so
// the time is nearly that of the attempt which coalesces.  One that has become pointless is left within
// 1024 runs.  Measured: exact sample of order 40 in fast mode 15.9 -> 9.6 ms.
//
// TinyMT: a draw warp holds up to KS words of rows of one parity (the rule's thresholds are then
// warp-uniform); lane l keeps the generator of cell 32 w + l of each, and two ballots turn a word's
// draws into its acceptance words.  Fast mode: a Philox block serves a quad of cells, so 32 lanes
// draw for four words at once (lane l: word l / 8, quad l % 8), each pair of lanes writing a byte
// of the moves.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <string>
#include <vector>

#include "domino_cluster.h"
#include "domino_planes.cuh"
#include "domino_sweep.h"
#include "rng.cuh"

namespace rt {

namespace {

__device__ __forceinline__ void cl_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

__device__ __forceinline__ uint32_t cl_remote(const void* local, int rank) {
  uint32_t r;
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(local);
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void cl_store(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
// A 4-byte store into another CTA's shared memory that also counts on that CTA's mbarrier
// (predicated, not branched: it sits on the run's critical path).
__device__ __forceinline__ void cl_send_if(bool on, uint32_t addr, uint32_t v, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t"
      "@p st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.u32 [%0], %1, [%2];\n\t}" ::"r"(addr),
      "r"(v), "r"(bar), "r"((uint32_t)on)
      : "memory");
}
__device__ __forceinline__ void cl_bar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((uint32_t)__cvta_generic_to_shared(bar)) : "memory");
}
__device__ __forceinline__ void cl_bar_expect_if(bool on, uint32_t bar, uint32_t bytes) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t"
      "@p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(bar),
      "r"(bytes), "r"((uint32_t)on)
      : "memory");
}
// Bounded wait for the phase of the given parity; false when it gave up.
__device__ __forceinline__ bool cl_bar_wait(uint32_t addr, uint32_t parity, long max_spin) {
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

constexpr int kClStopRuns = 1023;  // runs between the looks at the smaller attempts (a cluster barrier each)

// kSlots: words per draw warp (TinyMT: their generators are in registers); UI: words and chains
// per update lane.
template <int NCH, int kMode, int KS, int UI>
__global__ void __launch_bounds__(cl_max_threads(kMode == kClFast, KS), 1) k_cluster(ClArgs a) {
  extern __shared__ __align__(16) uint32_t sm[];
  __shared__ uint4 srule[4];
  __shared__ uint32_t s_differ[kClMaxCtas];
  __shared__ __align__(8) uint64_t s_bar[2][2];  // [from above, from below][run parity]
  __shared__ int s_cnt[2];
  __shared__ uint32_t s_colour[2];  // the colour of the run, by run parity
  __shared__ int s_failed;          // a wait gave up
  __shared__ uint32_t s_stop[2];    // a smaller attempt coalesced, by parity of the look
  constexpr bool kFast = kMode == kClFast, kParams = kMode == kClTmtParams;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = (int)(blockDim.x >> 5);
  const int ndraw = a.draw_warps, nslots = ndraw * KS;
  const int rank = (int)cooperative_groups::this_cluster().block_rank();
  // Coupling from the past: cluster `team` runs attempts team, team + teams, ... into chains of its own.
  const bool cftp = NCH == 2 && a.attempts > 0;
  const int team = cftp ? (int)blockIdx.x / a.ctas : 0, teams = cftp ? (int)gridDim.x / a.ctas : 1;
  const int r0 = a.row_start[rank], r1 = a.row_start[rank + 1], R = r1 - r0 + 1, wn = a.wn, wlo = a.wlo;
  // Acceptance tests: TinyMT on the tempered word t0 (the draw is t0 >> 9) with the interval ends
  // scaled by 2^9 (the host admits only intervals with lo_up = 0 whose products fit 32 bits);
  // fast mode on the 32-bit draw, lo_up = 0 again.  {width up, low down, width down}.
  if (tid < 4)
    srule[tid] = kFast ? make_uint4(a.rule.w_up[tid], a.rule.lo_dn[tid], a.rule.w_dn[tid], 0u)
                       : make_uint4(a.rule.w_up[tid] << 9, a.rule.lo_dn[tid] << 9, a.rule.w_dn[tid] << 9, 0u);
  // Shared memory: planes [R rows from r0 - 1][wn words from wlo][NCH][VD0, VD1, HE, HO]; the
  // a scratch word for lanes without one; the slots, x = (row << 16) | word, y = valid cells (0: no
  // word); the moves [run parity][slot].
  uint32_t* const pad = sm + R * 4 * wn * NCH;  // [8 words to the left, the word, the word above's]
  uint2* const sslot = reinterpret_cast<uint2*>(pad + kClPad);
  uint2* const smove = sslot + nslots;
  auto PL = [&](int ri, int p, int wi, int c) -> uint32_t* { return sm + ((ri * wn + wi) * NCH + c) * 4 + p; };

  // Slots: the words of each row parity in row order, in equal blocks over that parity's warps
  // (as many warps per parity as its share of the words asks for).
  for (int k = tid; k < nslots; k += (int)blockDim.x) sslot[k] = make_uint2(0u, 0u);
  if (tid < 2) s_cnt[tid] = 0;
  if (tid == 0) s_failed = 0;
  if (tid < 4) cl_bar_init(&s_bar[tid >> 1][tid & 1]);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
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
  const int c0 = s_cnt[0], c1 = s_cnt[1];
  const int need0 = (c0 + KS - 1) / KS, need1 = (c1 + KS - 1) / KS;
  int cw0 = c0 + c1 > 0 ? (ndraw * c0 + (c0 + c1) / 2) / (c0 + c1) : ndraw;
  cw0 = min(max(cw0, need0), ndraw - need1);
  const int cw1 = ndraw - cw0;
  const int per0 = cw0 ? (c0 + cw0 - 1) / cw0 : 1, per1 = cw1 ? (c1 + cw1 - 1) / cw1 : 1;
  for (int i = r0 + tid; i < r1; i += (int)blockDim.x) {
    int w0 = 0, before = 0;
    const int c = row_words(i, &w0);
    for (int q = r0 + ((r0 ^ i) & 1); q < i; q += 2) {
      int x;
      before += row_words(q, &x);
    }
    const int per = (i & 1) ? per1 : per0, first = (i & 1) ? cw0 : 0;
    const int lo = a.cand[i], hi = a.cand[a.N + i];
    for (int k = 0; k < c; ++k) {
      const int w = w0 + k, at = before + k;
      const int blo = max(lo - 32 * w, 0), bhi = min(hi - 32 * w, 31);
      const uint32_t valid = (0xffffffffu << blo) & (0xffffffffu >> (31 - bhi));
      sslot[(first + at / per) * KS + at % per] = make_uint2(((uint32_t)i << 16) | (uint32_t)w, valid);
    }
  }
  auto load_band = [&](const uint8_t* src) {
    cl_load_window<NCH>(sm, src, a.chain_stride, a.colour_stride, a.P, r0 - 1, R, wlo, wn);
  };
  if (!cftp) load_band(a.base);
  __syncthreads();

  // Update warps: lane item = a word of a chain.  Links: a neighbour whose facing row and this
  // CTA's facing row both hold words.  Each word of the row sends its new plane word every run;
  // the receiver's mbarrier of the run's parity counts the bytes.  A run's boundary words wait
  // for the neighbour's words of the run before, so a neighbour is at most one run ahead and
  // never changes a plane that is still to be read.  (Where only this side holds words the
  // neighbour needs them at the end only: plain stores.)
  const bool updates = warp >= ndraw;
  int rows_w0;
  const int other_up = rank > 0 ? row_words(r0 - 1, &rows_w0) : 0;
  const int other_dn = rank + 1 < a.ctas ? row_words(r1, &rows_w0) : 0;
  const bool link_up = other_up && row_words(r0, &rows_w0), link_dn = other_dn && row_words(r1 - 1, &rows_w0);
  const uint32_t bytes_up = (uint32_t)(other_up * NCH * 4), bytes_dn = (uint32_t)(other_dn * NCH * 4);
  uint32_t above[UI], here[UI];  // shared-memory addresses of the word in the row above and in its own
  uint32_t valid[UI], move_at[UI], up_addr[UI], dn_addr[UI];
  bool odd[UI], pub_up[UI], pub_dn[UI];
  bool wait_up = false, wait_dn = false;
  uint32_t up_bar = 0, dn_bar = 0;
  const bool silent = rank + 1 == a.silent_cta_plus1;  // test hook: sends nothing
#pragma unroll
  for (int u = 0; u < UI; ++u) {
    const int item = updates ? tid - 32 * ndraw + u * 32 * (nwarps - ndraw) : nslots * NCH;
    const int k = item / NCH, c = item % NCH;
    const uint2 e = k < nslots ? sslot[k] : make_uint2(0u, 0u);
    const bool mine = e.y != 0u;
    const int i = (int)(e.x >> 16), wi = (int)(e.x & 0xffffu) - wlo;
    valid[u] = e.y;
    move_at[u] = (uint32_t)__cvta_generic_to_shared(smove + (mine ? k : 0));
    odd[u] = i & 1;
    above[u] = (uint32_t)__cvta_generic_to_shared(mine ? PL(i - r0, 0, wi, c) : pad + 12);
    here[u] = (uint32_t)__cvta_generic_to_shared(mine ? PL(i - r0 + 1, 0, wi, c) : pad + 8);
    pub_up[u] = mine && rank > 0 && i == r0 && !silent;
    pub_dn[u] = mine && rank + 1 < a.ctas && i == r1 - 1 && !silent;
    // where the neighbours keep the planes: the last row of the CTA above, the halo row of the CTA below
    up_addr[u] = pub_up[u] ? cl_remote(PL(r0 - a.row_start[rank - 1], 0, wi, c), rank - 1) : 0u;
    dn_addr[u] = pub_dn[u] ? cl_remote(PL(0, 0, wi, c), rank + 1) : 0u;
    wait_up = wait_up || (link_up && __any_sync(~0u, mine && i == r0));
    wait_dn = wait_dn || (link_dn && __any_sync(~0u, mine && i == r1 - 1));
  }
  const uint32_t bar0 = (uint32_t)__cvta_generic_to_shared(&s_bar[0][0]), bar1 = bar0 + 16u;
  bool plain = false;  // does any lane of the warp store without a link
#pragma unroll
  for (int u = 0; u < UI; ++u)
    plain = plain || __any_sync(~0u, (pub_up[u] && !link_up) || (pub_dn[u] && !link_dn));
  if (updates && rank > 0) up_bar = cl_remote(&s_bar[1][0], rank - 1);
  if (updates && rank + 1 < a.ctas) dn_bar = cl_remote(&s_bar[0][0], rank + 1);
  const uint32_t move_bytes = (uint32_t)(nslots * sizeof(uint2));

  // Draw warps: the generators and the run's moves.
  const int par = updates ? 0 : (int)((sslot[warp * KS].x >> 16) & 1u);
  auto gen_index = [&](int s, bool* v) -> int64_t {
    const uint2 e = sslot[warp * KS + s];
    *v = !updates && ((e.y >> lane) & 1u);
    return (int64_t)((int)(e.x >> 16) - 1) * a.cols + (32 * (int)(e.x & 0xffffu) + lane - 1);
  };
  uint4 gen[kFast ? 1 : KS];
  if constexpr (!kFast) {
#pragma unroll
    for (int s = 0; s < KS; ++s) {
      gen[s] = make_uint4(0u, 0u, 0u, 0u);
      if (updates) continue;
      bool v;
      const int64_t g = gen_index(s, &v);
      if (!cftp && v) gen[s] = a.tmt[g];
    }
  }
  uint32_t f_row[kFast ? KS / 4 : 1], f_quad[kFast ? KS / 4 : 1];  // fast mode: this lane's quads
  int groups = 0;                                                  // groups of four words this warp draws for
  if constexpr (kFast) {
#pragma unroll
    for (int g = 0; g < KS / 4; ++g) {
      const uint2 e = updates ? make_uint2(0u, 0u) : sslot[warp * KS + 4 * g + (lane >> 3)];
      f_row[g] = e.x >> 16;
      f_quad[g] = (e.x & 0xffffu) * 8u + (uint32_t)(lane & 7);
      if (__any_sync(~0u, e.y)) groups = g + 1;
    }
  }
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
  auto draw_run = [&](uint32_t run, int64_t h, uint32_t reseed_to, uint2* out) {
    const uint4 rl = srule[par | ((int)(run >> 31) << 1)];
    if constexpr (!kFast) {
      if ((run >> 30) & 1u) {  // InitTinyMT for an epoch (tinymt.clh:183-203, as k_tmt_seed)
#pragma unroll
        for (int s = 0; s < KS; ++s) {
          bool v;
          const int64_t g = gen_index(s, &v);
          uint32_t m1, m2, tm;
          params_of(s, m1, m2, tm);
          if (v) gen[s] = tmt_seed(reseed_to + (uint32_t)g, m1, m2, tm);
        }
      }
      cl_moves_tmt<KS>(gen, rl, (int)(run & 0x3fffffffu), out + warp * KS, params_of);
    } else {
#pragma unroll
      for (int g = 0; g < KS / 4; ++g) {
        if (g > 0 && g >= groups) break;
        cl_moves_fast(a.seed, a.stream, h, f_row[g], f_quad[g], rl, out + warp * KS + 4 * g);
      }
    }
  };

  bool failed = false;
  uint32_t seq = 0;  // runs so far, over all attempts: run seq counts on barrier seq & 1
  const int n_att = cftp ? a.attempts : 1;
  // Whether a smaller attempt has coalesced, as the first CTA of the cluster sees it: all its CTAs leave
  // at the same run.  A cluster barrier each; a look's word is written again two looks later.
  uint32_t looks = 0;
  auto tell_stop = [&](int attempt) {
    if (rank == 0 && tid < a.ctas)
      cl_store(cl_remote(&s_stop[looks & 1], tid), *static_cast<volatile int*>(a.best) < attempt ? 1u : 0u);
  };
  auto told_stop = [&]() { return *static_cast<volatile uint32_t*>(&s_stop[looks++ & 1]) != 0u; };
  auto stop_at = [&](int j, int attempt) {
    if ((j & kClStopRuns) != kClStopRuns) return false;
    tell_stop(attempt);
    cl_arrive();
    cl_wait();
    return told_stop();
  };
  bool stopped = false;
  for (int att = team; att < n_att; att += teams) {
    int nruns = a.nruns, epoch = 0;
    const uint32_t* runs = a.runs;
    int64_t h = a.h0;
    if (cftp) {
      if (kFast) {
        nruns = (int)(2 * (a.first_sweeps << (a.attempt0 + att)));
        h = -(int64_t)nruns;
      } else {
        const int4 d = a.attempt_desc[att];
        runs += d.x;
        nruns = d.y;
        epoch = d.z;
      }
      load_band(a.start_base);
    }
    auto run_at = [&](int j) -> uint32_t {
      if (kFast) return ((h + j) & 1) ? 1u : 0x80000001u;  // even half-sweeps black (colour 1)
      return j < nruns ? __ldg(&runs[j]) : 0u;
    };
    uint32_t run = run_at(0), next = run_at(1);
    uint32_t seed_next = 0u;
    if (!updates && nruns > 0) {
      if (!kFast && ((run >> 30) & 1u)) seed_next = __ldg(&a.epoch_seeds[epoch++]);
      draw_run(run, h, seed_next, smove + (seq & 1) * nslots);
    }
    if (!updates && lane == 0 && warp == 0) s_colour[seq & 1] = run >> 31;
    if (cftp) tell_stop(att);
    cl_arrive();  // the windows are loaded, the first run's moves drawn
    cl_wait();
    if (cftp && told_stop()) {
      stopped = true;
      break;
    }
    // One barrier per run joins the update warps, in run j, and the draw warps, a run ahead.
    if (updates) {
      const bool arms = warp == ndraw && lane == 0;
      const bool waits = wait_up || wait_dn;
      for (int j = 0; j < nruns; ++j, ++seq) {
        const uint32_t b = seq & 1u;
        // After a wait gave up the CTA arms no barrier (the phase that never came is still open)
        // and sends nothing (the neighbour may be behind): the neighbours give up in turn.
        bool live = !*static_cast<volatile int*>(&s_failed);
        cl_bar_expect_if(arms && link_up && live, bar0 + 8u * b, bytes_up);
        cl_bar_expect_if(arms && link_dn && live, bar1 + 8u * b, bytes_dn);
        const uint32_t t = s_colour[b];
        uint2 move[UI];
#pragma unroll
        for (int u = 0; u < UI; ++u) move[u] = cl_lds2(move_at[u] + b * move_bytes);
        if (waits && j > 0) {  // (the vote wants all the warp's lanes, whatever each has read of s_failed)
          const uint32_t last = seq - 1, at = 8u * (last & 1u), phase = (last >> 1) & 1u;
          if (wait_up && live && !cl_bar_wait(bar0 + at, phase, a.max_spin)) live = false;
          if (wait_dn && live && !cl_bar_wait(bar1 + at, phase, a.max_spin)) live = false;
          if (!__all_sync(~0u, live)) {
            live = false;
            failed = true;
            s_failed = 1;
          }
        }
        const uint32_t off_u = t ? 0u : 4u, off_d = 4u - off_u;
#pragma unroll
        for (int u = 0; u < UI; ++u) {
          const uint2 ab = cl_lds2(above[u]);
          const uint4 me = cl_lds4(here[u]);
          const uint32_t west = cl_lds(here[u] - 16u * NCH + 12u);
          const bool aligned = odd[u] == (t != 0u);  // left HE, right HO of the same word
          const uint32_t U = t ? ab.x : ab.y, D = t ? me.y : me.x;
          const uint32_t lft = aligned ? me.z : __funnelshift_l(west, me.w, 1), rgt = aligned ? me.w : me.z;
          // Flippable: up = down, left = right, up != left (states 3 and 12); T: cells whose state
          // at the end of the run differs.
          const uint32_t flip = ~(U ^ D) & ~(lft ^ rgt) & (U ^ lft) & valid[u];
          const uint32_t T = flip & ((U & ~move[u].x) | (~U & move[u].y));
          const uint32_t new_u = U ^ T, new_d = D ^ T;
          cl_send_if(pub_up[u] && link_up && live, up_addr[u] + off_u, new_u, up_bar + 8u * b);
          cl_send_if(pub_dn[u] && link_dn && live, dn_addr[u] + off_d, new_d, dn_bar + 8u * b);
          cl_sts(above[u] + off_u, new_u);
          cl_sts(here[u] + off_d, new_d);
          cl_sts(here[u] + 8u, me.z ^ T);
          // HO: the word itself, or (left edges of an unaligned row) bit k - 1 of this word and bit
          // 31 of the word to the left, whose other bits belong to that word's cells.
          cl_xor(here[u] + 12u, aligned ? T : T >> 1);
          cl_xor_if(here[u] - 16u * NCH + 12u, aligned ? 0u : T << 31);
          if (plain) {
            if (pub_up[u] && !link_up) cl_store(up_addr[u] + off_u, new_u);
            if (pub_dn[u] && !link_dn) cl_store(dn_addr[u] + off_d, new_d);
          }
        }
        if ((j & 63) != 63) {
          cl_cta_sync();
        } else {  // a CTA that gave up leaves within 64 runs; a coupling's runs on, without waits, to meet its cluster
          if (__syncthreads_or(failed ? 1 : 0) && !cftp) {
            failed = true;
            break;
          }
          if (cftp && stop_at(j, att)) {
            stopped = true;
            ++seq;
            break;
          }
        }
      }
    } else {
      for (int j = 0; j < nruns; ++j, ++seq) {
        const uint32_t after = run_at(j + 2);
        if (j + 1 < nruns) {
          if (!kFast && ((next >> 30) & 1u)) seed_next = __ldg(&a.epoch_seeds[epoch++]);
          if (lane == 0 && warp == 0) s_colour[(seq + 1) & 1] = next >> 31;
          draw_run(next, h + j + 1, seed_next, smove + ((seq + 1) & 1) * nslots);
        }
        next = after;
        if ((j & 63) != 63) {
          cl_cta_sync();
        } else {
          if (__syncthreads_or(0) && !cftp) {
            failed = true;
            break;
          }
          if (cftp && stop_at(j, att)) {
            stopped = true;
            ++seq;
            break;
          }
        }
      }
    }
    // The neighbours' last words are in.
    if (nruns > 0 && !failed && !*static_cast<volatile int*>(&s_failed)) {
      const uint32_t last = seq - 1;
      if (link_up && !cl_bar_wait(bar0 + 8u * (last & 1u), (last >> 1) & 1u, a.max_spin)) failed = true;
      if (link_dn && !cl_bar_wait(bar1 + 8u * (last & 1u), (last >> 1) & 1u, a.max_spin)) failed = true;
    }
    // A CTA that gave up tells the others, and all stay until what is in flight has landed.
    if (__syncthreads_or(failed ? 1 : 0) && tid == 0) {
      *static_cast<volatile int*>(a.error + team) = 1;
      for (int k = 0; k < 64; ++k) __nanosleep(1000);
    }
    cl_arrive();
    cl_wait();
    if (*static_cast<volatile int*>(a.error + team)) {
      stopped = true;
      break;
    }
    if (!cftp || stopped) break;
    // Coalescence: does any plane word of the CTA's rows differ between the two chains?
    uint32_t differ = 0;
    if (NCH == 2) {
      const uint4* p0 = reinterpret_cast<const uint4*>(sm) + wn * NCH;
      for (int k = tid; k < (R - 1) * wn; k += (int)blockDim.x) {
        const uint4 x = p0[2 * k], y = p0[2 * k + 1];
        differ |= (x.x ^ y.x) | (x.y ^ y.y) | (x.z ^ y.z) | (x.w ^ y.w);
      }
    }
    const uint32_t band_differs = (uint32_t)__syncthreads_or(differ != 0u ? 1 : 0);
    if (tid < a.ctas) cl_store(cl_remote(&s_differ[rank], tid), band_differs);
    cl_arrive();
    cl_wait();
    uint32_t any = 0;
    for (int k = 0; k < a.ctas; ++k) any |= s_differ[k];
    if (!any) {
      if (rank == 0 && tid == 0) atomicMin(a.best, att);
      break;
    }
    __syncthreads();  // s_differ read before the next attempt's flags
  }
  if (stopped && cftp) return;
  __syncthreads();
  cl_store_window<NCH>(sm, a.base + (size_t)team * a.team_stride, a.chain_stride, a.colour_stride, a.P, a.cols, r0 - 1, R, wlo, wn);
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

template <int NCH, int kMode, int UI>
void* cl_kernel_ks(int ks) {
  if constexpr (kMode == kClFast) {
    return ks == 4 ? (void*)k_cluster<NCH, kMode, 4, UI>
                   : (ks == 8 ? (void*)k_cluster<NCH, kMode, 8, UI> : (void*)k_cluster<NCH, kMode, 16, UI>);
  } else {
    switch (ks) {
      case 1: return (void*)k_cluster<NCH, kMode, 1, UI>;
      case 2: return (void*)k_cluster<NCH, kMode, 2, UI>;
      case 4: return (void*)k_cluster<NCH, kMode, 4, UI>;
      default: return (void*)k_cluster<NCH, kMode, 8, UI>;
    }
  }
}

template <int NCH>
void* cl_kernel(int mode, int ks, int ui) {
  if (mode == kClFast) return ui == 1 ? cl_kernel_ks<NCH, kClFast, 1>(ks) : cl_kernel_ks<NCH, kClFast, 2>(ks);
  return mode == kClTmt ? cl_kernel_ks<NCH, kClTmt, 1>(ks) : cl_kernel_ks<NCH, kClTmtParams, 1>(ks);
}

// Cluster size by the words drawn per half-sweep: one CTA where its draws are done before a
// cluster's exchange would be (TinyMT order 5: 0.19 us per half-sweep against 0.22 on 16 CTAs,
// order 16: 0.31 / 0.22; fast mode, which exchanges every half-sweep, order 16: 0.35 / 0.43,
// order 22 0.43 / 0.43), else the largest.
int cl_ctas_for(int64_t words, bool fast) {
  return fast ? (words <= 40 ? 1 : kClMaxCtas) : (words <= 16 ? 1 : kClMaxCtas);
}

}  // namespace

// Measured on a GB300, us per half-sweep, cluster / one band per SM (domino_grid.cu).  TinyMT: order 64
// 0.30 / 0.53, 100 0.37 / 0.51, 120 (686 words) 0.44 / 0.46, 130 (779) 0.65 / 0.56.  Fast mode:
// order 100 0.60 / 0.94, 220 (1915) 0.95 / 1.13, 250 (2442) 1.03 / 1.15 with one chain and 1.21 / 1.15
// with two, 260 (2615) 1.12 / 1.07.  Beyond, the draws of 16 SMs take longer than the exchange of
// 152 bands through L2.
int64_t cl_auto_words(bool fast) { return fast ? 2400 : 700; }

void ClPlan::build(const std::vector<int>& lo, const std::vector<int>& hi, int N, int nch, bool fast, int ctas_asked) {
  ok = false;
  why.clear();
  words = draw_cells = 0;
  const int rows = N - 2;
  auto has = [&](int i) { return i >= 1 && i <= rows && lo[i] >= 0; };
  std::vector<int> cnt(N + 1, 0);
  int w0 = INT_MAX, w1 = -1, first = -1, last = -1;
  for (int i = 1; i <= rows; ++i) {
    if (!has(i)) continue;
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
  if (words > (int64_t)kClMaxCtas * 24 * 16 || N > 0xffff) {
    why = "too many words for one thread-block cluster";
    return;
  }
  // The vertices around the candidates change too: a row above and below, a word left and
  // right (and one more word of margin for the edges of those).
  first = std::max(1, first - 1);
  last = std::min(rows, last + 1);
  wlo = w0 - 2;
  wn = w1 - w0 + 5;
  ctas = std::min(ctas_asked > 0 ? std::min(ctas_asked, kClMaxCtas) : cl_ctas_for(words, fast), last - first + 1);
  // Rows: contiguous bands, the largest (in words) as small as possible.
  auto pack = [&](int64_t cap, int* start) -> bool {
    int k = 0;
    int64_t in = 0;
    start[0] = first;
    for (int i = first; i <= last; ++i) {
      if (in > 0 && in + cnt[i] > cap) {
        if (++k >= ctas) return false;
        start[k] = i;
        in = 0;
      }
      in += cnt[i];
    }
    for (int q = k + 1; q <= ctas; ++q) start[q] = last + 1;
    return true;
  };
  int64_t a = 1, b = words;
  for (int i = first; i <= last; ++i) a = std::max<int64_t>(a, cnt[i]);
  while (a < b) {
    const int64_t mid = (a + b) / 2;
    if (pack(mid, row_start)) b = mid;
    else a = mid + 1;
  }
  pack(a, row_start);
  while (ctas > 1 && row_start[ctas - 1] > last) --ctas;  // no empty bands
  // Words per draw warp: the fewest that fit (more warps hide more latency), each warp of one row
  // parity; TinyMT at most 8, the generators live in registers.
  int rows_max = 0;
  int64_t par[kClMaxCtas][2] = {};
  for (int k = 0; k < ctas; ++k) {
    rows_max = std::max(rows_max, row_start[k + 1] - row_start[k]);
    for (int i = row_start[k]; i < row_start[k + 1]; ++i) par[k][i & 1] += cnt[i];
  }
  auto warps_for = [&](int ks) {
    int64_t w = 0;
    for (int k = 0; k < ctas; ++k) w = std::max<int64_t>(w, (par[k][0] + ks - 1) / ks + (par[k][1] + ks - 1) / ks);
    return w;
  };
  slots = 0;
  for (int ks : {1, 2, 4, 8, 16}) {
    if (fast ? ks < 4 : ks > 8) continue;  // fast mode: a warp draws for four words at once
    if (warps_for(ks) <= cl_max_threads(fast, ks) / 32 - kClUpdateWarps) {
      slots = ks;
      break;
    }
  }
  if (!slots) {
    why = "too many words for one thread-block cluster";
    return;
  }
  draw_warps = (int)warps_for(slots);
  const int items = draw_warps * slots * nch;
  per_lane = items > 32 * kClUpdateWarps ? 2 : 1;
  update_warps = (items + 32 * per_lane - 1) / (32 * per_lane);
  smem_bytes = ((size_t)(rows_max + 1) * 4 * wn * nch + kClPad) * sizeof(uint32_t) +
               3 * (size_t)draw_warps * slots * sizeof(uint2);
  // Every CTA's window spans all the domain's words, so a long bent domain of few words a row needs much of it.
  if (smem_bytes > kClMaxSmem) {
    why = "band window exceeds shared memory";
    return;
  }
  ok = true;
}

#define RT_CUDA_C(expr)                                                                 \
  do {                                                                                  \
    cudaError_t _e = (expr);                                                            \
    if (_e != cudaSuccess)                                                              \
      return fail(RT_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(_e));     \
  } while (0)

ClusterEngine::~ClusterEngine() {
  for (void* p : {(void*)d_runs, (void*)d_epoch, (void*)d_result, (void*)d_teams}) dev_free(p, stream);
}

rt_status ClusterEngine::prepare(DmSampler& s) {
  ready = false;
  plan.ok = false;
  nch = s.active;
  bands_asked = s.eff_bands;
  stream = s.stream;
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
    if (fast ? s.rule.lo_up[c] != 0 : s.rule.lo_up[c] != 0 || s.rule.w_up[c] >= (1u << 23) || w_dn >= (1u << 23) || lo_dn + w_dn > (1u << 23)) {
      plan.why = "rule intervals outside the cluster kernel's compare range";
      return RT_OK;
    }
  }
  plan.build(s.cand_lo, s.cand_hi, s.N, nch, fast, s.eff_bands);
  if (!plan.ok) return RT_OK;
  const int mode = fast ? kClFast : (s.tmt_params ? kClTmtParams : kClTmt);
  kernel = nch == 1 ? cl_kernel<1>(mode, plan.slots, plan.per_lane) : cl_kernel<2>(mode, plan.slots, plan.per_lane);
  if (dev_allow_smem(kernel, plan.smem_bytes) != cudaSuccess ||
      cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    plan.ok = false;
    plan.why = "the device does not allow the launch";
    return RT_OK;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)plan.ctas;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)plan.ctas);
  cfg.blockDim = dim3((unsigned)plan.threads());
  cfg.dynamicSmemBytes = plan.smem_bytes;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters < 1) {
    cudaGetLastError();
    plan.ok = false;
    plan.why = "the cluster does not fit the device";
    return RT_OK;
  }
  if (!d_result) {
    if (rt_status st = dev_alloc(&d_result, (1 + kClTeams) * sizeof(int), stream)) return st;
  }
  ready = true;
  return RT_OK;
}

namespace {

ClArgs cl_args(const ClusterEngine& e, DmSampler& s) {
  ClArgs a{};
  a.base = s.base;
  a.N = s.N;
  a.P = s.P;
  a.cols = s.N / 2 - 2;
  a.ctas = e.plan.ctas;
  a.draw_warps = e.plan.draw_warps;
  a.chain_stride = s.chain_stride;
  a.colour_stride = s.colour_stride;
  a.tmt = s.tmt;
  a.tmt_params = s.tmt_params;
  a.cand = s.d_cand;
  std::copy(e.plan.row_start, e.plan.row_start + kClMaxCtas + 1, a.row_start);
  a.wlo = e.plan.wlo;
  a.wn = e.plan.wn;
  a.rule = s.rule;
  a.stream = s.opts.fast_stream;
  a.best = e.d_result;
  a.error = e.d_result + 1;
  a.max_spin = s.test_max_spin > 0 ? s.test_max_spin : test_silence().spin(1L << 22);
  a.silent_cta_plus1 = s.test_silent_band >= 0 ? s.test_silent_band + 1 : test_silence().next_plus1();
  return a;
}

rt_status cl_launch(const ClusterEngine& e, DmSampler& s, ClArgs& a, int teams = 1) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)e.plan.ctas;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(e.plan.ctas * teams));
  cfg.blockDim = dim3((unsigned)e.plan.threads());
  cfg.dynamicSmemBytes = e.plan.smem_bytes;
  cfg.stream = s.stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (!e.pending_error_check) RT_CUDA_C(cudaMemsetAsync(e.d_result, 0, (1 + kClTeams) * sizeof(int), s.stream));
  void* args[] = {&a};
  RT_CUDA_C(cudaLaunchKernelExC(&cfg, e.kernel, args));
  s.launches++;
  return RT_OK;
}

}  // namespace

namespace {
rt_status cl_gave_up() {
  return fail(RT_ERR_TIMEOUT, "cluster sweep: a wait gave up (a neighbour's boundary words never came)");
}
}  // namespace

rt_status ClusterEngine::check_error(DmSampler& s) {
  if (!pending_error_check) return RT_OK;
  int err = 0;
  RT_CUDA_C(cudaMemcpyAsync(&err, d_result + 1, sizeof(int), cudaMemcpyDeviceToHost, s.stream));
  RT_CUDA_C(cudaStreamSynchronize(s.stream));
  pending_error_check = false;
  return err ? cl_gave_up() : RT_OK;
}

rt_status ClusterEngine::launch(DmSampler& s, const uint8_t* colours_host, int64_t steps, uint64_t fast_seed, int64_t h0) {
  const int64_t chunk_max = 65536;  // bounds one launch to a fraction of a second
  std::vector<uint32_t> runs;
  for (int64_t done = 0; done < steps;) {
    const int64_t n = std::min(chunk_max, steps - done);
    ClArgs a = cl_args(*this, s);
    if (s.opts.rng_mode == RT_RNG_FAST) {
      a.seed = fast_seed;
      a.h0 = h0 + done;
      a.nruns = (int)n;
    } else {
      runs.clear();
      append_runs(colours_host + done, n, false, &runs);
      if (runs_cap < (int64_t)runs.size()) {
        dev_free(d_runs, s.stream);
        d_runs = nullptr;
        runs_cap = 0;
        if (rt_status st = dev_alloc(&d_runs, runs.size() * sizeof(uint32_t), s.stream)) return st;
        runs_cap = (int64_t)runs.size();
      }
      RT_CUDA_C(cudaMemcpyAsync(d_runs, runs.data(), runs.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, s.stream));
      a.runs = d_runs;
      a.nruns = (int)runs.size();
    }
    if (rt_status st = cl_launch(*this, s, a)) return st;
    pending_error_check = true;
    done += n;
  }
  return RT_OK;
}

rt_status ClusterEngine::cftp(DmSampler& s, int a0, int n, const std::vector<std::vector<RunEngine::Epoch>>& epochs,
                              int64_t first_sweeps, uint64_t fast_seed, int* attempts_run, bool* coalesced) {
  *attempts_run = 0;
  *coalesced = false;
  const bool fast = s.opts.rng_mode == RT_RNG_FAST;
  if (n < 1 || n > 40 || s.active != 2) return fail(RT_ERR_INVALID_ARGUMENT, "cluster cftp: 1..40 attempts, 2 chains");
  if (!fast && (int)epochs.size() < n) return fail(RT_ERR_INVALID_ARGUMENT, "cluster cftp: epochs missing");
  ClArgs a = cl_args(*this, s);
  std::vector<uint32_t> runs, seeds;
  std::vector<int4> desc;
  if (!fast) {
    for (int k = 0; k < n; ++k) {
      int4 d = make_int4((int)runs.size(), 0, (int)seeds.size(), 0);
      for (const RunEngine::Epoch& e : epochs[k]) {
        if (!e.colours || e.colours->empty()) continue;
        seeds.push_back(e.seed);
        append_runs(e.colours->data(), (int64_t)e.colours->size(), true, &runs);
      }
      d.y = (int)runs.size() - d.x;
      desc.push_back(d);
    }
    if (runs_cap < (int64_t)runs.size()) {
      dev_free(d_runs, s.stream);
      d_runs = nullptr;
      runs_cap = 0;
      if (rt_status st = dev_alloc(&d_runs, runs.size() * sizeof(uint32_t), s.stream)) return st;
      runs_cap = (int64_t)runs.size();
    }
    const size_t desc_off = (seeds.size() * sizeof(uint32_t) + 15) / 16 * 16;
    const size_t eb = desc_off + desc.size() * sizeof(int4);
    if (epoch_cap < eb) {
      dev_free(d_epoch, s.stream);
      d_epoch = nullptr;
      epoch_cap = 0;
      if (rt_status st = dev_alloc(&d_epoch, eb, s.stream)) return st;
      epoch_cap = eb;
    }
    RT_CUDA_C(cudaMemcpyAsync(d_runs, runs.data(), runs.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, s.stream));
    RT_CUDA_C(cudaMemcpyAsync(d_epoch, seeds.data(), seeds.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, s.stream));
    RT_CUDA_C(cudaMemcpyAsync(reinterpret_cast<uint8_t*>(d_epoch) + desc_off, desc.data(), desc.size() * sizeof(int4),
                              cudaMemcpyHostToDevice, s.stream));
    a.runs = d_runs;
    a.epoch_seeds = d_epoch;
    a.attempt_desc = reinterpret_cast<const int4*>(reinterpret_cast<uint8_t*>(d_epoch) + desc_off);
  }
  a.attempts = n;
  a.attempt0 = a0;
  a.first_sweeps = first_sweeps;
  a.seed = fast_seed;
  a.start_base = s.base + 2 * s.chain_stride;
  // Attempts side by side, a cluster each: look-backs double, so the time is about that of the attempt which
  // coalesces, not the sum of all up to it.
  const int teams = std::min(n, kClTeams);
  a.team_stride = 2 * s.chain_stride;
  if (!d_teams)
    if (rt_status st = dev_alloc(&d_teams, kClTeams * a.team_stride, stream)) return st;
  a.base = d_teams;
  for (int k = 0; k < teams; ++k)  // the cells that no attempt writes
    RT_CUDA_C(cudaMemcpyAsync(d_teams + k * a.team_stride, a.start_base, a.team_stride, cudaMemcpyDeviceToDevice, s.stream));
  if (rt_status st = check_error(s)) return st;
  RT_CUDA_C(cudaMemsetAsync(d_result, 0, (1 + kClTeams) * sizeof(int), s.stream));
  RT_CUDA_C(cudaMemsetAsync(d_result, 0x7f, sizeof(int), s.stream));  // no attempt yet
  pending_error_check = true;  // the words are cleared
  rt_status launched = cl_launch(*this, s, a, teams);
  pending_error_check = false;
  if (launched) return launched;
  int res[1 + kClTeams] = {};
  RT_CUDA_C(cudaMemcpyAsync(res, d_result, sizeof res, cudaMemcpyDeviceToHost, s.stream));
  RT_CUDA_C(cudaStreamSynchronize(s.stream));
  for (int k = 0; k < teams; ++k)
    if (res[1 + k]) return cl_gave_up();
  *coalesced = res[0] < n;
  *attempts_run = *coalesced ? res[0] + 1 : n;
  const int last = *attempts_run - 1;
  RT_CUDA_C(cudaMemcpyAsync(s.base, d_teams + last % teams * a.team_stride, a.team_stride, cudaMemcpyDeviceToDevice, s.stream));
  return RT_OK;
}

}  // namespace rt
