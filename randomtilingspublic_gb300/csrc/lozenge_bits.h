// Bit-plane engine of the lozenge sweep (see lozenge_bits.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "lozenge_resident.h"
#include "rt_internal.h"

namespace rt {

constexpr int kLbMaxCtas = 160;     // bands
constexpr int kLbClusterCtas = 16;  // CTAs of a cluster

constexpr int kLbTeams = 4;         // attempts of a coupling from the past side by side

// Exchange between bands: none (one CTA), through the shared memory of one cluster, or through L2.
enum LbForm : int { kLbOne = 0, kLbCluster = 1, kLbGrid = 2 };

struct LbPlan {
  bool ok = false;
  LbForm form = kLbOne;
  int bands = 0, slots = 0, draw_warps = 0, update_warps = 0;  // slots: words per draw warp
  int wlo = 0, wn = 0, w0 = 0, words = 0;  // window words [wlo, wlo + wn); words that hold candidates
  int row_start[kLbMaxCtas + 1] = {};
  size_t smem = 0;
  void* kernel = nullptr;
  int threads() const { return 32 * (draw_warps + update_warps); }
};

struct LbState {
  LbPlan plan;
  int nch = 0;
  cudaStream_t stream = nullptr;
  int* d_rows = nullptr;       // row_start
  uint32_t* d_runs = nullptr;
  int64_t runs_cap = 0;
  uint64_t* d_xbuf = nullptr;  // kLbGrid: tagged words
  size_t xbuf_bytes = 0;
  int* d_error = nullptr;      // {a band gave up, smallest attempt that coalesced}
  uint8_t* d_epoch = nullptr;  // epoch seeds then attempt descriptors
  size_t epoch_cap = 0;
  uint8_t* d_teams = nullptr;  // two chains per team
  bool pending = false;
  ~LbState();
};

// The plan for candidates lo / hi (each row's first and last slot that can flip; -1: none).
LbPlan lb_plan(const LzResidentGeom& g, const LzResidentRule& rule, const std::vector<int>& lo, const std::vector<int>& hi,
               bool tinymt, bool params);

// As lz_resident_run; d_cand: [2][N], first (INT_MAX: none) and last candidate slot of each row.
rt_status lb_run(LbState& st, const LzResidentGeom& g, uint8_t* base, const LzResidentRule& rule, bool tinymt, uint4* tmt,
                 const uint4* params, const int* d_cand, const uint8_t* colours_host, int64_t steps, uint64_t fast_seed,
                 uint32_t fast_stream, int64_t h0, cudaStream_t s);

// Coupling from the past of a kLbOne plan in one launch: attempts 0 .. n - 1 of chains 0 and 1 from the start states,
// kLbTeams at a time, a CTA each, into base.  TinyMT: attempt k runs the epochs epochs[k] in order; fast mode: steps
// [-3 first_sweeps << k, 0).  Returns the attempts run and whether the last coalesced.
struct LbEpoch {
  uint32_t seed;
  const std::vector<uint8_t>* colours;
};
rt_status lb_cftp(LbState& st, const LzResidentGeom& g, uint8_t* base, const uint8_t* start, const LzResidentRule& rule,
                  bool tinymt, const uint4* params, const int* d_cand, int n,
                  const std::vector<std::vector<LbEpoch>>& epochs, int64_t first_sweeps, uint64_t fast_seed,
                  uint32_t fast_stream, int* attempts_run, bool* coalesced, cudaStream_t s);

// RT_ERR_TIMEOUT when a band of an earlier launch gave up waiting (synchronises with s).
rt_status lb_error(LbState& st, cudaStream_t s);

}  // namespace rt
