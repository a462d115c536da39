// Cluster engine of the domino sweep (see domino_cluster.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "domino_rules.h"
#include "domino_runs.h"
#include "rt_internal.h"

namespace rt {

struct DmSampler;

constexpr int kClMaxCtas = 16;   // CTAs of the cluster
constexpr size_t kClMaxSmem = 200 * 1024;  // dynamic shared memory of a CTA, at most
constexpr int kClUpdateWarps = 8;  // warps that update the words, at most
// Threads per CTA, at most: 64 registers a thread, 80 where the generators of 8 words need them.
constexpr int cl_max_threads(bool fast, int slots) { return !fast && slots > 4 ? 768 : 1024; }

struct ClArgs {
  uint8_t* base;
  int N, P, cols, ctas, draw_warps;
  size_t chain_stride, colour_stride;
  uint4* tmt;
  const uint4* tmt_params;
  const int* cand;                 // [2][N]: each row's first (INT_MAX: none) and last candidate column
  int row_start[kClMaxCtas + 1];   // CTA k owns colour-array rows [row_start[k], row_start[k + 1])
  int wlo, wn;                     // the window's first word and words per row (every CTA's)
  DmRule rule;
  const uint32_t* runs;            // TinyMT: (colour << 31) | (epoch start << 30) | length
  int nruns;                       // fast mode: half-sweeps
  uint64_t seed;                   // fast mode
  uint32_t stream;
  int64_t h0;
  // Coupling from the past in one launch (attempts > 0, two chains), as in RunArgs.
  int attempts, attempt0;
  int64_t first_sweeps;
  const uint8_t* start_base;
  const int4* attempt_desc;
  const uint32_t* epoch_seeds;
  size_t team_stride;  // bytes between the chains of two teams (clusters that run attempts side by side)
  int* best;           // smallest attempt that coalesced
  int* error;          // [team], set when a bounded wait gave up
  long max_spin;
  int silent_cta_plus1;
};

struct ClPlan {
  bool ok = false;
  std::string why;
  int ctas = 0, slots = 0;                // cluster size, words per draw warp
  int draw_warps = 0, update_warps = 0;   // warps per CTA
  int per_lane = 1;                       // words and chains per update lane
  int threads() const { return 32 * (draw_warps + update_warps); }
  int row_start[kClMaxCtas + 1] = {};
  int wlo = 0, wn = 0;
  int64_t words = 0, draw_cells = 0;
  size_t smem_bytes = 0;
  // From each colour-array row's first and last flip-candidate column (-1: none).  ctas: the
  // cluster size asked for (0: by size).
  void build(const std::vector<int>& lo, const std::vector<int>& hi, int N, int nch, bool fast, int ctas_asked);
};

// Words per half-sweep up to which the automatic choice is the cluster.
int64_t cl_auto_words(bool fast);

constexpr int kClTeams = 4;  // attempts of a coupling from the past side by side

struct ClusterEngine {
  ClPlan plan;
  bool ready = false;
  int nch = 0, bands_asked = 0;
  void* kernel = nullptr;
  cudaStream_t stream = nullptr;
  uint32_t* d_runs = nullptr;
  int64_t runs_cap = 0;
  uint32_t* d_epoch = nullptr;  // epoch seeds then attempt descriptors
  size_t epoch_cap = 0;
  int* d_result = nullptr;     // {smallest attempt that coalesced, error of each team}
  uint8_t* d_teams = nullptr;  // two chains per team
  bool pending_error_check = false;

  ~ClusterEngine();
  rt_status prepare(DmSampler& s);
  rt_status launch(DmSampler& s, const uint8_t* colours_host, int64_t steps, uint64_t fast_seed, int64_t h0);
  // As RunEngine::cftp.
  rt_status cftp(DmSampler& s, int a0, int n, const std::vector<std::vector<RunEngine::Epoch>>& epochs,
                 int64_t first_sweeps, uint64_t fast_seed, int* attempts_run, bool* coalesced);
  rt_status check_error(DmSampler& s);
};

}  // namespace rt
