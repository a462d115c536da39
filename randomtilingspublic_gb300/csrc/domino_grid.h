// Grid engine of the domino sweep (see domino_grid.cu).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>
#include <vector>

#include "domino_rules.h"
#include "domino_runs.h"
#include "rt_internal.h"

namespace rt {

struct DmSampler;

constexpr int kGrMaxBands = 160;
constexpr int kGrTeams = 4;  // attempts of a coupling from the past side by side

struct GrPlan {
  bool ok = false;
  std::string why;
  int bands = 0, slots = 0, draw_warps = 0, update_warps = 0, per_lane = 1;  // slots: words per draw warp
  int row_start[kGrMaxBands + 1] = {};
  int windows[2 * kGrMaxBands] = {};  // each band's first window word and window words
  int xlo = 0, xn = 0;                // first word and words of an exchange row
  int64_t words = 0, draw_cells = 0;
  size_t smem_bytes = 0;
  int depth = 1;            // runs between exchanges (1: k_grid, more: k_deep)
  int first = 0, last = 0;  // k_deep: first and last row of any band
  int threads() const { return 32 * (draw_warps + update_warps); }
  // From each colour-array row's first and last flip-candidate column (-1: none).
  void build(const std::vector<int>& lo, const std::vector<int>& hi, int N, int nch, bool fast, int bands_max);
  bool build_deep(const std::vector<int>& lo, const std::vector<int>& hi, int N, int nch, bool fast, int bands_max, int runs);
};

struct GridEngine {
  GrPlan plan;
  bool ready = false;
  int nch = 0, bands_max = 0, sms = 0;  // the plan's most bands: those asked for, else the device's SMs
  void* kernel = nullptr;
  cudaStream_t stream = nullptr;
  int* d_rows = nullptr;       // the plan's row_start and windows, then the error word
  uint64_t* d_xbuf = nullptr;  // tagged words
  size_t xbuf_bytes = 0;
  uint32_t* d_runs = nullptr;
  int64_t runs_cap = 0;
  bool pending_error_check = false;
  int* d_team = nullptr;         // couplings: {smallest attempt that coalesced, error, -, -, [k] bands that differ, done}
  uint8_t* d_teams = nullptr;    // two chains of each attempt side by side
  uint64_t* d_xteams = nullptr;  // their tagged words

  ~GridEngine();
  rt_status prepare(DmSampler& s);
  // Is this the plan for `asked` bands (0: one per SM)?
  bool serves(int asked) const { return bands_max == (asked > 0 ? std::min(asked, sms) : sms); }
  rt_status launch(DmSampler& s, const uint8_t* colours_host, int64_t steps, uint64_t fast_seed, int64_t h0);
  // As RunEngine::cftp, attempts [a0, a0 + n) side by side (n <= kGrTeams), where depth > 1.
  rt_status cftp(DmSampler& s, int a0, int n, const std::vector<std::vector<RunEngine::Epoch>>& epochs,
                 int64_t first_sweeps, uint64_t fast_seed, int* attempts_run, bool* coalesced);
  rt_status check_error(DmSampler& s);
};

}  // namespace rt
