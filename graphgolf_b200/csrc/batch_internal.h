// batch_internal.h -- the batch object shared by the translation units that
// enqueue batch evaluations (the batch API and the device annealing engine).
// Not part of the public C ABI.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include <vector>

#include "apsp_kernel.cuh"

struct ggb_batch {
  int device = -1;
  int sms = 0;
  size_t l2 = 0;
  int n = 0;
  std::vector<int> N, bn, grp, d;
  std::vector<int> by_size;          // graphs in order of N: the order of their adjacencies
  std::vector<long long> off;        // ints; a multiple of 8 (16-byte boundaries in d_adj16 as well)
  long long adj_ints = 0;
  int* d_adj = nullptr;
  int* h_adj = nullptr;              // pinned staging for ggb_batch_eval
  uint16_t* d_adj16 = nullptr;       // 16-bit ids on their way to d_adj (every N <= 65536)
  ggb::BatchGraph* d_graphs = nullptr;
  ggb::BatchOut* d_out = nullptr;
  ggb::BatchOut* h_out = nullptr;
  // the plan
  int R = 0, T = 0, n_teams = 0, ctas = 0;
  std::vector<int> team_start, team_list;
  std::vector<long long> team_off, team_cells;
  ggb::ApspCtrl* d_ctrl = nullptr;   // [max_teams]
  ggb::ApspCtrl* h_ctrl = nullptr;
  int* d_tstart = nullptr;           // [max_teams + 1]
  int* d_tlist = nullptr;            // [n]
  long long* d_toff = nullptr;       // [max_teams]
  long long* d_tcells = nullptr;     // [max_teams]
  uint4* d_scratch = nullptr;
  size_t cap_scratch = 0;            // uint4
  // full-row stamps of the plan (4096-source windows, some degree <= 16):
  // team t's slice starts at team_soff[t]; stamp_ints == 0 when unused
  std::vector<long long> team_soff;
  long long stamp_ints = 0;
  long long* d_tsoff = nullptr;      // [max_teams]
  unsigned* d_stamps = nullptr;
  size_t cap_stamps = 0;             // unsigned
  // The automatic plan splits the graphs over three kernels: small ones on
  // shared-memory windows (apsp_slice.cuh), mid-size ones level by level on
  // teams (apsp_levels.cuh), the rest on teams of windows as a fixed plan has
  // them all.
  bool split = false;
  // What ggb_batch_get_plan reports for the automatic plan (0: the cost model's
  // fixed plan), set by the autotuner
  int best_fixed_R = 0, best_fixed_T = 0;
  struct SliceLaunch { int words, threads, first, items; size_t smem; };
  std::vector<SliceLaunch> slices;          // by shared memory, so that small graphs share an SM
  std::vector<ggb::SliceItem> slice_items;
  std::vector<int> slice_words;             // per graph: row words of its slices, 0: not a slice graph
  ggb::SliceItem* d_items = nullptr;  size_t cap_items = 0;
  ggb::ApspCtrl* d_records = nullptr;       // [n], all zero between launches
  int lT = 0, l_teams = 0;                  // level-by-level teams (l_teams == 0: none)
  size_t l_smem = 0;
  std::vector<int> l_start, l_list;
  std::vector<long long> l_off, l_cells;
  int* d_lint = nullptr;      size_t cap_lint = 0;       // l_start, l_list
  long long* d_lll = nullptr; size_t cap_lll = 0;        // l_off, l_cells
  ggb::ApspCtrl* d_lctrl = nullptr;         // [2 * max_teams]: the teams, then the window launch behind them
  ggb::ApspCtrl* h_lctrl = nullptr;
  unsigned long long* d_lists = nullptr; size_t cap_lists = 0;
  int occ[6] = {0, 0, 0, 0, 0, 0};   // co-resident batch CTAs per SM, per log2(R)
  int max_teams = 0;                 // largest CTA count of any plan
  long long timeout_ns = 2000000000LL;
  cudaStream_t stream = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  cudaStream_t copies = nullptr;     // uploads beside running kernels (eval_parts)
  cudaEvent_t arrived = nullptr;
  cudaEvent_t ev[6] = {};            // around each of the last evaluation's `timed` launches
  int timed = 0;
  bool pending = false;
  // Graph i is patch_base with patch[i] applied instead of its own adjacency
  // (device; only while every graph is on slices, see all_slices).
  const int* patch_base = nullptr;
  const ggb::Swap* patch = nullptr;
  // Kernels of one evaluation: the level-by-level launch and the windows behind
  // it, the window teams, the slices.
  int kernels() const { return (l_teams > 0 ? 2 : 0) + (n_teams > 0 ? 1 : 0) + (int)slices.size(); }
  bool all_slices() const { return split && l_teams == 0 && n_teams == 0 && !slice_items.empty(); }
  const int* stop = nullptr;         // device flag: the launch does nothing while it is non-zero
  int* sticky = nullptr;             // device flag: first error code of any launch (set, never cleared)
};

namespace ggb {

// The parts of an evaluation, in the order batch_enqueue() takes them.
enum { kPartClear = 1, kPartLevels = 2, kPartWindows = 4, kPartSlices = 8, kPartAll = 15 };

// Enqueues one evaluation of the batch's device adjacency on `st` (zeroing
// of the control blocks and results, then the kernels), or some parts of it;
// usable inside a stream capture.
int batch_enqueue(ggb_batch* b, cudaStream_t st, int parts = kPartAll);

}  // namespace ggb
