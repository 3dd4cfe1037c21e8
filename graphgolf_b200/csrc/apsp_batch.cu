// apsp_batch.cu -- exact APSP of many graphs, of uneven sizes, in one launch.
//
// A batch is a fixed list of graphs (nodes, based_nodes, groups, degree each)
// whose adjacency arrays sit packed in one device buffer.  A fixed plan
// evaluates all of them in one cooperative launch of apsp_batch_kernel: the
// launch's CTAs form teams of `team_ctas` CTAs, the graphs are dealt to the
// teams longest-first (each to the team with the least modelled work so far),
// and every team runs its graphs' source windows exactly as the single-graph
// kernel runs one graph's, with a barrier of its own.  The automatic plan
// (plan_split) sends small graphs to shared-memory windows and mid-size ones to
// level-by-level teams first, each in launches of their own.  Per graph the
// answer is the one ggb_eval_general gives (general/evaluation.c:153-263 per
// graph); the plan changes only the time.
//
// The launches (with the memsets of their control blocks) are captured once per
// plan in a CUDA graph and replayed, so a step of a batched annealing loop costs
// one graph launch.  ggb_batch_autotune times the automatic plan and every
// feasible (window width, team size) pair on the batch's current adjacency and
// keeps the fastest.  The mixed workload of 257 graphs (512 to 16384 vertices,
// d = 12): 4.6 ms of kernels with the automatic plan, 5.7 ms with the best fixed
// one.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <numeric>
#include <queue>
#include <vector>

#include "../../include/graphgolf_b200.h"
#include "apsp_kernel.cuh"
#include "apsp_levels.cuh"
#include "apsp_slice.cuh"
#include "batch_internal.h"
#include "core_internal.h"

using ggb::core_fail;

#define BCUDA(call)                                                                                  \
  do {                                                                                               \
    cudaError_t e_ = (call);                                                                         \
    if (e_ != cudaSuccess)                                                                           \
      return core_fail(GGB_ECUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, \
                       __LINE__);                                                                    \
  } while (0)

namespace {

constexpr int kMaxR = 32;   // widest window of the batch kernel: 4096 sources

const void* batch_kernel_for(int R) {
  switch (R) {
    case 1: return (const void*)ggb::apsp_batch_kernel<1>;
    case 2: return (const void*)ggb::apsp_batch_kernel<2>;
    case 4: return (const void*)ggb::apsp_batch_kernel<4>;
    case 8: return (const void*)ggb::apsp_batch_kernel<8>;
    case 16: return (const void*)ggb::apsp_batch_kernel<16>;
    case 32: return (const void*)ggb::apsp_batch_kernel<32>;
    default: return nullptr;
  }
}

size_t batch_smem_for(int R) {
  switch (R) {
    case 1: return ggb::apsp_smem_bytes<1>();
    case 2: return ggb::apsp_smem_bytes<2>();
    case 4: return ggb::apsp_smem_bytes<4>();
    case 8: return ggb::apsp_smem_bytes<8>();
    case 16: return ggb::apsp_smem_bytes<16>();
    case 32: return ggb::apsp_smem_bytes<32>();
    default: return 0;
  }
}

int log2i(int x) {
  int r = 0;
  while ((1 << r) < x) ++r;
  return r;
}

template <typename T>
int dev_alloc(T** p, size_t n) {
  if (cudaMalloc(p, std::max<size_t>(n, 1) * sizeof(T)) != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    return core_fail(GGB_ENOMEM, "cudaMalloc of %zu bytes failed", n * sizeof(T));
  }
  return GGB_OK;
}

}  // namespace

namespace {

template <typename T>
int regrow(T** p, size_t* cap, size_t n) {
  if (n <= *cap && *p) return GGB_OK;
  cudaFree(*p);
  *p = nullptr;
  *cap = 0;
  const int rc = dev_alloc(p, n);
  if (rc == GGB_OK) *cap = n;
  return rc;
}

// Modelled seconds of one graph on a team of T CTAs with windows of 128*R
// sources: per window the two-hop seeding plus about five dense sweeps of
// d gathered 16R-byte rows per vertex, each sweep at least one memory round
// trip and one team barrier.  A CTA gathers about 1e11 bytes/s from L2.
double graph_cost(int N, int d, int nsrc, int R, int T) {
  const double W = 128.0 * R;
  const double nwin = std::ceil(nsrc / W);
  const double dd = std::max(d, 1);
  const double rate = 1.0e11 * T;
  const double bar = 1.5e-6 + 0.01e-6 * T;
  const double seed = (double)N * (dd + dd * dd) * 4.0 / rate + bar + 1.5e-6;
  const double level = std::max((double)N * (dd * (16.0 * R + 4.0) + 32.0 * R) / rate, 1.5e-6) + bar;
  return nwin * (seed + 5.0 * level);
}

// Teams of *T CTAs for n graphs; *T is cut to the CTAs there are.
int team_count(const ggb_batch* b, int n, int R, int* T) {
  const int ctas_max = b->occ[log2i(R)] * b->sms;
  *T = std::max(1, std::min(*T, ctas_max));
  return std::max(1, std::min(ctas_max / *T, n));
}

// Deals the graphs to the teams (longest first, each to the least loaded
// team); returns the modelled makespan and in *spill the teams' working set over
// 60 % of L2, from where the gathers begin to spill to HBM, in units of L2.
double deal(const ggb_batch* b, const std::vector<int>& ids, int R, int T, std::vector<std::vector<int>>* teams,
            double* spill) {
  const int n_teams = team_count(b, (int)ids.size(), R, &T);
  std::vector<double> cost(b->n);
  for (int i : ids) cost[i] = graph_cost(b->N[i], b->d[i], b->bn[i], R, T);
  std::vector<int> order(ids);
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return cost[x] > cost[y]; });
  using Load = std::pair<double, int>;
  std::priority_queue<Load, std::vector<Load>, std::greater<Load>> pq;
  for (int t = 0; t < n_teams; ++t) pq.push({0.0, t});
  teams->assign(n_teams, {});
  double makespan = 0.0;
  for (int i : order) {
    Load l = pq.top();
    pq.pop();
    l.first += cost[i];
    (*teams)[l.second].push_back(i);
    makespan = std::max(makespan, l.first);
    pq.push(l);
  }
  // the teams running at once: each team's adjacency and two matrices
  double ws = 0.0;
  for (const auto& l : *teams) {
    long long mx = 0;
    for (int i : l) mx = std::max<long long>(mx, (long long)b->N[i] * (b->d[i] * 4 + 32 * R));
    ws += (double)mx;
  }
  *spill = std::max(0.0, ws / (double)b->l2 - 0.6);
  return makespan;
}

// Deals the graphs to the teams and returns the modelled makespan with the price
// of a working set past L2; fills the plan arrays when `keep`.  (The price is steep:
// with a mild one for large graphs 64 graphs of 10 000 vertices, d = 3 took 13.6 ms, 8.1
// with this one, and 16 of 20 000 12.4, 8.7.)
double make_plan(ggb_batch* b, const std::vector<int>& ids, int R, int T, bool keep) {
  std::vector<std::vector<int>> lists;
  double spill = 0.0;
  const double makespan = deal(b, ids, R, T, &lists, &spill) * (1.0 + 1.5 * std::min(1.0, spill / 0.6));
  if (!keep) return makespan;
  const int n_teams = team_count(b, (int)ids.size(), R, &T);
  b->R = R;
  b->T = T;
  b->n_teams = n_teams;
  b->ctas = n_teams * T;
  b->team_start.assign(n_teams + 1, 0);
  b->team_list.clear();
  b->team_off.assign(n_teams, 0);
  b->team_cells.assign(n_teams, 0);
  long long off = 0;
  for (int t = 0; t < n_teams; ++t) {
    b->team_start[t] = (int)b->team_list.size();
    long long cells = 1;
    for (int i : lists[t]) {
      b->team_list.push_back(i);
      cells = std::max<long long>(cells, (long long)b->N[i] * R);
    }
    b->team_off[t] = off;
    b->team_cells[t] = cells;
    off += 2 * cells;
  }
  b->team_start[n_teams] = (int)b->team_list.size();
  // Stamps pay where the stamping sweeps run: 4096-source windows, degree <= 16.
  b->team_soff.assign(n_teams, 0);
  b->stamp_ints = 0;
  bool stamping = false;
  for (int i : ids) stamping = stamping || (R == 32 && b->d[i] <= 16);
  if (stamping) {
    for (int t = 0; t < n_teams; ++t) {
      int mx = 0;
      for (int k = b->team_start[t]; k < b->team_start[t + 1]; ++k) mx = std::max(mx, b->N[b->team_list[k]]);
      b->team_soff[t] = b->stamp_ints;
      b->stamp_ints += (mx + 31) / 32 * 32;   // each slice on a 128-byte boundary
    }
  }
  return makespan;
}

int drop_graph(ggb_batch* b) {
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  b->exec = nullptr;
  b->graph = nullptr;
  return GGB_OK;
}

// Uploads the windows plan made by make_plan(keep = true).
int upload_windows(ggb_batch* b) {
  if (int rc = regrow(&b->d_scratch, &b->cap_scratch, (size_t)(b->team_off.back() + 2 * b->team_cells.back())))
    return rc;
  BCUDA(cudaMemcpyAsync(b->d_tstart, b->team_start.data(), b->team_start.size() * sizeof(int),
                        cudaMemcpyHostToDevice, b->stream));
  BCUDA(cudaMemcpyAsync(b->d_tlist, b->team_list.data(), b->team_list.size() * sizeof(int),
                        cudaMemcpyHostToDevice, b->stream));
  BCUDA(cudaMemcpyAsync(b->d_toff, b->team_off.data(), b->team_off.size() * sizeof(long long),
                        cudaMemcpyHostToDevice, b->stream));
  BCUDA(cudaMemcpyAsync(b->d_tcells, b->team_cells.data(), b->team_cells.size() * sizeof(long long),
                        cudaMemcpyHostToDevice, b->stream));
  if (b->stamp_ints > 0) {
    if ((size_t)b->stamp_ints > b->cap_stamps) {
      if (b->d_stamps) cudaFree(b->d_stamps);
      b->d_stamps = nullptr;
      b->cap_stamps = 0;
      int rc = dev_alloc(&b->d_stamps, (size_t)b->stamp_ints);
      if (rc) return rc;
      b->cap_stamps = (size_t)b->stamp_ints;
    }
    BCUDA(cudaMemcpyAsync(b->d_tsoff, b->team_soff.data(), b->team_soff.size() * sizeof(long long),
                          cudaMemcpyHostToDevice, b->stream));
  }
  BCUDA(cudaStreamSynchronize(b->stream));
  return GGB_OK;
}

// ---- the automatic plan ----------------------------------------------------------

constexpr size_t kSliceSmemMax = 224 * 1024;

std::vector<int> all_graphs(const ggb_batch* b) {
  std::vector<int> ids(b->n);
  std::iota(ids.begin(), ids.end(), 0);
  return ids;
}

// Modelled seconds of one graph level by level on T CTAs (measured at
// N = 16384, d = 12: 11 ms / T + 70 us).
double levels_cost(int N, int d, int T) {
  const double x = N / 16384.0;
  return 11.0e-3 * x * x * (d + 1) / 13.0 / T + 70.0e-6;
}

// Slices for the graphs of `ids`: rows of 32 sources while every window then
// has an SM to itself (one step of an annealer), else of 64 (fewer stagings and
// fewer wavefronts a source).  Launches by shared memory, largest graphs first.
void plan_slices(ggb_batch* b, const std::vector<int>& ids) {
  b->slices.clear();
  b->slice_items.clear();
  long long w32 = 0;
  for (int i : ids) w32 += (b->bn[i] + 31) / 32;
  const int words = w32 <= b->sms ? 1 : 2, width = 32 * words;
  long long windows = 0;
  for (int i : ids) windows += (b->bn[i] + width - 1) / width;
  const int per = (int)std::max<long long>(1, windows / (8LL * b->sms));   // windows a CTA
  auto smem = [&](int i) { return ggb::slice_smem_bytes((b->N[i] + 31) / 32 * 32, words, (b->d[i] + 1) / 2); };
  std::vector<int> order(ids);
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return smem(x) > smem(y); });
  const size_t limit[3] = {72 * 1024, 110 * 1024, kSliceSmemMax};   // three, two CTAs or one an SM
  int bucket = -1;
  for (int i : order) {
    const size_t sm = smem(i);
    const int k = sm <= limit[0] ? 0 : sm <= limit[1] ? 1 : 2;
    if (k != bucket) {
      b->slices.push_back({words, 0, (int)b->slice_items.size(), 0, sm});
      bucket = k;
    }
    auto& launch = b->slices.back();
    const int np = (b->N[i] + 31) / 32 * 32;
    launch.threads = std::max(launch.threads, std::min(np, k == 0 ? 640 : k == 1 ? 768 : 1024));
    const int nw = (b->bn[i] + width - 1) / width, ctas = (nw + per - 1) / per;
    for (int t = 0; t < nw; t += per) b->slice_items.push_back({i, t, std::min(nw, t + per), ctas});
    launch.items = (int)b->slice_items.size() - launch.first;
    b->slice_words[i] = words;
  }
}

void model_choice(ggb_batch* b, const std::vector<int>& ids, int* R, int* T);

// ---- slices or teams -------------------------------------------------------------
// Two models of the kernels' time in us, for random graphs, fitted to 800 batches of
// 2 to 256 graphs of 64 to 7000 vertices, equal and mixed, d = 3 to 24, each timed both
// ways (80 % of the predictions within 15 % for slices, 11 % for teams).  The slices
// are taken while theirs is under 0.92 of the teams': half a percent behind the
// best of both on average, 7 % slower than teams at worst, 28 % than slices.  Slices
// alone took up to 1.7 times as long as teams (64 graphs of 2000 vertices, d = 8: 225
// us, 147), teams alone up to 4 times as long as slices (200 vertices: 12 us, 42).

// Levels of a random d-regular graph of N vertices: its share q of unreached
// pairs falls like d (d-1)^(k-1) / N at first, then q -> q^(d-1).
double expected_levels(int N, int d) {
  if (d < 3) return N;
  double lq = std::log(std::max(1e-300, 1.0 - std::min(0.999999, (1.0 + d) / N)));
  int k = 1;
  for (; k < 200 && 2.0 * std::log((double)N) + lq > std::log(2.0); ++k)
    lq = lq < -1e-12 ? lq * (d - 1) : std::log1p(-std::min(0.999999, std::pow(d - 1.0, k) * d / N));
  return k;
}

// The slices planned in b: what the windows gather (in fours, and less at high
// degrees, whose rows are full early), barriers and staging, by how many CTAs share
// an SM; the last window, and the launch.
double slices_us(const ggb_batch* b) {
  constexpr double kGather[3] = {1.9e-4, 1.5e-4, 0.73e-4}, kLevel[3] = {0.035, 0.0, 1.46};
  double us = 0.0;
  for (const auto& l : b->slices) {
    const int k = l.smem <= 72 * 1024 ? 0 : l.smem <= 110 * 1024 ? 1 : 2;
    const double share = std::min((double)(3 - k), std::max(1.0, (double)l.items / b->sms));
    double sum = 0.0, last = 0.0, levels = 0.0, row = 0.0;
    for (int t = l.first; t < l.first + l.items; ++t) {
      const auto& it = b->slice_items[t];
      const int N = b->N[it.graph], pairs = (b->d[it.graph] + 1) / 2, windows = it.end - it.first;
      if (it.first == 0) {   // a graph's first item
        levels = expected_levels(N, b->d[it.graph]);
        row = (levels - 1.0) * std::pow(4.0 * ((pairs + 1) / 2), 0.7) + 0.5 * levels * pairs;
      }
      const double gathers = windows * N * row * (l.words == 1 ? 0.6 : 1.0);
      sum += gathers * kGather[k] + windows * levels * kLevel[k] + 4.6e-4 * N * pairs;
      last = std::max(last, gathers * 2.5e-5 * share + 0.23 * windows * levels);
    }
    us += sum / b->sms + last + 9.2;
  }
  return us;
}

// The graphs of ids on window teams, as the cost model would plan them: the
// gathered bytes (rows of 64 bytes and less are slower, and high degrees skip more of them),
// barriers, seeding (slower where rows are not a multiple of four ids), and the gathers
// that spill out of L2.
double windows_us(ggb_batch* b, const std::vector<int>& ids) {
  int R = 1, T = 1;
  model_choice(b, ids, &R, &T);
  std::vector<std::vector<int>> teams;
  double spill = 0.0, us = 0.0;
  deal(b, ids, R, T, &teams, &spill);
  team_count(b, (int)ids.size(), R, &T);
  for (const auto& team : teams) {
    double gathers = 0.0, rest = 0.0;
    for (int i : team) {
      const double N = b->N[i], d = std::max(b->d[i], 1), levels = expected_levels(b->N[i], b->d[i]);
      const double windows = std::ceil(b->bn[i] / (128.0 * R));
      gathers += windows * (levels - 1.0) * N * (std::pow(d, 0.7) + 2.0) * 16.0 * R / T;
      rest += windows * (3.0 * levels + 1.1 + (b->d[i] % 4 ? 1.3e-4 : 4.4e-5) * N * (d + d * d) * 4.0 / T);
    }
    us = std::max(us, gathers * ((R <= 4 ? 2.4e-5 : 1.5e-5) + 1.9e-4 * std::min(spill, 2.0)) + rest);
  }
  return us + 9.5;
}

// Level-by-level teams for the graphs of `ids`: the team size with the least
// modelled makespan.
void plan_levels(ggb_batch* b, const std::vector<int>& ids) {
  b->l_teams = 0;
  if (ids.empty()) return;
  double best = 1e300;
  for (int T : {148, 74, 49, 37, 29, 24, 21, 18, 16}) {
    T = std::min(T, b->sms);
    const int n_teams = std::max(1, std::min(b->sms / T, (int)ids.size()));
    std::vector<int> order(ids);
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
      return levels_cost(b->N[x], b->d[x], T) > levels_cost(b->N[y], b->d[y], T);
    });
    std::vector<double> load(n_teams, 0.0);
    std::vector<std::vector<int>> lists(n_teams);
    for (int i : order) {
      const int t = (int)(std::min_element(load.begin(), load.end()) - load.begin());
      load[t] += levels_cost(b->N[i], b->d[i], T);
      lists[t].push_back(i);
    }
    const double m = *std::max_element(load.begin(), load.end());
    if (m >= best * 0.999) continue;
    best = m;
    b->lT = T;
    b->l_teams = n_teams;
    b->l_start.assign(1, 0);
    b->l_list.clear();
    b->l_off.clear();
    b->l_cells.clear();
    b->l_smem = 0;
    long long off = 0;
    for (const auto& l : lists) {
      long long cells = 0;
      for (int i : l) {
        b->l_list.push_back(i);
        cells = std::max<long long>(cells, (long long)b->N[i] * ggb::levels_pitch(b->N[i]));
        b->l_smem = std::max(b->l_smem, ggb::levels_smem_bytes(b->N[i], b->d[i]));
      }
      b->l_start.push_back((int)b->l_list.size());
      b->l_off.push_back(off);
      b->l_cells.push_back(cells);
      off += 2 * cells;
    }
  }
}

int upload_split(ggb_batch* b) {
  int rc;
  if (!b->slice_items.empty()) {
    if ((rc = regrow(&b->d_items, &b->cap_items, b->slice_items.size()))) return rc;
    BCUDA(cudaMemcpyAsync(b->d_items, b->slice_items.data(), b->slice_items.size() * sizeof(ggb::SliceItem),
                          cudaMemcpyHostToDevice, b->stream));
  }
  if (b->l_teams > 0) {
    const size_t nt = (size_t)b->l_teams;
    const size_t words = ggb::kLevelsListWords + (ggb::kLevelsCounters + 1) / 2;
    if ((rc = regrow(&b->d_lint, &b->cap_lint, nt + 1 + b->l_list.size())) ||
        (rc = regrow(&b->d_lll, &b->cap_lll, 2 * nt)) || (rc = regrow(&b->d_lists, &b->cap_lists, nt * words)) ||
        (rc = regrow(&b->d_scratch, &b->cap_scratch, (size_t)(b->l_off.back() + 2 * b->l_cells.back()))))
      return rc;
    BCUDA(cudaMemcpyAsync(b->d_lint, b->l_start.data(), (nt + 1) * sizeof(int), cudaMemcpyHostToDevice, b->stream));
    BCUDA(cudaMemcpyAsync(b->d_lint + nt + 1, b->l_list.data(), b->l_list.size() * sizeof(int),
                          cudaMemcpyHostToDevice, b->stream));
    BCUDA(cudaMemcpyAsync(b->d_lll, b->l_off.data(), nt * sizeof(long long), cudaMemcpyHostToDevice, b->stream));
    BCUDA(cudaMemcpyAsync(b->d_lll + nt, b->l_cells.data(), nt * sizeof(long long), cudaMemcpyHostToDevice,
                          b->stream));
  }
  BCUDA(cudaStreamSynchronize(b->stream));
  return GGB_OK;
}

// No kernels: nothing of a plan whose buffers could not be had is launched.
void no_plan(ggb_batch* b) {
  b->slices.clear();
  b->slice_items.clear();
  b->slice_words.assign(b->n, 0);
  b->l_teams = 0;
  b->n_teams = b->ctas = 0;
  b->stamp_ints = 0;
}

// The automatic plan.  Falls back to one windows plan for all graphs when the
// workspace of the other kernels cannot be had.
int plan_split(ggb_batch* b) {
  drop_graph(b);
  b->split = true;
  b->best_fixed_R = b->best_fixed_T = 0;
  b->slice_words.assign(b->n, 0);
  // Slices: as for a single graph (plan_slice in apsp_core.cu) while every
  // window has an SM to itself; with more windows than that up to fewer gathers a
  // level, and where slices_us and windows_us say so.
  // Level by level: from 8193 vertices like a single graph; with teams enough
  // to hide its barriers from 4500 (52 graphs of 4096 to 8192 vertices, d = 12:
  // 1198 us, 1309 from 6000 on, 1462 as windows).  Degree 4 has more levels, and
  // windows of 4096 sources fit some sizes well (level by level / windows, 64 graphs): 7000
  // 3103 / 2807, 8000 3696 / 2864, 8600 4139 / 6500, 9000 5081 / 7150, 10000 5843 /
  // 5435, 11000 6905 / 7870.
  long long w32 = 0;
  int over = 0;
  for (int i = 0; i < b->n; ++i) {
    w32 += (b->bn[i] + 31) / 32;
    over += b->N[i] > 4500;
  }
  const long long most = w32 <= b->sms ? 45000 : 30000;
  const int from = over >= 8 ? 4500 : 8192;
  std::vector<int> small, mid, rest;
  for (int i = 0; i < b->n; ++i) {
    const int N = b->N[i], d = b->d[i];
    const size_t smem = ggb::slice_smem_bytes((N + 31) / 32 * 32, 2, (d + 1) / 2);
    if ((long long)N * (d + 1) <= most && N <= ggb::kSliceMaxN && smem <= kSliceSmemMax) small.push_back(i);
    else if (b->grp[i] == 1 && d >= 4 && d <= 32 && N > from && N <= 22000) mid.push_back(i);
    else rest.push_back(i);
  }
  bool levels_pay = from == 8192;
  for (int i : mid) levels_pay = levels_pay || b->d[i] > 4 || b->N[i] > 10500 || (b->N[i] > 8192 && b->N[i] <= 9500);
  if (!levels_pay) {
    rest.insert(rest.end(), mid.begin(), mid.end());
    mid.clear();
  }
  // The kernels follow one another and each has its tail.  With graphs for the
  // level-by-level teams the split pays (1.0 to 2.1 times); with small
  // graphs beside window teams only it does not always (29 graphs of 109 to 5162
  // vertices, d = 15: 625 us, 529 on teams alone; 89 of 86 to 4844, d = 14: 1050,
  // 925; 16 of 540 to 4897, d = 15: 395, 556): those stay on teams.
  if (mid.empty() && !rest.empty()) {
    rest = all_graphs(b);
    small.clear();
  }
  plan_slices(b, small);
  long long windows = 0;
  for (int i : small) windows += (b->bn[i] + 63) / 64;
  if (windows > 2LL * b->sms && slices_us(b) > 0.92 * windows_us(b, small)) {
    rest.insert(rest.end(), small.begin(), small.end());
    plan_slices(b, {});
    b->slice_words.assign(b->n, 0);
  }
  plan_levels(b, mid);
  int rc = upload_split(b);
  if (rc == GGB_ENOMEM) {
    no_plan(b);
    rest = all_graphs(b);
    rc = GGB_OK;
  }
  b->n_teams = b->ctas = 0;
  b->stamp_ints = 0;
  if (!rc && !rest.empty()) {
    int R = 1, T = 1;
    model_choice(b, rest, &R, &T);
    make_plan(b, rest, R, T, true);
    rc = upload_windows(b);
  }
  if (rc) no_plan(b);
  return rc;
}

// One windows plan for all graphs.
int plan_fixed(ggb_batch* b, int R, int T) {
  drop_graph(b);
  no_plan(b);
  b->split = false;
  make_plan(b, all_graphs(b), R, T, true);
  const int rc = upload_windows(b);
  if (rc) no_plan(b);
  return rc;
}

ggb::BatchArgs batch_args(const ggb_batch* b) {
  ggb::BatchArgs a;
  a.graphs = b->d_graphs;
  a.out = b->d_out;
  a.team_ctrl = b->d_ctrl;
  a.team_start = b->d_tstart;
  a.team_list = b->d_tlist;
  a.scratch = b->d_scratch;
  a.team_off = b->d_toff;
  a.team_cells = b->d_tcells;
  a.timeout_ns = b->timeout_ns;
  a.stop = b->stop;
  a.sticky = b->sticky;
  a.n_teams = b->n_teams;
  a.team_ctas = b->T;
  a.stamps = b->stamp_ints > 0 ? b->d_stamps : nullptr;
  a.team_soff = b->stamp_ints > 0 ? b->d_tsoff : nullptr;
  return a;
}

}  // namespace

namespace {

int coop(const void* fn, int ctas, size_t smem, void** params, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(ggb::kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  BCUDA(cudaLaunchKernelExC(&cfg, fn, params));
  return GGB_OK;
}

}  // namespace

// The launches themselves: the largest work first.  The slices clear nothing
// and need nothing cleared; the teams' control blocks and results are zeroed
// (kPartClear, before any part's results are written).
int ggb::batch_enqueue(ggb_batch* b, cudaStream_t st, int parts) {
  int rc;
  if ((parts & kPartClear) && (b->l_teams > 0 || b->n_teams > 0 || b->slices.empty()))
    BCUDA(cudaMemsetAsync(b->d_out, 0, (size_t)b->n * sizeof(ggb::BatchOut), st));
  if ((parts & kPartLevels) && b->l_teams > 0) {
    const size_t words = ggb::kLevelsListWords + (ggb::kLevelsCounters + 1) / 2;
    BCUDA(cudaMemsetAsync(b->d_lctrl, 0, (size_t)2 * b->l_teams * sizeof(ggb::ApspCtrl), st));
    BCUDA(cudaMemset2DAsync(b->d_lists + ggb::kLevelsListWords, words * 8, 0, ggb::kLevelsCounters * sizeof(unsigned),
                            b->l_teams, st));
    ggb::BatchArgs a = batch_args(b);
    a.team_ctrl = b->d_lctrl;
    a.team_start = b->d_lint;
    a.team_list = b->d_lint + b->l_teams + 1;
    a.scratch = b->d_scratch;   // the launches of a batch follow one another: one scratch
    a.team_off = b->d_lll;
    a.team_cells = b->d_lll + b->l_teams;
    a.n_teams = b->l_teams;
    a.team_ctas = b->lT;
    a.stamps = nullptr;
    a.team_soff = nullptr;
    size_t w = words;
    void* params[] = {(void*)&a, (void*)&b->d_lists, (void*)&w};
    if ((rc = coop((const void*)ggb::apsp_batch_levels_kernel, b->l_teams * b->lT, b->l_smem, params, st))) return rc;
    // graphs that were not served: asymmetric ones, or with too many levels past the list
    a.behind = b->d_lctrl;
    a.team_ctrl = b->d_lctrl + b->l_teams;
    void* params2[] = {(void*)&a};
    if ((rc = coop(batch_kernel_for(32), b->l_teams * b->lT, batch_smem_for(32), params2, st))) return rc;
  }
  if ((parts & kPartWindows) && b->n_teams > 0) {
    BCUDA(cudaMemsetAsync(b->d_ctrl, 0, (size_t)b->n_teams * sizeof(ggb::ApspCtrl), st));
    if (b->stamp_ints > 0) BCUDA(cudaMemsetAsync(b->d_stamps, 0, (size_t)b->stamp_ints * sizeof(unsigned), st));
    ggb::BatchArgs args = batch_args(b);
    void* params[] = {(void*)&args};
    if ((rc = coop(batch_kernel_for(b->R), b->ctas, batch_smem_for(b->R), params, st))) return rc;
  }
  if (!(parts & kPartSlices)) return GGB_OK;
  for (const auto& l : b->slices) {
    if (l.words == 1)
      ggb::slice_batch_kernel<1><<<l.items, l.threads, l.smem, st>>>(b->d_graphs, b->d_items + l.first, b->d_records,
                                                                    b->d_out, b->patch_base, b->patch, b->stop,
                                                                    b->sticky);
    else
      ggb::slice_batch_kernel<2><<<l.items, l.threads, l.smem, st>>>(b->d_graphs, b->d_items + l.first, b->d_records,
                                                                    b->d_out, b->patch_base, b->patch, b->stop,
                                                                    b->sticky);
    BCUDA(cudaGetLastError());
  }
  return GGB_OK;
}

namespace {

int capture(ggb_batch* b) {
  if (b->exec) return GGB_OK;
  BCUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
  int rc = ggb::batch_enqueue(b, b->stream);
  cudaGraph_t gph = nullptr;
  const cudaError_t e = cudaStreamEndCapture(b->stream, &gph);
  if (rc) {
    if (gph) cudaGraphDestroy(gph);
    return rc;
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return core_fail(GGB_ECUDA, "capturing the batch launch failed: %s", cudaGetErrorString(e));
  }
  b->graph = gph;
  BCUDA(cudaGraphInstantiate(&b->exec, gph, 0));
  return GGB_OK;
}

int launch(ggb_batch* b, cudaStream_t st, bool use_graph) {
  BCUDA(cudaSetDevice(b->device));
  BCUDA(cudaEventRecord(b->ev[0], st));
  if (use_graph) {
    int rc = capture(b);
    if (rc) return rc;
    BCUDA(cudaGraphLaunch(b->exec, st));
  } else {
    int rc = ggb::batch_enqueue(b, st);
    if (rc) return rc;
  }
  BCUDA(cudaEventRecord(b->ev[1], st));
  b->timed = 1;
  ggb::core_add_launches(b->kernels());
  b->pending = true;
  return GGB_OK;
}

// What an upload needs first: every adjacency, and a staging buffer that feeds
// no earlier copy.
int check_upload(ggb_batch* b, const int* const* adj, cudaStream_t st) {
  BCUDA(cudaSetDevice(b->device));
  BCUDA(cudaStreamSynchronize(st));
  for (int i = 0; i < b->n; ++i)
    if ((size_t)b->N[i] * b->d[i] && !adj[i]) return core_fail(GGB_EINVAL, "batch graph %d: null adjacency", i);
  return GGB_OK;
}

// Uploads graphs by_size[from, to).  The copy into the pinned buffer is spread
// over the staging threads; each unit of 128 Ki ids or more is sent as soon as
// it is copied, as 16-bit ids when they fit (stage.cu).
int upload_range(ggb_batch* b, const int* const* adj, int from, int to, cudaStream_t st) {
  if (from >= to) return GGB_OK;
  const size_t lo = (size_t)b->off[b->by_size[from]];
  const size_t hi = to < b->n ? (size_t)b->off[b->by_size[to]] : (size_t)b->adj_ints;
  std::vector<ggb::StageSeg> segs(to - from);
  for (int r = from; r < to; ++r) {
    const int i = b->by_size[r];
    segs[r - from] = {adj[i], (size_t)b->off[i] - lo, (size_t)b->N[i] * b->d[i]};
  }
  BCUDA(ggb::stage_upload_ids(b->device, b->h_adj + lo, b->d_adj16 ? b->d_adj16 + lo : nullptr, b->d_adj + lo,
                              segs.data(), to - from, hi - lo, st));
  return GGB_OK;
}

// Upload and launches of the automatic plan, kernel by kernel: each starts when
// its graphs have arrived, while the next one's are copied and sent.  257 graphs
// of 512 to 16384 vertices, d = 12 (27 MB of 16-bit ids): 6150 us a call, 6980
// with the whole upload first.
int eval_parts(ggb_batch* b, const int* const* adj) {
  std::vector<char> kind(b->n, 1);                 // 0 slices, 1 windows, 2 level by level
  for (int i = 0; i < b->n; ++i)
    if (b->slice_words[i]) kind[i] = 0;
  if (b->l_teams > 0)
    for (int i : b->l_list) kind[i] = 2;
  int end[3] = {0, 0, 0}, order[3] = {0, 1, 2};    // graphs up to by_size[end) are needed
  for (int r = 0; r < b->n; ++r) end[(int)kind[b->by_size[r]]] = r + 1;
  std::sort(order, order + 3, [&](int x, int y) { return end[x] < end[y]; });
  const int bits[3] = {ggb::kPartSlices, ggb::kPartWindows, ggb::kPartLevels};
  // a launch that has not been collected may still run on another stream, with
  // the same adjacencies, workspaces and control blocks (graph launches wait for
  // one another)
  if (b->pending) {
    BCUDA(cudaStreamWaitEvent(b->stream, b->ev[1], 0));
    BCUDA(cudaStreamWaitEvent(b->copies, b->ev[1], 0));
  }
  int rc = ggb::batch_enqueue(b, b->stream, ggb::kPartClear), at = 0;
  if (rc) return rc;
  b->timed = 0;
  for (int p : order) {
    if (end[p] == 0) continue;
    if ((rc = upload_range(b, adj, at, end[p], b->copies))) return rc;
    at = std::max(at, end[p]);
    BCUDA(cudaEventRecord(b->arrived, b->copies));
    BCUDA(cudaStreamWaitEvent(b->stream, b->arrived, 0));
    BCUDA(cudaEventRecord(b->ev[2 * b->timed], b->stream));
    if ((rc = ggb::batch_enqueue(b, b->stream, bits[p]))) return rc;
    BCUDA(cudaEventRecord(b->ev[2 * b->timed + 1], b->stream));
    b->timed += 1;
  }
  ggb::core_add_launches(b->kernels());
  b->pending = true;
  return GGB_OK;
}

// Sources per window of graph i under the current plan.
int window_bits_of(const ggb_batch* b, int i) {
  if (!b->split) return 128 * b->R;
  if (b->slice_words[i]) return 32 * b->slice_words[i];
  if (b->l_teams > 0 && std::find(b->l_list.begin(), b->l_list.end(), i) != b->l_list.end())
    return 128 * ggb::levels_pitch(b->N[i]);
  return 128 * b->R;
}

int collect(ggb_batch* b, cudaStream_t st, ggb_result* res) {
  BCUDA(cudaMemcpyAsync(b->h_out, b->d_out, (size_t)b->n * sizeof(ggb::BatchOut), cudaMemcpyDeviceToHost, st));
  if (b->n_teams > 0)
    BCUDA(cudaMemcpyAsync(b->h_ctrl, b->d_ctrl, (size_t)b->n_teams * sizeof(ggb::ApspCtrl), cudaMemcpyDeviceToHost,
                          st));
  if (b->l_teams > 0)
    BCUDA(cudaMemcpyAsync(b->h_lctrl, b->d_lctrl, (size_t)2 * b->l_teams * sizeof(ggb::ApspCtrl),
                          cudaMemcpyDeviceToHost, st));
  BCUDA(cudaStreamSynchronize(st));
  b->pending = false;
  auto report = [&](int error, int info, int gi) {
    if (error == ggb::kErrAdj)
      return core_fail(GGB_EADJ, "batch graph %d: adjacency entry outside [0, nodes)", gi);
    if (error == ggb::kErrTimeout)
      return core_fail(GGB_ETIMEOUT, "batch graph %d: a team-barrier wait ran out (CTA %d)", gi, info);
    return core_fail(GGB_ECUDA, "batch graph %d: device error code %d", gi, error);
  };
  // a team that failed left its graphs from the failing one on undone
  auto check_team = [&](const ggb::ApspCtrl& c, const int* list, int k0, int k1) {
    if (c.error == 0) return (int)GGB_OK;
    for (int k = k0; k < k1; ++k)
      if (!b->h_out[list[k]].done) return report(c.error, c.error_info, list[k]);
    return report(c.error, c.error_info, -1);
  };
  int rc;
  for (int t = 0; t < b->n_teams; ++t)
    if ((rc = check_team(b->h_ctrl[t], b->team_list.data(), b->team_start[t], b->team_start[t + 1]))) return rc;
  for (int t = 0; t < 2 * b->l_teams; ++t) {
    const int k = t % b->l_teams;
    // (a level-by-level team names the graph; those left to the windows are undone as well)
    if (t < b->l_teams && b->h_lctrl[t].error == ggb::kErrAdj)
      return report(ggb::kErrAdj, 0, b->h_lctrl[t].error_info);
    if ((rc = check_team(b->h_lctrl[t], b->l_list.data(), b->l_start[k], b->l_start[k + 1]))) return rc;
  }
  for (int i = 0; i < b->n; ++i)
    if (b->h_out[i].error) return report(b->h_out[i].error, 0, i);
  for (int i = 0; i < b->n; ++i) {
    const ggb::BatchOut& o = b->h_out[i];
    if (!o.done) return core_fail(GGB_ECUDA, "batch graph %d was not evaluated", i);
    if (!res) continue;
    ggb_partial p;
    p.diam = o.diam;
    p.disconnected = o.disconnected;
    p.sum = o.sum;
    p.levels = o.levels;
    p.windows = o.windows;
    p.window_bits = window_bits_of(b, i);
    p.dense_levels = o.dense_levels;
    rc = ggb_finish_general(b->N[i], &p, res + i);
    if (rc) return rc;
  }
  return GGB_OK;
}

void destroy(ggb_batch* b) {
  if (!b) return;
  if (b->device >= 0) cudaSetDevice(b->device);
  if (b->stream) cudaStreamSynchronize(b->stream);
  if (b->copies) cudaStreamSynchronize(b->copies);
  drop_graph(b);
  cudaFree(b->d_adj);
  cudaFree(b->d_adj16);
  cudaFreeHost(b->h_adj);
  cudaFree(b->d_graphs);
  cudaFree(b->d_out);
  cudaFreeHost(b->h_out);
  cudaFree(b->d_ctrl);
  cudaFreeHost(b->h_ctrl);
  cudaFree(b->d_tstart);
  cudaFree(b->d_tlist);
  cudaFree(b->d_toff);
  cudaFree(b->d_tcells);
  cudaFree(b->d_tsoff);
  cudaFree(b->d_stamps);
  cudaFree(b->d_scratch);
  cudaFree(b->d_items);
  cudaFree(b->d_records);
  cudaFree(b->d_lint);
  cudaFree(b->d_lll);
  cudaFree(b->d_lctrl);
  cudaFreeHost(b->h_lctrl);
  cudaFree(b->d_lists);
  for (auto& e : b->ev)
    if (e) cudaEventDestroy(e);
  if (b->stream) cudaStreamDestroy(b->stream);
  if (b->copies) cudaStreamDestroy(b->copies);
  if (b->arrived) cudaEventDestroy(b->arrived);
  cudaGetLastError();
  delete b;
}

int create(int n_graphs, const int* nodes, const int* based_nodes, const int* groups, const int* degree,
           ggb_batch* b) {
  b->n = n_graphs;
  b->N.assign(nodes, nodes + n_graphs);
  b->bn.assign(based_nodes, based_nodes + n_graphs);
  b->grp.assign(groups, groups + n_graphs);
  b->d.assign(degree, degree + n_graphs);
  b->off.resize(n_graphs);
  for (int i = 0; i < n_graphs; ++i) {
    const int Ni = nodes[i], bi = based_nodes[i], gi = groups[i], di = degree[i];
    if (Ni <= 0 || bi <= 0 || gi <= 0 || di < 0)
      return core_fail(GGB_EINVAL, "batch graph %d: nodes, based_nodes, groups must be > 0, degree >= 0", i);
    if ((long long)bi * gi != Ni)
      return core_fail(GGB_EINVAL, "batch graph %d: nodes (%d) != based_nodes*groups (%d*%d)", i, Ni, bi, gi);
    if ((long long)Ni * di > INT_MAX) return core_fail(GGB_EINVAL, "batch graph %d: nodes*degree too large", i);
  }
  // Adjacencies lie in order of size, so that the graphs of one kernel of the
  // automatic plan arrive together (eval_parts).
  b->by_size.resize(n_graphs);
  std::iota(b->by_size.begin(), b->by_size.end(), 0);
  std::stable_sort(b->by_size.begin(), b->by_size.end(), [&](int x, int y) { return nodes[x] < nodes[y]; });
  long long off = 0;
  for (int i : b->by_size) {
    b->off[i] = off;
    off += ((long long)nodes[i] * degree[i] + 7) / 8 * 8;
  }
  b->adj_ints = off;
  int dev = 0;
  BCUDA(cudaGetDevice(&dev));
  b->device = dev;
  BCUDA(cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, dev));
  int l2 = 0;
  BCUDA(cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev));
  b->l2 = (size_t)l2;
  for (int R = 1; R <= kMaxR; R *= 2) {
    int nb = 0;
    BCUDA(cudaFuncSetAttribute(batch_kernel_for(R), cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)batch_smem_for(R)));
    BCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, batch_kernel_for(R), ggb::kThreads,
                                                        batch_smem_for(R)));
    if (nb < 1) return core_fail(GGB_ECUDA, "batch kernel R=%d cannot be resident", R);
    b->occ[log2i(R)] = nb;
    b->max_teams = std::max(b->max_teams, nb * b->sms);
  }
  for (const void* k : {(const void*)ggb::slice_batch_kernel<1>, (const void*)ggb::slice_batch_kernel<2>,
                        (const void*)ggb::apsp_batch_levels_kernel})
    BCUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSliceSmemMax));
  if (const char* s = getenv("GGB_BARRIER_TIMEOUT_NS")) b->timeout_ns = atoll(s);
  BCUDA(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
  BCUDA(cudaStreamCreateWithFlags(&b->copies, cudaStreamNonBlocking));
  for (auto& e : b->ev) BCUDA(cudaEventCreate(&e));
  BCUDA(cudaEventCreateWithFlags(&b->arrived, cudaEventDisableTiming));
  int rc = dev_alloc(&b->d_adj, (size_t)b->adj_ints);
  if (rc) return rc;
  if (cudaHostAlloc(&b->h_adj, std::max<size_t>((size_t)b->adj_ints, 1) * sizeof(int), cudaHostAllocDefault) !=
      cudaSuccess) {
    cudaGetLastError();
    b->h_adj = nullptr;
    return core_fail(GGB_ENOMEM, "pinned staging of %lld ints failed", b->adj_ints);
  }
  // Graphs of at most 65536 vertices have 16-bit ids: uploads send them narrowed.
  if (*std::max_element(b->N.begin(), b->N.end()) <= 65536 &&
      (rc = dev_alloc(&b->d_adj16, (size_t)b->adj_ints)))
    return rc;
  if ((rc = dev_alloc(&b->d_graphs, (size_t)n_graphs))) return rc;
  if ((rc = dev_alloc(&b->d_out, (size_t)n_graphs))) return rc;
  const size_t mt = (size_t)b->max_teams;
  if ((rc = dev_alloc(&b->d_ctrl, mt))) return rc;
  if ((rc = dev_alloc(&b->d_tstart, mt + 1))) return rc;
  if ((rc = dev_alloc(&b->d_tlist, (size_t)n_graphs))) return rc;
  if ((rc = dev_alloc(&b->d_toff, mt))) return rc;
  if ((rc = dev_alloc(&b->d_tcells, mt))) return rc;
  if ((rc = dev_alloc(&b->d_tsoff, mt))) return rc;
  if ((rc = dev_alloc(&b->d_records, (size_t)n_graphs)) || (rc = dev_alloc(&b->d_lctrl, 2 * mt))) return rc;
  // set_plan below waits for b->stream, so these come before any launch and upload
  BCUDA(cudaMemsetAsync(b->d_records, 0, (size_t)n_graphs * sizeof(ggb::ApspCtrl), b->stream));
  BCUDA(cudaMemsetAsync(b->d_adj, 0, std::max<size_t>((size_t)b->adj_ints, 1) * sizeof(int), b->stream));
  BCUDA(cudaHostAlloc(&b->h_lctrl, 2 * mt * sizeof(ggb::ApspCtrl), cudaHostAllocDefault));
  BCUDA(cudaHostAlloc(&b->h_out, (size_t)n_graphs * sizeof(ggb::BatchOut), cudaHostAllocDefault));
  BCUDA(cudaHostAlloc(&b->h_ctrl, mt * sizeof(ggb::ApspCtrl), cudaHostAllocDefault));
  std::vector<ggb::BatchGraph> gs(n_graphs);
  for (int i = 0; i < n_graphs; ++i) {
    gs[i].adj = b->d_adj + b->off[i];
    gs[i].N = b->N[i];
    gs[i].d = b->d[i];
    gs[i].n_src = b->bn[i];
    gs[i].groups = b->grp[i];
    gs[i].vec4 = (b->d[i] % 4 == 0) ? 1 : 0;   // every graph starts on a 16-byte boundary
    gs[i].win_first = 0;
    gs[i].win_stride = 1;
    gs[i].win_bits = 0;
  }
  BCUDA(cudaMemcpy(b->d_graphs, gs.data(), gs.size() * sizeof(ggb::BatchGraph), cudaMemcpyHostToDevice));
  return ggb_batch_set_plan(b, 0, 0);
}

// The plan the model prefers: the (R, T) pair with the least modelled makespan.
void model_choice(ggb_batch* b, const std::vector<int>& ids, int* R, int* T) {
  double best = 1e300;
  int nsrc_max = 0;
  for (int i : ids) nsrc_max = std::max(nsrc_max, b->bn[i]);
  for (int r = 1; r <= kMaxR; r *= 2) {
    for (int t = 1; t <= b->occ[log2i(r)] * b->sms; t *= 2) {
      const double m = make_plan(b, ids, r, t, false);
      if (m < best * 0.999) { best = m; *R = r; *T = t; }
    }
    if (128 * r >= nsrc_max) break;
  }
}

}  // namespace

extern "C" {

int ggb_batch_create(int n_graphs, const int* nodes, const int* based_nodes, const int* groups, const int* degree,
                     ggb_batch** out) {
  if (!out || !nodes || !based_nodes || !groups || !degree || n_graphs <= 0)
    return core_fail(GGB_EINVAL, "ggb_batch_create: null pointer or n_graphs <= 0");
  *out = nullptr;
  ggb_batch* b = new ggb_batch();
  int rc = create(n_graphs, nodes, based_nodes, groups, degree, b);
  if (rc) {
    destroy(b);
    return rc;
  }
  *out = b;
  return GGB_OK;
}

void ggb_batch_destroy(ggb_batch* b) { destroy(b); }

int ggb_batch_set_plan(ggb_batch* b, int window_bits, int team_ctas) {
  if (!b) return core_fail(GGB_EINVAL, "null batch");
  if (window_bits < 0 || team_ctas < 0) return core_fail(GGB_EINVAL, "negative plan value");
  int R = window_bits / 128, T = team_ctas;
  if (window_bits && (window_bits % 128 || (R & (R - 1)) || R > kMaxR))
    return core_fail(GGB_EINVAL, "window_bits must be 128 * 2^k, at most %d", 128 * kMaxR);
  BCUDA(cudaSetDevice(b->device));
  if (!R && !T) return plan_split(b);
  if (!R || !T) {
    int mr = 1, mt = 1;
    model_choice(b, all_graphs(b), &mr, &mt);
    if (!R) R = mr;
    if (!T) T = mt;
  }
  return plan_fixed(b, R, T);
}

int ggb_batch_get_plan(const ggb_batch* b, int* window_bits, int* team_ctas, int* teams) {
  if (!b) return core_fail(GGB_EINVAL, "null batch");
  int R = b->R, T = b->T, n = b->n_teams;
  if (b->split) {
    // a fixed plan that serves all graphs, for callers that keep a plan and set it
    // again: with the window teams of the automatic plan alone the mixed workload
    // took 7.9 ms, 5.8 with the best fixed plan (automatic 4.7)
    R = b->best_fixed_R;
    T = b->best_fixed_T;
    if (!R) model_choice(const_cast<ggb_batch*>(b), all_graphs(b), &R, &T);   // (keeps nothing)
    n = team_count(b, b->n, R, &T);
  }
  if (window_bits) *window_bits = 128 * R;
  if (team_ctas) *team_ctas = T;
  if (teams) *teams = n;
  return GGB_OK;
}

int ggb_batch_adj_device(ggb_batch* b, int graph, int** adj_dev) {
  if (!b || !adj_dev || graph < 0 || graph >= b->n) return core_fail(GGB_EINVAL, "bad batch graph index");
  *adj_dev = b->d_adj + b->off[graph];
  return GGB_OK;
}

int ggb_batch_upload(ggb_batch* b, const int* const* adj, void* stream) {
  if (!b || !adj) return core_fail(GGB_EINVAL, "null pointer");
  int rc = check_upload(b, adj, stream ? (cudaStream_t)stream : b->stream);
  if (rc) return rc;
  return upload_range(b, adj, 0, b->n, stream ? (cudaStream_t)stream : b->stream);
}

int ggb_batch_launch(ggb_batch* b, void* stream) {
  if (!b) return core_fail(GGB_EINVAL, "null batch");
  return launch(b, stream ? (cudaStream_t)stream : b->stream, true);
}

int ggb_batch_collect(ggb_batch* b, void* stream, ggb_result* results) {
  if (!b) return core_fail(GGB_EINVAL, "null batch");
  BCUDA(cudaSetDevice(b->device));
  return collect(b, stream ? (cudaStream_t)stream : b->stream, results);
}

int ggb_batch_eval(ggb_batch* b, const int* const* adj, ggb_result* results) {
  if (!b || !adj) return core_fail(GGB_EINVAL, "null pointer");
  const int kernels = (b->n_teams > 0) + (b->l_teams > 0) + !b->slices.empty();
  int rc = check_upload(b, adj, b->stream);
  if (rc) return rc;
  if (b->split && kernels > 1) {
    rc = eval_parts(b, adj);
    if (rc) {   // nothing of this call stays in flight
      cudaStreamSynchronize(b->copies);
      cudaStreamSynchronize(b->stream);
    }
  } else {
    rc = upload_range(b, adj, 0, b->n, b->stream);
    if (!rc) rc = launch(b, b->stream, true);
  }
  if (rc) return rc;
  return collect(b, b->stream, results);
}

int ggb_batch_kernel_ms(const ggb_batch* b, double* ms) {
  if (!b || !ms) return core_fail(GGB_EINVAL, "null pointer");
  if (b->pending) return core_fail(GGB_EPERM, "the last launch has not been collected");
  double sum = 0.0;
  for (int i = 0; i < std::max(1, b->timed); ++i) {
    float f = 0.f;
    BCUDA(cudaEventElapsedTime(&f, b->ev[2 * i], b->ev[2 * i + 1]));
    sum += f;
  }
  *ms = sum;
  return GGB_OK;
}

int ggb_batch_autotune(ggb_batch* b, int iters, int* window_bits, int* team_ctas, double* best_ms) {
  if (!b) return core_fail(GGB_EINVAL, "null batch");
  if (iters <= 0) iters = 2;
  BCUDA(cudaSetDevice(b->device));
  const int nsrc_max = *std::max_element(b->bn.begin(), b->bn.end());
  double best = 1e300;
  int bR = 0, bT = 0, rc;
  // the least time of `iters` launches of the current plan, after one that warms up
  auto time_plan = [&](double* ms_min) -> int {
    *ms_min = 1e300;
    for (int it = 0; it <= iters; ++it) {
      int rc = launch(b, b->stream, false);
      if (rc) return rc;
      if ((rc = collect(b, b->stream, nullptr))) return rc;
      float f = 0.f;
      BCUDA(cudaEventElapsedTime(&f, b->ev[0], b->ev[1]));
      if (it > 0) *ms_min = std::min(*ms_min, (double)f);
    }
    return GGB_OK;
  };
  if ((rc = plan_split(b)) || (rc = time_plan(&best))) return rc;   // bR == 0: the automatic plan
  double best_fixed = 1e300;
  int fR = 0, fT = 0;
  for (int r = 1; r <= kMaxR; r *= 2) {
    const int ctas_max = b->occ[log2i(r)] * b->sms;
    std::vector<int> ts;
    for (int t = 1; t <= ctas_max; t *= 2) ts.push_back(t);
    for (int t : {b->sms / 4, b->sms / 2, b->sms})
      if (t >= 1 && t <= ctas_max && std::find(ts.begin(), ts.end(), t) == ts.end()) ts.push_back(t);
    for (int t : ts) {
      double ms = 0.0;
      if ((rc = plan_fixed(b, r, t)) || (rc = time_plan(&ms))) return rc;
      if (ms < best) { best = ms; bR = r; bT = t; }
      if (ms < best_fixed) { best_fixed = ms; fR = r; fT = t; }
    }
    if (128 * r >= nsrc_max) break;   // wider windows only add zero bits
  }
  rc = bR ? plan_fixed(b, bR, bT) : plan_split(b);
  if (rc) return rc;
  b->best_fixed_R = fR;
  b->best_fixed_T = fT;
  if ((rc = ggb_batch_get_plan(b, window_bits, team_ctas, nullptr))) return rc;
  if (best_ms) *best_ms = best;
  return GGB_OK;
}

}  // extern "C"
