// apsp_levels.cuh -- mid-size graphs with a symmetric adjacency, level by
// level over all sources at once (sm_100a).
//
// From a few thousand to about twenty thousand vertices the whole N x N bit
// matrix of a level fits in L2, so no windows are needed: a team of CTAs keeps
// S_k and S_{k+1} as two matrices of N rows.  Bit s of S_k[v] is bit v of
// S_k[s] (apsp_sym.cuh), so a level sweeps only the lower triangle, in parts of
// 256 bits -- part p of row v for p <= v / 256 -- and fills the upper one with
// 256 x 256-bit transposes: half of the gathers at the price of one more
// barrier, where windows of 4096 sources would save 25 to 37 % of them.
//
//   seed        S_2 of every row in shared memory (one warp per vertex, two-hop
//               ids), the counts of S_1 and S_2, and the symmetry check;
//   level       sweep, barrier, decision (level_decision), transposes, barrier;
//   last        once the next level is expected to leave few pairs unreached
//               (q -> q^(d-1) for a share q of unreached pairs), its sweep
//               writes nothing and lists them; they are resolved through a hash
//               table as in apsp_sym.cuh.  A list that overflows has the level
//               swept again in full.
//
// An asymmetric adjacency, or pairs still unresolved after kSymPasses levels,
// is left to eval_windows (kLevelsNotServed).
//
// Bound: the latency of a task's chain (ids, then two groups of eight gathers)
// and two barriers a level: 906 MB through L2 at 6.5 TB/s for N = 16384, d = 12 on
// the whole GPU, issue slots 31 % busy.
// Measured, kernel us: N = 16384, d = 12 144 on 148 CTAs (the persistent kernel
// with its ball 182), 218 on 74, 370 on 37 (467 there), 745 on 16 (948).
//
// Graphs that it does not suit, whole call, us, against the persistent kernel:
// one asymmetric row, d = 8, which costs the seeding, 187 / 169 at N = 12000, 271 / 185
// at 16000; a random core whose vertices carry a leaf each, rows of 7, where the
// list overflows and a level is swept twice, 182 / 159 at 8600, 355 / 228 at 12000,
// 394 / 234 at 16000; two components, d = 8, 136 / 100 at 12000, 171 / 121 at 16000;
// circulants of 20 to 4000 levels between 15 % faster and 20 % slower.
#pragma once
#include "apsp_sym.cuh"

namespace ggb {

constexpr unsigned kLevelsList = 1u << 18;     // listed pairs per team
constexpr unsigned kLevelsTarget = 1u << 14;   // pairs expected when the last sweep is chosen
constexpr int kLevelsSet = 2 + kSymPasses;       // counters of a graph: list_n, pairs left after each pass, flags
constexpr int kLevelsFlags = 1 + kSymPasses;     // of them the flags: 1 asymmetric, 2 an id out of range
constexpr int kLevelsCounters = 3 * kLevelsSet;  // per team: three sets in rotation

enum : int { kLevelsFailed = 0, kLevelsDone = 1, kLevelsNotServed = 2 };

// Per-team workspace of the list.
struct LevelsList {
  unsigned* counters;           // [3][kLevelsSet], zeroed before the launch
  unsigned long long* list;     // [kLevelsList]
  unsigned long long* hash;     // [2 * kLevelsList]
  unsigned char* hlev;          // [2 * kLevelsList]
};
// Its size in 8-byte words.
constexpr size_t kLevelsListWords = 3 * (size_t)kLevelsList + kLevelsList / 4;

// The workspace in one allocation: list, keys, levels, counters.
inline LevelsList levels_list(unsigned long long* p) {
  LevelsList l;
  l.list = p;
  l.hash = p + kLevelsList;
  l.hlev = reinterpret_cast<unsigned char*>(l.hash + 2 * (size_t)kLevelsList);
  l.counters = reinterpret_cast<unsigned*>(p + kLevelsListWords);
  return l;
}

// uint4 of a matrix row: parts of 256 bits.
__host__ __device__ __forceinline__ int levels_pitch(int N) { return (N + 255) / 256 * 2; }

// Shared memory of the seeding rows: the row and the neighbour ids per warp.
__host__ __device__ __forceinline__ size_t levels_smem_bytes(int N, int d) {
  return (size_t)kWarps * (levels_pitch(N) + (d + 3) / 4) * sizeof(uint4);
}

// S_2 of the rows warp_id, warp_id + n_warps, ... into rows; c[0] and c[2]
// receive the counts of S_1 and S_2.
template <int VEC>
__device__ __forceinline__ void levels_seed(const int* __restrict__ adj, int N, int d, uint4* __restrict__ rows, int C,
                                            uint4* s_row, long long warp_id, long long n_warps, unsigned (&c)[4],
                                            bool& bad, bool& asym) {
  const int lane = threadIdx.x & 31;
  unsigned* const row = reinterpret_cast<unsigned*>(s_row);
  int* const nb1 = reinterpret_cast<int*>(s_row + C);
  const unsigned all = d >= 32 ? 0xffffffffu : (1u << d) - 1u;
  const int per = d / VEC, rpi = 32 / per;
  const int roff = lane / per, part = lane - roff * per;
  const bool active = roff < rpi;
  for (long long v = warp_id; v < N; v += n_warps) {
    for (int i = lane; i < C; i += 32) s_row[i] = make_uint4(0u, 0u, 0u, 0u);
    int x1 = -1;
    if (lane < d) {
      x1 = __ldg(adj + v * d + lane);
      if ((unsigned)x1 >= (unsigned)N) { bad = true; x1 = -1; }
      nb1[lane] = x1;
    }
    __syncwarp();
    unsigned n1 = 0, n2 = 0;
    if (lane == 0) { row[v >> 5] = 1u << (v & 31); n1 = 1; }
    __syncwarp();
    if (x1 >= 0) {
      const unsigned m = 1u << (x1 & 31);
      n1 += !(smem_or_old(row + (x1 >> 5), m) & m);
    }
    __syncwarp();
    unsigned back = 0u;
    for (int r0 = 0; r0 < d; r0 += 4 * rpi) {
      AdjVec<VEC> val[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int j = r0 + t * rpi + roff;
        const int u = (active && j < d) ? nb1[j] : -1;
        val[t].fill(-1);
        if (u >= 0) val[t].load(adj + (long long)u * d + part * VEC);
      }
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int j = r0 + t * rpi + roff;
        if (!active || j >= d) continue;
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          const int x = val[t].at(e);
          if (x == (int)v) back |= 1u << j;
          if ((unsigned)x < (unsigned)N) {
            const unsigned m = 1u << (x & 31);
            n2 += !(smem_or_old(row + (x >> 5), m) & m);
          }
        }
      }
    }
    if (__reduce_or_sync(0xffffffffu, back) != all) asym = true;
    c[0] += n1;
    c[2] += n1 + n2;
    __syncwarp();
    for (int i = lane; i < C; i += 32) st_cg(rows + (size_t)v * C + i, s_row[i]);
    __syncwarp();
  }
}

// Lower triangle of one level from src into dst; LAST as in sym_sweep.
// c_diag counts the diagonal parts, c_off the parts below them.
template <bool LAST>
__device__ __forceinline__ void levels_sweep(const SymArgs& s, const uint4* __restrict__ src, uint4* __restrict__ dst,
                                             const int* __restrict__ adj, int N, int d, int vec4, int C, bool early,
                                             long long warp_id, long long n_warps, unsigned& c_diag, unsigned& c_off) {
  constexpr int U = 8;
  bool full = false;
  const int lane = threadIdx.x & 31, h = lane >> 4, hl = lane & 15;
  // half-warp tasks: row v of the column group i (16 parts, 4096 bits), v >= 4096 i
  const int groups = (C / 2 + 15) / 16;
  long long tasks = 0;
  for (int i = 0; i < groups; ++i) tasks += N - 4096 * i;
  for (long long tb = warp_id * 2; tb < tasks; tb += n_warps * 2) {
    long long t = tb + h;
    const bool task = t < tasks;
    if (!task) t = tb;
    int i = 0;
    while (t >= N - 4096 * i) { t -= N - 4096 * i; ++i; }
    const int v = 4096 * i + (int)t;
    const int p = 16 * i + hl, dp = v >> 8;      // this lane's part, the diagonal's
    const bool live = task && p <= dp;
    const size_t col = 2 * (size_t)p;
    const int* arow = adj + (long long)v * d;
    const int nv = min(256, N - 256 * p);        // valid bits of the part
    uint4 acc[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
    if (live) ld_cg2(src + (size_t)v * C + col, acc);
    bool need = live;
    for (int j = 0; j < d; j += U) {
      int u[U];
      if (vec4 && j + U <= d) {
#pragma unroll
        for (int q = 0; q < U; q += 4) {
          const int4 x = __ldg(reinterpret_cast<const int4*>(arow + j + q));
          u[q] = x.x; u[q + 1] = x.y; u[q + 2] = x.z; u[q + 3] = x.w;
        }
      } else {
#pragma unroll
        for (int q = 0; q < U; ++q) u[q] = j + q < d ? __ldg(arow + j + q) : v;
      }
      if (j > 0 || early) {
        need = live && (nv < 256 || (acc[0].x & acc[0].y & acc[0].z & acc[0].w & acc[1].x & acc[1].y & acc[1].z &
                                     acc[1].w) != 0xffffffffu);
        if (!__any_sync(0xffffffffu, need)) break;
      }
      uint4 x[U][2];
#pragma unroll
      for (int q = 0; q < U; ++q) {
        if (need && j + q < d) {
          ld_cg2(src + (size_t)u[q] * C + col, x[q]);
        } else {
          x[q][0] = make_uint4(0u, 0u, 0u, 0u);
          x[q][1] = make_uint4(0u, 0u, 0u, 0u);
        }
      }
#pragma unroll
      for (int q = 0; q < U; ++q) {
        or_into(acc[0], x[q][0]);
        or_into(acc[1], x[q][1]);
      }
    }
    if (!live) continue;
    const unsigned cc = popc4(acc[0]) + popc4(acc[1]);
    if (p == dp) c_diag += cc; else c_off += cc;
    if constexpr (LAST) {
      if (cc != (unsigned)nv)
        for (int k = 0; k < 8; ++k) list_missing(s, word_of(acc, k), nv - 32 * k, v, 256 * p + 32 * k, p == dp, full, kLevelsList);
    } else {
      st_cg2(dst + (size_t)v * C + col, acc);
    }
  }
}

// The upper triangle of m from its lower one.
__device__ __forceinline__ void levels_transposes(uint4* m, int N, int C, long long warp_id, long long n_warps) {
  const int lane = threadIdx.x & 31;
  const Transpose32 tr(lane);
  const int nt = C / 2;
  const int tiles = nt * (nt - 1) / 2;
  for (long long t = warp_id; t < tiles; t += n_warps) {
    int tv = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)t)) * 0.5f);
    while (tv * (tv - 1) / 2 > (int)t) --tv;
    while ((tv + 1) * tv / 2 <= (int)t) ++tv;
    const int tp = (int)t - tv * (tv - 1) / 2;   // tp < tv
    transpose_tile(m + (size_t)256 * tv * C + 2 * tp, C, N - 256 * tv, m + (size_t)256 * tp * C + 2 * tv, C, lane, tr);
  }
}

// One graph on the `ncta` CTAs of a team (this one is number `cta`), as
// eval_windows: m0 and m1 are its two matrices of N rows of levels_pitch(N)
// uint4; `turn` counts the team's graphs, `name` stands for this one in an
// error.  kLevelsFailed: a wait ran out or an error was reported, the caller
// leaves the kernel.
//
// A CTA that is done with a graph goes on to the team's next one without a
// barrier, so nothing the next graph's seeding writes may be read late for this
// one: what a graph's CTAs tell one another lies in its own set of counters.  A
// set is cleared in the graph before its use, two after its last readers, whose
// CTAs have all arrived at a barrier since.
__device__ __forceinline__ int eval_levels(const ApspArgs& a, const LevelsList& ws, unsigned turn, int name, uint4* m0, uint4* m1,
                                           int cta, int ncta, ApspSmem& sm, unsigned* s_dyn,
                                           unsigned long long& bar_target, unsigned& gl, EvalOut& out) {
  const int N = a.N, d = a.d, C = levels_pitch(N);
  const int warp = threadIdx.x >> 5;
  const long long warp_id = (long long)cta * kWarps + warp, n_warps = (long long)ncta * kWarps;
  ApspCtrl* const ctrl = a.ctrl;
  unsigned* const set = ws.counters + (turn % 3) * kLevelsSet;
  SymArgs s;
  s.list_n = set;
  s.list = ws.list;
  s.hash = ws.hash;
  s.hlev = ws.hlev;
  auto barrier = [&]() -> bool {
    bar_target += (unsigned)ncta;
    return grid_barrier(ctrl, bar_target, a.timeout_ns, &sm.flag);
  };
  if (cta == 0)
    for (int i = threadIdx.x; i < kLevelsSet; i += blockDim.x) ws.counters[((turn + 1) % 3) * kLevelsSet + i] = 0u;
  long long sum = 0, prev_total = N, dense = 0;
  int kk = 0, act = 0;
  // ---- S_1 and S_2 -----------------------------------------------------------------
  {
    unsigned c[4] = {0u, 0u, 0u, 0u};
    bool bad = false, asym = false;
    uint4* const s_row = reinterpret_cast<uint4*>(s_dyn) + (size_t)warp * (C + (d + 3) / 4);
    if (a.vec4)
      levels_seed<4>(a.adj, N, d, m0, C, s_row, warp_id, n_warps, c, bad, asym);
    else
      levels_seed<1>(a.adj, N, d, m0, C, s_row, warp_id, n_warps, c, bad, asym);
    if (bad) set_error(ctrl, kErrAdj, name);
    const unsigned flags = __reduce_or_sync(0xffffffffu, (bad ? 2u : 0u) | (asym ? 1u : 0u));
    if ((threadIdx.x & 31) == 0 && flags) atomicOr(set + kLevelsFlags, flags);
    cta_add_counts<4>(c, ctrl, gl, sm.red);
  }
  if (!barrier()) return kLevelsFailed;
  read_level_counts(ctrl, gl, 2, sm.seen, sm.lvl);
  const long long c1 = sm.lvl[0], c2 = sm.lvl[2];
  __syncthreads();
  gl += 2;
  const unsigned flags = __ldcg(set + kLevelsFlags);
  if (flags & 2u) return kLevelsFailed;
  if (flags & 1u) return kLevelsNotServed;
  act = level_decision(1, c1, 0, N, N, N, 0, 1, prev_total, sum);
  if (!act) {
    kk = 1;
    act = level_decision(1, c2, 0, N, N, N, 0, 1, prev_total, sum);
    if (!act) kk = 2;
  }
  // ---- levels ----------------------------------------------------------------------
  uint4* cur = m0;
  uint4* nxt = m1;
  bool may_list = true, listed = false;
  const double pairs = (double)N * N;
  while (!act && kk < N) {
    const double q = 1.0 - (double)prev_total / pairs;
    // expected share of unreached pairs after this level: q^(d-1), in logs
    const bool last = may_list && 0.5 * pairs * exp((d - 1) * log(q)) <= (double)kLevelsTarget;
    const bool early = q * 200.0 <= 1.0;
    unsigned c[2] = {0u, 0u};
    if (last)
      levels_sweep<true>(s, cur, nullptr, a.adj, N, d, a.vec4, C, early, warp_id, n_warps, c[0], c[1]);
    else
      levels_sweep<false>(s, cur, nxt, a.adj, N, d, a.vec4, C, early, warp_id, n_warps, c[0], c[1]);
    cta_add_counts<2>(c, ctrl, gl, sm.red);
    if (!barrier()) return kLevelsFailed;
    read_level_counts(ctrl, gl, 1, sm.seen, sm.lvl);
    const long long total = sm.lvl[0] + 2 * sm.lvl[1];
    __syncthreads();
    ++gl;
    ++dense;
    if (last) {
      if (__ldcg(set) > kLevelsList) {           // swept again in full
        may_list = false;
        continue;
      }
      listed = true;
    }
    act = level_decision(1, total, 0, N, N, N, 0, 1, prev_total, sum);
    if (act || listed) break;
    levels_transposes(nxt, N, C, warp_id, n_warps);
    if (!barrier()) return kLevelsFailed;
    uint4* const x = cur;
    cur = nxt;
    nxt = x;
    ++kk;
  }
  // ---- the listed pairs --------------------------------------------------------------
  if (listed && !act) {
    const unsigned n = __ldcg(set);
    unsigned long long late = 0;
    int passes = 0;
    const int r = sym_resolve(s, set + 1, a.adj, d, n, kSymPasses, (unsigned)cta * kThreads + threadIdx.x,
                              (unsigned)ncta * kThreads, barrier, late, passes);
    if (r == kSymFailed) return kLevelsFailed;
    if (r == kSymTooLong) return kLevelsNotServed;
    // level kk's unreached pairs are in `sum` already
    sum += (long long)late - 2LL * n;
    kk += passes;
    act = r == kSymStalled ? 2 : 1;
  }
  out.sum = sum;
  out.levels = kk + 1;
  out.dense_levels = dense;
  out.diam = act == 1 ? kk + 1 : N + 1;
  out.disconnected = act == 1 ? 0 : 1;
  out.windows = 1;
  return kLevelsDone;
}

// ---- one graph, one team ---------------------------------------------------------
static __global__ void __launch_bounds__(kThreads, 1) apsp_levels_kernel(const ApspArgs a, const LevelsList ws) {
  __shared__ ApspSmem sm;
  extern __shared__ __align__(16) unsigned s_dyn[];
  if (threadIdx.x < 8) sm.seen[threadIdx.x >> 1][threadIdx.x & 1] = 0ULL;
  __syncthreads();
  unsigned long long bar_target = 0;
  unsigned gl = 0;
  EvalOut o;
  const int r = eval_levels(a, ws, 0u, (int)blockIdx.x, a.buf0, a.buf1, (int)blockIdx.x, (int)gridDim.x, sm, s_dyn, bar_target, gl, o);
  if (r == kLevelsFailed || blockIdx.x != 0 || threadIdx.x != 0) return;
  ApspCtrl* c = a.ctrl;
  if (r == kLevelsNotServed) {
    c->fallback = 1;
    return;
  }
  c->diam = o.diam;
  c->disconnected = o.disconnected;
  c->sum = o.sum;
  c->levels = o.levels;
  c->dense_levels = o.dense_levels;
  c->windows = o.windows;
  __threadfence();
  c->done = 1;
}

// ---- many graphs on teams, as apsp_batch_kernel --------------------------------------
// b.scratch + b.team_off[t] holds team t's two matrices (b.team_cells[t] apart),
// lists + t * list_words its list.  A graph that is not served keeps done = 0
// for the window launch behind this one.
static __global__ void __launch_bounds__(kThreads, 1) apsp_batch_levels_kernel(const BatchArgs b, unsigned long long* lists,
                                                                        size_t list_words) {
  __shared__ ApspSmem sm;
  extern __shared__ __align__(16) unsigned s_dyn[];
  const int team = (int)blockIdx.x / b.team_ctas, cta = (int)blockIdx.x % b.team_ctas;
  if (team >= b.n_teams) return;
  if (b.stop && ld_volatile_i32(b.stop) != 0) return;   // written before the launch: the same in every CTA
  if (threadIdx.x < 8) sm.seen[threadIdx.x >> 1][threadIdx.x & 1] = 0ULL;
  __syncthreads();
  unsigned long long* const words = lists + (size_t)team * list_words;
  LevelsList ws;
  ws.list = words;
  ws.hash = words + kLevelsList;
  ws.hlev = reinterpret_cast<unsigned char*>(words + 3 * (size_t)kLevelsList);
  ws.counters = reinterpret_cast<unsigned*>(words + kLevelsListWords);
  ApspArgs a;
  a.adj2 = nullptr;
  a.ctrl = b.team_ctrl + team;
  a.timeout_ns = b.timeout_ns;
  uint4* const m0 = b.scratch + b.team_off[team];
  uint4* const m1 = m0 + b.team_cells[team];
  unsigned long long bar_target = 0;
  unsigned gl = 0;
  const int k0 = b.team_start[team], k1 = b.team_start[team + 1];
  for (int k = k0; k < k1; ++k) {
    const int gi = b.team_list[k];
    const BatchGraph gr = b.graphs[gi];
    a.adj = gr.adj;
    a.N = gr.N;
    a.d = gr.d;
    a.vec4 = gr.vec4;
    EvalOut o;
    const int r = eval_levels(a, ws, (unsigned)(k - k0), gi, m0, m1, cta, b.team_ctas, sm, s_dyn, bar_target, gl, o);
    if (r == kLevelsFailed) {
      if (b.sticky && threadIdx.x == 0) atomicCAS(b.sticky, 0, max(1, ld_volatile_i32(&a.ctrl->error)));
      return;
    }
    if (r == kLevelsDone && cta == 0 && threadIdx.x == 0) {
      BatchOut* w = b.out + gi;
      w->sum = o.sum;
      w->levels = o.levels;
      w->dense_levels = o.dense_levels;
      w->diam = o.diam;
      w->disconnected = o.disconnected;
      w->windows = o.windows;
      w->error = 0;
      w->done = 1;
    }
  }
}

}  // namespace ggb
