// apsp_slice.cuh -- one source window per CTA, its bitset rows in shared
// memory (sm_100a).
//
// The persistent kernel (apsp_kernel.cuh) spreads every window over all SMs
// and pays a grid barrier per level; on graphs of a few thousand vertices and
// on graphs of large diameter those barriers are the evaluation.  The sources
// are independent, so here each CTA takes windows of at most 32 or 64 sources,
// keeps both bitset matrices of a window (N rows of 4 or 8 bytes) in its own
// shared memory, and exchanges no word with another CTA until its sums are
// done.  Same recurrence, same counts and same decisions per window as
// eval_windows (level_decision), so the integers are the same.
//
// slice_kernel takes every vertex at every level (small graphs);
// slice_push_kernel visits only the ring of vertices that receive new bits
// (lattice graphs, whose levels are many and thin).
#pragma once
#include "apsp_kernel.cuh"

namespace ggb {

constexpr int kSliceMaxN = 32768;    // ids travel as 16 bits

struct SliceArgs {
  const int* adj;            // [N][d] ids, or null when adj16 is given
  const uint16_t* adj16;     // [N][d] 16-bit ids
  const int* deg;            // entries of row v that count, in [0, d] (null: all)
  const Swap* patch;         // the graph is adj with this swap applied when it is valid (null: adj itself)
  ApspCtrl* ctrl;            // all zero between launches (the last CTA clears it)
  ApspCtrl* out;             // the result record (pinned host memory), written by the last CTA
  int N, d, pairs, np;       // np = N rounded up to 32
  int n_src1, split, ac, groups;
  int width;                 // sources per window, at most 32 * WORDS
  int nw1, nw2;              // windows of phase 1 and of the added centres
  // slice_push_kernel only: adj16 rows padded to dp ids (a multiple of 4), and
  // the lattice's height (device)
  int dp;
  const int* height;
};

template <int WORDS> struct SliceRow;
template <> struct SliceRow<1> {
  using T = unsigned;
  static __device__ __forceinline__ T bit(unsigned b) { return b < 32u ? 1u << b : 0u; }
  static __device__ __forceinline__ T full(int l) { return l >= 32 ? 0xffffffffu : (1u << l) - 1u; }
  static __device__ __forceinline__ unsigned popc(T x) { return __popc(x); }
};
template <> struct SliceRow<2> {
  using T = unsigned long long;
  static __device__ __forceinline__ T bit(unsigned b) { return b < 64u ? 1ull << b : 0ull; }
  static __device__ __forceinline__ T full(int l) { return l >= 64 ? ~0ull : (1ull << l) - 1ull; }
  static __device__ __forceinline__ unsigned popc(T x) { return __popcll(x); }
};

// Entries 2p and 2p + 1 of row v, of which the first dv count, as one word; a
// slot past them holds v itself, which the recurrence ignores.  An entry
// outside [0, N) is reported and replaced by v.
template <typename ID>
__device__ __forceinline__ unsigned pack_pair(const ID* __restrict__ row, int p, int dv, int v, int N, bool& bad) {
  unsigned a = 2 * p < dv ? (unsigned)__ldg(row + 2 * p) : (unsigned)v;
  unsigned b = 2 * p + 1 < dv ? (unsigned)__ldg(row + 2 * p + 1) : (unsigned)v;
  if (a >= (unsigned)N) { bad = true; a = (unsigned)v; }
  if (b >= (unsigned)N) { bad = true; b = (unsigned)v; }
  return a | (b << 16);
}

// Per-window counters of the two kernels: unreached pairs of the lo and hi
// rows.  All threads keep the same values.
struct SliceCount {
  unsigned lo, hi;               // unreached (vertex, source) pairs
  unsigned long long s_lo, s_hi; // their sums over the levels
  // The level's new bits; returns 1: complete, 2: nothing added (level_decision)
  __device__ __forceinline__ int level(int phase, unsigned n_lo, unsigned n_hi) {
    lo -= n_lo;
    hi -= n_hi;
    if ((phase == 1 ? lo | hi : hi) == 0u) return 1;
    if ((n_lo | n_hi) == 0u) return 2;
    s_lo += lo;
    s_hi += hi;
    return 0;
  }
};

// One CTA's windows added to the launch's record; the last CTA writes the
// record out and clears it for the next launch.
struct SliceTotals {
  unsigned long long s1_lo = 0, s1_hi = 0, s2 = 0;   // phase 1 lo / hi rows, phase 2
  int levels = 0, diam = 1, disconnected = 0, windows = 0;
};

// Adds a CTA's totals to the record; the last of n_ctas hands the whole to
// write(sum, levels, windows, diam, disconnected, error, info) and clears it.
template <typename Write>
__device__ __forceinline__ void slice_finish(ApspCtrl* c, int groups, unsigned n_ctas, const SliceTotals& r,
                                             Write write) {
  if (threadIdx.x != 0) return;
  const unsigned long long sum = r.s1_lo * (unsigned)groups + r.s1_hi * 2u * (unsigned)groups + r.s2;
  atomicAdd(reinterpret_cast<unsigned long long*>(&c->sum), sum);
  atomicAdd(reinterpret_cast<unsigned long long*>(&c->levels), (unsigned long long)r.levels);
  atomicMax(&c->diam, r.diam);
  if (r.disconnected) atomicOr(&c->disconnected, 1);
  atomicAdd(&c->windows, r.windows);
  __threadfence();
  if (atomicAdd(&c->bar, 1ULL) != (unsigned long long)n_ctas - 1) return;
  __threadfence();
  const int err = __ldcg(&c->error), info = __ldcg(&c->error_info), dm = __ldcg(&c->diam);
  const int dc = __ldcg(&c->disconnected), nw = __ldcg(&c->windows);
  const long long sm = __ldcg(&c->sum), lv = __ldcg(&c->levels);
  write(sm, lv, nw, dm, dc, err, info);
  c->error = 0;
  c->error_info = 0;
  c->diam = 0;
  c->disconnected = 0;
  c->sum = 0;
  c->levels = 0;
  c->windows = 0;
  c->asym = 0;
  c->cnt[0][0] = 0ULL;
  c->bar = 0ULL;
}

// The record of a single evaluation, in pinned host memory.
__device__ __forceinline__ void slice_finish(const SliceArgs& a, const SliceTotals& r) {
  slice_finish(a.ctrl, a.groups, gridDim.x, r, [&](long long sum, long long levels, int windows, int diam,
                                                   int disconnected, int error, int info) {
    ApspCtrl* o = a.out;
    o->error = error;
    o->error_info = info;
    o->diam = diam;
    o->disconnected = disconnected;
    o->sum = sum;
    o->levels = levels;
    o->dense_levels = levels - windows;
    o->windows = windows;
    o->trace_len = 0;
    o->done = 1;
  });
}

// ---- small graphs: every vertex at every level ----------------------------------
// The adjacency is staged in shared memory as 16-bit ids in pairs, transposed:
// word [p][v] holds entries 2p and 2p + 1 of row v, so that a warp's 32
// vertices read 128 contiguous bytes.  Level 1 needs no gather (a bit of S_1[v]
// is an id that lies in the window), and a thread's gathers stop once its row
// is full.
//
// Bound: at N = 256 the launch, the staging and the record's way out (11 us;
// the persistent kernel took 37); from N = 1024 on issue slots (56 to 65 % busy
// on the SMs with a window) and the shared-memory wavefronts of the random row
// reads: over all shared loads 2.2 a load with four-byte rows and 3.3 to 3.5 with
// eight-byte ones, the load/store data pipe 48 % busy at N = 4700, d = 6 and 67 % at
// N = 9000, d = 3 (N = 1024, d = 8: 15 us, was 27; N = 4700, d = 6: 39 us, was 48;
// N = 9000, d = 3: 90 us, was 228).
//
// Shared memory: two row buffers and the adjacency.
inline size_t slice_smem_bytes(int np, int words, int pairs) { return (size_t)np * (words * 8 + pairs * 4); }

// Windows t0, t0 + step, ... below t1 of one graph on this CTA.
template <int WORDS>
__device__ __forceinline__ SliceTotals slice_windows(const SliceArgs& a, int t0, int t1, int step) {
  using Row = SliceRow<WORDS>;
  using T = typename Row::T;
  extern __shared__ __align__(16) unsigned char s_raw[];
  __shared__ unsigned s_cnt[3][2];     // new bits of a level, lo and hi rows, in rotation
  const int N = a.N, np = a.np, pairs = a.pairs;
  const int tid = threadIdx.x, lane = tid & 31;
  T* const buf0 = reinterpret_cast<T*>(s_raw);
  T* const buf1 = buf0 + np;
  unsigned* const s_adj = reinterpret_cast<unsigned*>(buf1 + np);
  if (tid < 6) s_cnt[tid >> 1][tid & 1] = 0u;
  for (int v = tid; v < N; v += blockDim.x) {
    bool bad = false;
    const int dv = a.deg ? __ldg(a.deg + v) : a.d;
    if (a.adj16) {
      const uint16_t* row = a.adj16 + (size_t)v * a.d;
#pragma unroll 4
      for (int p = 0; p < pairs; ++p) s_adj[p * np + v] = pack_pair(row, p, dv, v, N, bad);
    } else {
      const int* row = a.adj + (size_t)v * a.d;
#pragma unroll 4
      for (int p = 0; p < pairs; ++p) s_adj[p * np + v] = pack_pair(row, p, dv, v, N, bad);
    }
    if (bad) set_error(a.ctrl, kErrAdj, v);
  }
  __syncthreads();
  if (a.patch && a.patch->valid) {
    // row x[q]'s entry pos[q] becomes x[q ^ 2]; the four rows are distinct
    if (tid < 4) {
      uint16_t* e = reinterpret_cast<uint16_t*>(s_adj + (a.patch->pos[tid] >> 1) * np + a.patch->x[tid]);
      e[a.patch->pos[tid] & 1] = (uint16_t)a.patch->x[tid ^ 2];
    }
    __syncthreads();
  }

  SliceTotals r;
  unsigned g = 0;                      // levels run so far: the rotation of s_cnt
  for (int t = t0; t < t1 && !r.disconnected; t += step) {
    const int phase = t < a.nw1 ? 1 : 2;
    const int first = (phase == 1 ? t : t - a.nw1) * a.width;
    const int l = min(a.width, (phase == 1 ? a.n_src1 : a.ac) - first);
    const int base = (phase == 1 ? 0 : N - a.ac) + first;
    const T full = Row::full(l);
    const int l_lo = max(0, min(l, a.split - base));   // sources among the lo rows
    SliceCount cnt = {(unsigned)a.split * l - l_lo, (unsigned)(N - a.split) * l - (l - l_lo), 0ull, 0ull};
    T* cur = buf0;
    T* nxt = buf1;
    int kk = 0, act = 0;
    for (;; ++kk) {
      const unsigned s0 = g % 3, s1 = (g + 1) % 3;   // this level's and the next's slots
      ++g;
      unsigned n_lo = 0, n_hi = 0;
      if (kk == 0) {
        for (int v = tid; v < N; v += blockDim.x) {
          const T own = Row::bit((unsigned)(v - base)) & full;
          T acc = own;
          for (int p = 0; p < pairs; ++p) {
            const unsigned w = s_adj[p * np + v];
            acc |= Row::bit((w & 0xffffu) - (unsigned)base) | Row::bit((w >> 16) - (unsigned)base);
          }
          acc &= full;
          nxt[v] = acc;
          const unsigned n = Row::popc(acc ^ own);
          if (v < a.split) n_lo += n; else n_hi += n;
        }
      } else {
        for (int v = tid; v < N; v += blockDim.x) {
          const T own = cur[v];
          T acc = own;
          for (int p = 0; p < pairs && acc != full; p += 2) {
            const unsigned w0 = s_adj[p * np + v];
            const unsigned w1 = p + 1 < pairs ? s_adj[(p + 1) * np + v] : w0;
            const T x0 = cur[w0 & 0xffffu], x1 = cur[w0 >> 16], x2 = cur[w1 & 0xffffu], x3 = cur[w1 >> 16];
            acc |= (x0 | x1) | (x2 | x3);
          }
          nxt[v] = acc;
          const unsigned n = Row::popc(acc ^ own);
          if (v < a.split) n_lo += n; else n_hi += n;
        }
      }
      n_lo = __reduce_add_sync(0xffffffffu, n_lo);
      if (a.split < N) n_hi = __reduce_add_sync(0xffffffffu, n_hi);
      if (lane == 0) {
        if (n_lo) atomicAdd(&s_cnt[s0][0], n_lo);
        if (n_hi) atomicAdd(&s_cnt[s0][1], n_hi);
      }
      // the next level's slots: last read after the barrier before the last one
      if (tid < 2) s_cnt[s1][tid] = 0u;
      __syncthreads();
      act = cnt.level(phase, s_cnt[s0][0], s_cnt[s0][1]);
      T* const x = cur;
      cur = nxt;
      nxt = x;
      if (act) break;
    }
    if (phase == 1) { r.s1_lo += cnt.s_lo; r.s1_hi += cnt.s_hi; } else r.s2 += cnt.s_hi;
    r.levels += kk + 1;
    ++r.windows;
    if (act == 2) { r.disconnected = 1; r.diam = N + 1; }
    else r.diam = max(r.diam, kk + 1);
  }
  return r;
}

template <int WORDS>
__global__ void __launch_bounds__(1024, 1) slice_kernel(const SliceArgs a) {
  slice_finish(a, slice_windows<WORDS>(a, (int)blockIdx.x, a.nw1 + a.nw2, (int)gridDim.x));
}

// ---- many small graphs, one launch ---------------------------------------------------
// CTA i takes the windows items[i] of one graph of a batch (see BatchGraph);
// each graph has a record of its own, and the last of its CTAs writes its
// BatchOut.  Nothing to clear before the launch.  With base, graph i is base
// with patch[i] applied (an annealer's candidates, never written out).
template <int WORDS>
__global__ void __launch_bounds__(1024, 1) slice_batch_kernel(const BatchGraph* __restrict__ graphs,
                                                              const SliceItem* __restrict__ items,
                                                              ApspCtrl* __restrict__ records, BatchOut* __restrict__ out,
                                                              const int* __restrict__ base,
                                                              const Swap* __restrict__ patch, const int* stop,
                                                              int* sticky) {
  if (stop && ld_volatile_i32(stop) != 0) return;   // written before the launch: the same in every CTA
  const SliceItem it = items[blockIdx.x];
  const BatchGraph gr = graphs[it.graph];
  SliceArgs a;
  a.adj = base ? base : gr.adj;
  a.patch = base ? patch + it.graph : nullptr;
  a.adj16 = nullptr;
  a.deg = nullptr;
  a.ctrl = records + it.graph;
  a.out = nullptr;
  a.N = gr.N;
  a.d = gr.d;
  a.pairs = (gr.d + 1) / 2;
  a.np = (gr.N + 31) / 32 * 32;
  a.n_src1 = gr.n_src;
  a.split = gr.N;
  a.ac = 0;
  a.groups = gr.groups;
  a.width = 32 * WORDS;
  a.nw1 = (gr.n_src + a.width - 1) / a.width;
  a.nw2 = 0;
  const SliceTotals r = slice_windows<WORDS>(a, it.first, it.end, 1);
  slice_finish(a.ctrl, gr.groups, (unsigned)it.ctas, r, [&](long long sum, long long levels, int windows, int diam,
                                                            int disconnected, int error, int) {
    BatchOut* o = out + it.graph;
    o->sum = sum;
    o->levels = levels;
    o->dense_levels = levels - windows;
    o->diam = diam;
    o->disconnected = disconnected;
    o->windows = windows;
    o->error = error;
    o->done = error ? 0 : 1;
    if (error && sticky) atomicCAS(sticky, 0, error);
  });
}

// ---- lattice graphs: rings of new bits -----------------------------------------
// On a lattice graph a window's new bits are a thin ring around its sources,
// and a level of slice_kernel spends its time on vertices that cannot change.
// Here a level visits only the vertices that received bits: each takes the new
// ones (D = X[v] & ~S[v]), adds them to its row and pushes them to its
// neighbours' words of the next level, S_{k+1}[u] = S_k[u] | OR of the D of the
// rows that u gathers from.  Pushing along row v reaches exactly the rows that
// gather from v when the adjacency is symmetric (u in row v implies v in row
// u); lattice_prep_kernel checks that, and a graph that is not runs every level
// over all vertices instead.  A neighbour that has the bits already is not
// pushed to.  One __syncthreads a level; a window of 6 x 6 sources on a
// 100 x 100 lattice with edges of length 3 changes about 1000 of its 10 000
// vertices a level.
//
// Bound: a level's chain (list entry, row, new bits, pushes, append, barrier: 2.5 us
// a level; 127 million warp instructions in all, issue slots 49 % busy) and the
// last windows (313 windows of 45 to 78 levels on 148 SMs).  100 x 100, degree 4, length 3:
// 347 us with the two preparing kernels, where the persistent kernel took 1305
// us (79 levels of two windows at a grid barrier each) and slice_kernel 670 us.
//
// The sources of a window lie close together, so that their rings overlap:
// strips of kStripRows lattice rows, taken column by column.  The lattice's
// height is read off the vertex numbering (lattice_height_kernel); a wrong
// guess costs time, never the answer.
constexpr int kStripRows = 6;        // about the side of 32 sources

inline size_t slice_push_smem_bytes(int np) { return (size_t)np * 16; }

// Source i of the order: strips of kStripRows rows of the H x (n / H) lattice.
__device__ __forceinline__ int strip_source(int i, int H, int n) {
  const int Wd = n / H;
  const int s = i / (kStripRows * Wd), rem = i - s * kStripRows * Wd;
  const int hs = min(kStripRows, H - s * kStripRows);
  return (rem / hs) * H + s * kStripRows + rem % hs;
}

static __global__ void __launch_bounds__(1024, 1) slice_push_kernel(const SliceArgs a) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  __shared__ unsigned s_cnt[3];        // new bits of a level, in rotation
  __shared__ unsigned s_n[3];          // vertices that received bits, in rotation
  __shared__ int s_next;
  const int N = a.N, np = a.np, dp = a.dp;
  const int tid = threadIdx.x, lane = tid & 31, T = blockDim.x;
  unsigned* const S = reinterpret_cast<unsigned*>(s_raw);
  unsigned* const X0 = S + np;
  unsigned* const X1 = X0 + np;
  uint16_t* const L0 = reinterpret_cast<uint16_t*>(X1 + np);
  uint16_t* const L1 = L0 + np;
  const bool asym = __ldcg(&a.ctrl->asym) != 0;
  const int H = __ldcg(a.height);
  unsigned long long* const ticket = &a.ctrl->cnt[0][0];
  SliceTotals r;
  unsigned g = 0;
  if (tid < 3) { s_cnt[tid] = 0u; s_n[tid] = 0u; }
  // after an error of the preparing kernels the rows are not valid: no window runs
  const int nw = __ldcg(&a.ctrl->error) ? 0 : a.nw1;
  for (int t = blockIdx.x; t < nw && !r.disconnected;) {
    const int first = t * a.width;
    const int l = min(a.width, a.n_src1 - first);
    const unsigned full = l >= 32 ? 0xffffffffu : (1u << l) - 1u;
    SliceCount cnt = {(unsigned)(N - 1) * l, 0u, 0ull, 0ull};
    __syncthreads();                   // the last window's rows and counters are done with
    if (tid == 0) s_next = (int)atomicAdd(ticket, 1ULL) + (int)gridDim.x;
    for (int v = tid; v < 3 * np; v += T) S[v] = 0u;
    if (tid < 3) s_n[tid] = 0u;
    __syncthreads();
    int kk = 0, act = 0;
    if (!asym) {
      for (int i = tid; i < l; i += T) {
        const int v = strip_source(first + i, H, a.n_src1);
        X0[v] = 1u << i;
        L0[i] = (uint16_t)v;
      }
      unsigned* X = X0;
      unsigned* Y = X1;
      uint16_t* L = L0;
      uint16_t* M = L1;
      int n = l;
      __syncthreads();
      // step 0 spreads S_0; step k + 1 makes S_{k+1} (level k)
      for (kk = -1;; ++kk) {
        const unsigned s0 = g % 3, s1 = (g + 1) % 3;
        ++g;
        unsigned n_new = 0;
        for (int i0 = tid - lane; i0 < n; i0 += T) {      // warp-uniform
          const int i = i0 + lane;
          const int v = i < n ? L[i] : -1;
          unsigned D = 0u;
          const uint2* row = reinterpret_cast<const uint2*>(a.adj16 + (size_t)max(v, 0) * dp);
          uint2 w = __ldg(row);
          if (v >= 0) {
            const unsigned own = S[v];
            D = X[v] & ~own;
            X[v] = 0u;
            if (D) {
              S[v] = own | D;
              n_new += __popc(D);
            }
          }
          if (!__any_sync(0xffffffffu, D != 0u)) continue;
          for (int j = 0;;) {
            const int u[4] = {(int)(w.x & 0xffffu), (int)(w.x >> 16), (int)(w.y & 0xffffu), (int)(w.y >> 16)};
            bool add[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              // a stale S[u] only pushes bits that u has by then
              add[q] = (D & ~S[u[q]]) != 0u;
              if (add[q]) add[q] = atomicOr(Y + u[q], D) == 0u;
            }
            unsigned b[4], c = 0u;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              b[q] = __ballot_sync(0xffffffffu, add[q]);
              c += __popc(b[q]);
            }
            if (c) {
              unsigned at = 0;
              if (lane == 0) at = atomicAdd(&s_n[s0], c);
              at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                if (add[q]) M[at + __popc(b[q] & ((1u << lane) - 1u))] = (uint16_t)u[q];
                at += __popc(b[q]);
              }
            }
            if ((j += 4) >= dp) break;
            w = __ldg(row + (j >> 2));
          }
        }
        n_new = __reduce_add_sync(0xffffffffu, n_new);
        if (lane == 0 && n_new) atomicAdd(&s_cnt[s0], n_new);
        // the next step's slots: last read after the barrier before the last one
        if (tid == 0) { s_cnt[s1] = 0u; s_n[s1] = 0u; }
        __syncthreads();
        n = (int)s_n[s0];
        unsigned* const x = X;
        X = Y;
        Y = x;
        uint16_t* const y = L;
        L = M;
        M = y;
        if (kk < 0) continue;
        act = cnt.level(1, s_cnt[s0], 0u);
        if (act) break;
      }
    } else {
      for (int i = tid; i < l; i += T) X0[strip_source(first + i, H, a.n_src1)] = 1u << i;
      unsigned* cur = X0;
      unsigned* nxt = X1;
      __syncthreads();
      for (;; ++kk) {
        const unsigned s0 = g % 3, s1 = (g + 1) % 3;
        ++g;
        unsigned n_new = 0;
        for (int v = tid; v < N; v += T) {
          const uint2* row = reinterpret_cast<const uint2*>(a.adj16 + (size_t)v * dp);
          const unsigned own = cur[v];
          unsigned acc = own;
          for (int j = 0; j < dp && acc != full; j += 4) {
            const uint2 w = __ldg(row + (j >> 2));
            acc |= (cur[w.x & 0xffffu] | cur[w.x >> 16]) | (cur[w.y & 0xffffu] | cur[w.y >> 16]);
          }
          nxt[v] = acc;
          n_new += __popc(acc ^ own);
        }
        n_new = __reduce_add_sync(0xffffffffu, n_new);
        if (lane == 0 && n_new) atomicAdd(&s_cnt[s0], n_new);
        if (tid == 0) s_cnt[s1] = 0u;
        __syncthreads();
        act = cnt.level(1, s_cnt[s0], 0u);
        unsigned* const x = cur;
        cur = nxt;
        nxt = x;
        if (act) break;
      }
    }
    r.s1_lo += cnt.s_lo;
    r.levels += kk + 1;
    ++r.windows;
    if (act == 2) { r.disconnected = 1; r.diam = N + 1; }
    else r.diam = max(r.diam, kk + 1);
    t = s_next;
  }
  slice_finish(a, r);
}

// The rows of a lattice graph for slice_push_kernel: row rh[i] of out16 holds
// rh of row i's entries (grid/evaluation.c:148-151), padded with its own id to
// dp entries (past deg[i] too, non-regular grids).  Checks what
// relabel_adjacency_kernel checks, reports an asymmetric adjacency in
// ctrl->asym, marks in diff[] the id differences of the edges and in inv[] the
// inverse permutation (both zero / -1 on entry).
template <typename ID>
__global__ void lattice_prep_kernel(const ID* __restrict__ adj, const int* __restrict__ rh,
                                    const int* __restrict__ deg, uint16_t* __restrict__ out16,
                                    int* __restrict__ inv, unsigned* __restrict__ diff, int N, int d, int dp,
                                    ApspCtrl* ctrl) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int r = rh[i];
  const int di = deg ? deg[i] : d;
  if ((unsigned)di > (unsigned)d) { set_error(ctrl, kErrDegree, i); return; }
  if ((unsigned)r >= (unsigned)N) { set_error(ctrl, kErrPerm, i); return; }
  inv[r] = i;
  uint16_t* out = out16 + (size_t)r * dp;
  for (int j = 0; j < dp; ++j) {
    const unsigned nb = j < di ? (unsigned)adj[(size_t)i * d + j] : (unsigned)i;
    if (nb >= (unsigned)N) { set_error(ctrl, kErrAdj, i); return; }
    const int rn = rh[nb];
    if ((unsigned)rn >= (unsigned)N) { set_error(ctrl, kErrPerm, (int)nb); return; }
    out[j] = (uint16_t)rn;
    if (j < di) {
      const int dn = deg ? min(max(deg[nb], 0), d) : d;
      bool back = (int)nb == i;
      for (int k = 0; k < dn && !back; ++k) back = (int)adj[(size_t)nb * d + k] == i;
      if (!back) ctrl->asym = 1;
      const unsigned df = (unsigned)abs(rn - r), m = 1u << (df & 31);
      if (!(__ldcg(diff + (df >> 5)) & m)) atomicOr(diff + (df >> 5), m);
    }
  }
}

// One CTA: every vertex is the image of one (kErrPerm otherwise), and the
// lattice's height.  Vertex x * H + y (grid/common.c:53-61) with edges of
// Manhattan length at most r has id differences 1 .. r, then H - (r - 1) ..
// H + (r - 1): the middle of the second run of differences is H.  A numbering
// without that structure gives H = n_src (the sources in id order).  Clears
// diff[] for the next launch.
static __global__ void __launch_bounds__(1024) lattice_height_kernel(const int* __restrict__ inv, unsigned* __restrict__ diff,
                                                              int N, int n_src, int* __restrict__ height,
                                                              ApspCtrl* ctrl) {
  __shared__ int s_at[3];              // first gap, first difference past it, first gap past that
  const int words = (N + 31) / 32;
  for (int v = threadIdx.x; v < N; v += blockDim.x)
    if (inv[v] < 0) set_error(ctrl, kErrPerm, v);
  if (threadIdx.x < 3) s_at[threadIdx.x] = N;
  __syncthreads();
  for (int k = 0; k < 3; ++k) {
    const int from = k == 0 ? 1 : s_at[k - 1];
    for (int w = from / 32 + (int)threadIdx.x; w < words; w += blockDim.x) {
      unsigned m = k == 1 ? diff[w] : ~diff[w];
      if (w == from / 32) m &= 0xffffffffu << (from & 31);
      if (m) {
        atomicMin(&s_at[k], w * 32 + __ffs(m) - 1);
        break;
      }
    }
    __syncthreads();
  }
  for (int w = threadIdx.x; w < words; w += blockDim.x) diff[w] = 0u;
  if (threadIdx.x == 0) {
    const int h = (s_at[1] + s_at[2]) / 2;
    *height = s_at[2] < N && h > 1 && n_src % h == 0 ? h : n_src;
  }
}

}  // namespace ggb
