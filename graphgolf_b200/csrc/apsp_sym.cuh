// apsp_sym.cuh -- large graphs with a symmetric adjacency: half of every dense
// level (sm_100a).
//
// When u in row v implies v in row u (every undirected graph; sym_ball_kernel
// checks it), distances are symmetric: bit s of S_k[v] is bit v of S_k[s].
// Windows of W sources are taken in order, and window i sweeps only the rows
// v >= i*W.  The rows below are the transposes of blocks that the earlier
// windows have made, kept per level in a triangular store; a transpose reads
// and writes each row part once where the sweep gathers d of them.  A pair
// (v, s) in two different blocks is counted twice, one in the same block once.
//
//   sym_ball_kernel   S_3 of every window (three-hop balls built in shared
//                     memory, one warp per vertex), the totals of S_1 .. S_3,
//                     and the symmetry check;
//   apsp_sym_kernel   window 0 level by level (all rows), until so few pairs
//                     are unreached that a list can hold those of all windows:
//                     that level is k*.  The other windows run levels 4 .. k*-1
//                     (sweep, transpose, store) and then one last sweep to
//                     level k* that writes no row: it counts, and lists the
//                     pairs still unreached.  Nothing is decided between the
//                     levels of a window; the barriers are split, and the last
//                     sweep of one window runs while the one behind the next
//                     window's first level fills;
//                     then the listed pairs are resolved level by level: (v, s)
//                     is reached at k+1 when (u, s) was reached by k for some u
//                     in row v, looked up in a hash table of the listed pairs.
//
// Everything the totals need is the number of unreached pairs per level,
// U_k = N^2 - |S_k|: the distance sum is the sum of U_k and the diameter the
// first k with U_k = 0 (general/evaluation.c:183-200 summed over the windows).
// A level, or a pass over the list, that reaches nothing new is a fixed point:
// the graph is disconnected.  An asymmetric adjacency, more levels than the
// store holds, or more unreached pairs than the list holds set ctrl->fallback,
// and the persistent kernel launched behind this one, which returns at once
// otherwise, evaluates the graph.
//
// Measured (whole call, us, against the persistent kernel with its ball):
// N = 65536, d = 16 1218 / 1836 (ball 271 / 380, sweeps 910 / 1425); d = 8
// 1528 / 2312; N = 16384, d = 12 182 / 216; N = 100000, d = 12 3240 / 6930;
// N = 262144, d = 12 30 900 / 67 900.  Bound: L2 gathers (N = 65536,
// d = 16: 12.1 GB through L2 at 13.1 TB/s, and 2.4 GB read from HBM, where the
// ball and part of the store lie), and for the ball the load/store data pipe
// (92 % busy).  Tried and not kept: S_3 in halves too (the ball kernel 9 %
// faster, its transposes cost more), sweeps that write every row twice instead
// of choosing between two places (4 % slower), a prefetch of the next window's
// ball slice into L2 (2 % slower), windows of 1024 to 2048 sources, 768 or 1024
// threads with 6 or 4 neighbour rows in flight (10 to 20 % slower), half a warp
// per 1 KB row with two parts a lane (5 % slower).
//
// A graph that is left to the persistent kernel has paid for the ball and the
// first window, and that kernel runs without a ball of its own.  Whole call, us,
// against the persistent kernel with its ball, at N = 65536 (and 20000): one
// asymmetric row, d = 8 2970 / 2290 (361 / 354), d = 12 2810 / 2080 (385 / 314); a
// random core whose vertices carry a leaf each, rows of 7, 3880 / 3200 (515 /
// 459); two components, d = 8, which stall in the first window, 657 / 384 (229 /
// 150).  Circulants of 24 to 334 levels gain by the wider windows at
// N = 65536 (334 levels 108 / 141 ms) and lose 1 to 10 % at 20000 and 30000.  Warps
// that stop working once the list is too long changed nothing: the time lies
// before that.
#pragma once
#include "apsp_kernel.cuh"

namespace ggb {

constexpr int kSymFirst = 4;            // first swept level (S_3 comes from the ball)
constexpr int kSymLevels = 16;          // levels the counters hold past which the kernel falls back
constexpr unsigned kSymList = 1u << 22; // listed pairs
// Pairs predicted for the list at k*, and at the last level the store can
// hold.  A listed pair costs about 1 ns of hashing and look-ups: with 2^20 as
// the only bound N = 20000, d = 5 took 1010 us, with 2^16 (one more sweep) 278.
constexpr unsigned kSymTarget = 1u << 16, kSymTargetLast = 1u << 20;
constexpr unsigned long long kSymEmpty = ~0ull;

struct SymArgs {
  uint4* ball;                    // [window][N][R]: S_3, window i's rows from i * W on
  uint4* tri;                     // stored levels, tri_cells each: window i's rows from (i + 1) * W on
  size_t tri_cells;
  int stored;                     // levels the store holds (4, 5, ...)
  unsigned long long* cnt;        // zeroed: [0] |S_1|, [1] |S_2|, [2 + L] window 0 at level L,
                                  // [2 + kSymLevels + 8 + L] weighted |S_L| of the other windows
  unsigned* list_n;               // zeroed: [0] listed pairs, [1 + p] pairs left after pass p
  unsigned long long* list;       // (v << 32) | s
  unsigned long long* hash;       // 2 * kSymList keys
  unsigned char* hlev;            // level of a hashed pair, 255: unreached
};
constexpr int kSymCnt0 = 2, kSymCntW = 2 + kSymLevels + 8, kSymCounters = kSymCntW + kSymLevels + 8;
constexpr int kSymPasses = 250;         // passes over the list (levels fit a byte), then the kernel falls back

// ---- S_3 of every window ----------------------------------------------------------
// One warp per vertex: the row of all sources within three steps, in shared
// memory (n_row uint4), beside the one- and two-hop ids.
__host__ __device__ __forceinline__ int sym_ball_warp_u4(int N, int d) { return ball_row_u4(N) + (d + d * d + 3) / 4; }

template <int VEC>
__global__ void __launch_bounds__(kBallThreads, 3) sym_ball_kernel(const int* __restrict__ adj, int N, int d, int R,
                                                                   uint4* __restrict__ ball,
                                                                   unsigned long long* __restrict__ cnt,
                                                                   ApspCtrl* ctrl) {
  extern __shared__ uint4 s_ball[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int row_u4 = ball_row_u4(N), log_r = 31 - __clz(R), live_u4 = ((N + 128 * R - 1) >> (7 + log_r)) << log_r;
  uint4* const row4 = s_ball + (size_t)warp * sym_ball_warp_u4(N, d);
  unsigned* const row = reinterpret_cast<unsigned*>(row4);
  int* const nb1 = reinterpret_cast<int*>(row4 + row_u4);
  int* const nb2 = nb1 + d;
  const unsigned all = d >= 32 ? 0xffffffffu : (1u << d) - 1u;
  const int per = d / VEC, rpi = 32 / per;         // lanes a row, rows a step (per <= 32)
  const int roff = lane / per, part = lane - roff * per;
  const bool active = roff < rpi;
  bool bad = false, asym = false;
  unsigned long long c1 = 0, c2 = 0, c3 = 0;
  for (long long v = (long long)blockIdx.x * warps + warp; v < N; v += (long long)gridDim.x * warps) {
    for (int i = lane; i < row_u4; i += 32) row4[i] = make_uint4(0u, 0u, 0u, 0u);
    int x1 = -1;
    if (lane < d) {
      x1 = __ldg(adj + v * d + lane);
      if ((unsigned)x1 >= (unsigned)N) { bad = true; x1 = -1; }
      nb1[lane] = x1;
    }
    __syncwarp();
    // S_1 = {v} u N(v), counting the bits that are new
    unsigned n1 = 0, n2 = 0;
    if (lane == 0) { row[v >> 5] = 1u << (v & 31); n1 = 1; }
    __syncwarp();
    if (x1 >= 0) {
      const unsigned m = 1u << (x1 & 31);
      n1 += !(smem_or_old(row + (x1 >> 5), m) & m);
    }
    __syncwarp();
    // S_2: the neighbours' rows; row j must hold v.  An id equal to v is not
    // kept: its row is row v again.
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
          int x = val[t].at(e);
          if (x == (int)v) {
            back |= 1u << j;
            x = -1;
          } else if ((unsigned)x < (unsigned)N) {
            const unsigned m = 1u << (x & 31);
            n2 += !(smem_or_old(row + (x >> 5), m) & m);
          }
          nb2[j * d + part * VEC + e] = x;
        }
      }
    }
    if (__reduce_or_sync(0xffffffffu, back) != all) asym = true;
    c1 += n1;
    c2 += n1 + n2;
    __syncwarp();
    // S_3
    scatter_plain<VEC>(adj, N, d, nb2, d * d, row, N, lane);
    __syncwarp();
    unsigned n3 = 0;
    for (int idx = lane; idx < live_u4; idx += 32) {
      const uint4 x = idx < row_u4 ? row4[idx] : make_uint4(0u, 0u, 0u, 0u);
      st_cg(ball + ((((size_t)(idx >> log_r) * N + v) << log_r) | (unsigned)(idx & (R - 1))), x);
      n3 += popc4(x);
    }
    c3 += n3;
    __syncwarp();
  }
  if (bad) set_error(ctrl, kErrAdj, (int)blockIdx.x);
  if (asym) ctrl->asym = 1;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    c1 += __shfl_xor_sync(0xffffffffu, c1, o);
    c2 += __shfl_xor_sync(0xffffffffu, c2, o);
    c3 += __shfl_xor_sync(0xffffffffu, c3, o);
  }
  if (lane == 0) {
    atomicAdd(cnt, c1);
    atomicAdd(cnt + 1, c2);
    atomicAdd(cnt + kSymCntW + kSymFirst - 1, c3);
  }
}

// ---- transposes ---------------------------------------------------------------------
// 32 x 32 transposes, one word a lane: bit r of lane c's word becomes bit c of
// lane r's.  Five exchanges; each rotates the partner's word into place and
// merges it under a mask (three instructions), shift and mask by lane.
struct Transpose32 {
  unsigned keep[5];
  int rot[5];
  __device__ __forceinline__ explicit Transpose32(int lane) {
    const unsigned low[5] = {0x0000ffffu, 0x00ff00ffu, 0x0f0f0f0fu, 0x33333333u, 0x55555555u};
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      const int m = 16 >> f;
      keep[f] = (lane & m) ? ~low[f] : low[f];
      rot[f] = (lane & m) ? 32 - m : m;
    }
  }
  __device__ __forceinline__ unsigned operator()(unsigned x) const {
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      const unsigned y = __shfl_xor_sync(0xffffffffu, x, 16 >> f);
      const unsigned z = __funnelshift_l(y, y, rot[f]);
      x = (x & keep[f]) | (z & ~keep[f]);
    }
    return x;
  }
};

// A 256 x 256 bit tile by one warp: src = the 32 bytes of its first row (rows
// src_stride uint4 apart, `rows` of them, the others zero), dst likewise; every
// access is a whole 32-byte sector.
__device__ __forceinline__ void transpose_tile(const uint4* __restrict__ src, size_t src_stride, int rows,
                                               uint4* __restrict__ dst, size_t dst_stride, int lane,
                                               const Transpose32& tr) {
  unsigned w[8][8];   // [group of 32 rows][word]
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    const int r = 32 * g + lane;
    uint4 x[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
    if (r < rows) ld_cg2(src + (size_t)r * src_stride, x);
    w[g][0] = x[0].x; w[g][1] = x[0].y; w[g][2] = x[0].z; w[g][3] = x[0].w;
    w[g][4] = x[1].x; w[g][5] = x[1].y; w[g][6] = x[1].z; w[g][7] = x[1].w;
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) {
#pragma unroll
    for (int g = 0; g < 8; ++g) w[g][c] = tr(w[g][c]);
    const uint4 y[2] = {make_uint4(w[0][c], w[1][c], w[2][c], w[3][c]),
                        make_uint4(w[4][c], w[5][c], w[6][c], w[7][c])};
    st_cg2(dst + (size_t)(32 * c + lane) * dst_stride, y);
  }
}

// ---- one half sweep -----------------------------------------------------------------
// Appends the unset bits among the `nv` valid ones of word `x` (bit b is
// source s0 + b) of row v; in the diagonal block only sources below v.  A
// thread that has seen the list full (`full`) appends no more: the unreached
// pairs of a graph whose first window lies close to everything while the others
// do not can exceed 2^32 (from 92 682 vertices on), but the counter ends below
// cap + 32 a thread.
__device__ __forceinline__ void list_missing(const SymArgs& s, unsigned x, int nv, int v, int s0, bool diag,
                                             bool& full, unsigned cap = kSymList) {
  if (full) return;
  unsigned m = ~x & (nv >= 32 ? 0xffffffffu : (1u << max(nv, 0)) - 1u);
  if (diag) {
    const int b = v - s0;                       // sources s0 .. v - 1
    m &= b >= 32 ? 0xffffffffu : b <= 0 ? 0u : (1u << b) - 1u;
  }
  if (!m) return;
  unsigned at = atomicAdd(s.list_n, (unsigned)__popc(m));
  full = at >= cap;
  while (m) {
    const int b = __ffs(m) - 1;
    m &= m - 1;
    if (at < cap) s.list[at] = ((unsigned long long)(unsigned)v << 32) | (unsigned)(s0 + b);
    ++at;
  }
}

__device__ __forceinline__ unsigned word_of(const uint4 (&r)[2], int k) {
  const uint4& q = k < 4 ? r[0] : r[1];
  return (k & 3) == 0 ? q.x : (k & 3) == 1 ? q.y : (k & 3) == 2 ? q.z : q.w;
}

// The rows of one window at one level lie in two places: row u at
// (u < split ? lo : hi) + u * R.
struct SymRows {
  const uint4* lo;
  const uint4* hi;
  int split;
};

// Rows first .. N - 1 of one level, LP lanes a row and 32 bytes a lane and
// part: S_{k+1} from src, rows below v_next into lo and the others into hi
// (row u at + u * R).  LAST: nothing is written; the unreached pairs are
// listed.  c_diag counts rows below v_next, c_off the rest.
template <int R, bool LAST>
__device__ __forceinline__ void sym_sweep(const SymArgs& s, const SymRows src, uint4* __restrict__ lo,
                                          uint4* __restrict__ hi, const int* __restrict__ adj, int N, int d, int vec4,
                                          int first, int v_next, int l, bool early, long long warp_id,
                                          long long n_warps, unsigned& c_diag, unsigned& c_off, bool& full) {
  constexpr int LP = R / 2 < 32 ? R / 2 : 32;     // lanes a row
  constexpr int PPL = R / (2 * LP);               // 32-byte parts a lane
  constexpr int G = 32 / LP;                      // rows a warp and step
  constexpr int U = 8 / PPL;                      // neighbour rows in flight
  const int lane = threadIdx.x & 31, h = lane / LP, hl = lane % LP;
  const bool wide = l == 128 * R;
  for (long long vb = first + warp_id * G; vb < N; vb += n_warps * G) {
    const bool live = vb + h < N;
    const int v = (int)(live ? vb + h : vb);      // a dead group reads a live row and drops the result
    const int* arow = adj + (long long)v * d;
    uint4 acc[PPL][2];
#pragma unroll
    for (int p = 0; p < PPL; ++p)
      ld_cg2((v < src.split ? src.lo : src.hi) + (size_t)v * R + 2 * (hl + p * LP), acc[p]);
    bool need[PPL];
#pragma unroll
    for (int p = 0; p < PPL; ++p) need[p] = true;
    for (int j = 0; j < d; j += U) {
      int u[U];
      if (vec4 && j + U <= d) {
#pragma unroll
        for (int q = 0; q < U; q += 4) {
          const int4 t = __ldg(reinterpret_cast<const int4*>(arow + j + q));
          u[q] = t.x; u[q + 1] = t.y; u[q + 2] = t.z; u[q + 3] = t.w;
        }
      } else {
#pragma unroll
        for (int q = 0; q < U; ++q) u[q] = j + q < d ? __ldg(arow + j + q) : v;
      }
      if (wide && (j > 0 || early)) {
        // parts whose 256 bits are all set need no further gathers (before the
        // first group too, at the price of a round trip, where most are full)
#pragma unroll
        for (int p = 0; p < PPL; ++p)
          need[p] = (acc[p][0].x & acc[p][0].y & acc[p][0].z & acc[p][0].w & acc[p][1].x & acc[p][1].y & acc[p][1].z &
                     acc[p][1].w) != 0xffffffffu;
        bool any = false;
#pragma unroll
        for (int p = 0; p < PPL; ++p) any = any || need[p];
        if (!__any_sync(0xffffffffu, any)) break;
      }
      uint4 x[U][PPL][2];
#pragma unroll
      for (int q = 0; q < U; ++q)
#pragma unroll
        for (int p = 0; p < PPL; ++p) {
          if (need[p] && j + q < d) {
            ld_cg2((u[q] < src.split ? src.lo : src.hi) + (size_t)u[q] * R + 2 * (hl + p * LP), x[q][p]);
          } else {
            x[q][p][0] = make_uint4(0u, 0u, 0u, 0u);
            x[q][p][1] = make_uint4(0u, 0u, 0u, 0u);
          }
        }
#pragma unroll
      for (int q = 0; q < U; ++q)
#pragma unroll
        for (int p = 0; p < PPL; ++p) {
          or_into(acc[p][0], x[q][p][0]);
          or_into(acc[p][1], x[q][p][1]);
        }
    }
    unsigned cc = 0;
#pragma unroll
    for (int p = 0; p < PPL; ++p) cc += popc4(acc[p][0]) + popc4(acc[p][1]);
    if (!live) continue;
    const bool diag = v < v_next;
    if (diag) c_diag += cc; else c_off += cc;
    if constexpr (LAST) {
#pragma unroll
      for (int p = 0; p < PPL; ++p) {
        const int b0 = 256 * (hl + p * LP);        // first bit of the part
        const int nv = min(256, l - b0);
        if (nv > 0 && popc4(acc[p][0]) + popc4(acc[p][1]) != (unsigned)nv)
          for (int k = 0; k < 8; ++k) list_missing(s, word_of(acc[p], k), nv - 32 * k, v, first + b0 + 32 * k, diag, full);
      }
    } else {
#pragma unroll
      for (int p = 0; p < PPL; ++p) {
        st_cg2((diag ? lo : hi) + (size_t)v * R + 2 * (hl + p * LP), acc[p]);
      }
    }
  }
}

// The rows below window i of one level, from the blocks of the earlier
// windows: 256 x 256 tiles over the warps.  Row v of window k lies at
// src + k_base(k) + v * R.
template <int R, typename KBase>
__device__ __forceinline__ void sym_transposes(const uint4* __restrict__ src, KBase k_base, uint4* __restrict__ dst,
                                               int i, int l, long long warp_id, long long n_warps) {
  constexpr int W = 128 * R, TU = W / 256;
  const int lane = threadIdx.x & 31;
  const Transpose32 tr(lane);
  // (a last window of fewer sources has the rest of its columns cleared)
  const long long tasks = (long long)i * TU * TU;
  for (long long t = warp_id; t < tasks; t += n_warps) {
    const int k = (int)(t / (TU * TU)), q = (int)(t % (TU * TU));
    const int tv = q / TU, tu = q % TU;
    const uint4* rows = src + k_base(k) + (long long)(i * W + 256 * tv) * R + 2 * tu;
    transpose_tile(rows, R, l - 256 * tv, dst + (size_t)(k * W + 256 * tu) * R + 2 * tv, R, lane, tr);
  }
}

__device__ __forceinline__ unsigned sym_slot(unsigned long long key) {
  key ^= key >> 31;
  key *= 0x9e3779b97f4a7c15ull;
  return (unsigned)(key >> 32);
}

// Warp sums of x added to *to (shared or global).
__device__ __forceinline__ void sym_add(unsigned long long x, unsigned long long* to) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  if ((threadIdx.x & 31) == 0 && x) atomicAdd(to, x);
}

// grid_barrier in two halves, with work of its own between them.
__device__ __forceinline__ void grid_arrive(ApspCtrl* c) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&c->bar, 1ULL);
  }
}
__device__ __forceinline__ bool grid_wait(ApspCtrl* c, unsigned long long target, long long timeout_ns, int* s_flag) {
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    const unsigned long long t0 = globaltimer_ns();
    while (ld_acquire_u64(&c->bar) < target) {
      if (ld_volatile_i32(&c->error) != 0) { ok = 0; break; }
      if ((long long)(globaltimer_ns() - t0) > timeout_ns) {
        set_error(c, kErrTimeout, (int)blockIdx.x);
        ok = 0;
        break;
      }
      __nanosleep(64);
    }
    __threadfence();
    *s_flag = ok;
  }
  __syncthreads();
  return *s_flag != 0;
}

// Lists the unreached pairs of window 0 from its rows at level k*.
template <int R>
__device__ __forceinline__ void sym_list_window0(const SymArgs& s, const SymRows rows, int N, int l,
                                                 long long warp_id, long long n_warps, bool& full) {
  constexpr int LP = R / 2 < 32 ? R / 2 : 32, PPL = R / (2 * LP), G = 32 / LP;
  const int lane = threadIdx.x & 31, h = lane / LP, hl = lane % LP;
  for (long long vb = warp_id * G; vb + h < N; vb += n_warps * G) {
    const int v = (int)(vb + h);
#pragma unroll
    for (int p = 0; p < PPL; ++p) {
      uint4 x[2];
      ld_cg2((v < rows.split ? rows.lo : rows.hi) + (size_t)v * R + 2 * (hl + p * LP), x);
      const int b0 = 256 * (hl + p * LP), nv = min(256, l - b0);
      if (nv > 0 && popc4(x[0]) + popc4(x[1]) != (unsigned)nv)
        for (int k = 0; k < 8; ++k) list_missing(s, word_of(x, k), nv - 32 * k, v, b0 + 32 * k, v < l, full);
    }
  }
}

enum : int { kSymFailed = 0, kSymResolved = 1, kSymStalled = 2, kSymTooLong = 3 };

// Resolves the n > 0 listed pairs, unreached at level k, level by level on the
// `nt` threads of a team (this one is number tid): pass p makes level k + 1 + p.
// late receives twice the sum of the unreached pairs at levels k, k + 1, ...,
// passes the levels it took; left[p] (zeroed) the pairs left after pass p.
template <typename Barrier>
__device__ __forceinline__ int sym_resolve(const SymArgs& s, unsigned* left, const int* __restrict__ adj, int d,
                                           unsigned n, int max_passes, unsigned tid, unsigned nt, Barrier barrier,
                                           unsigned long long& late, int& passes) {
  unsigned size = 1024;
  while (size < 2 * n) size <<= 1;
  const unsigned mask = size - 1;
  for (unsigned i = tid; i < size; i += nt) {
    __stcg(s.hash + i, kSymEmpty);
    s.hlev[i] = 255;
  }
  if (!barrier()) return kSymFailed;
  auto key_of_pair = [](unsigned x, unsigned y) {
    return x > y ? ((unsigned long long)x << 32) | y : ((unsigned long long)y << 32) | x;
  };
  for (unsigned i = tid; i < n; i += nt) {
    const unsigned long long e = __ldcg(s.list + i);
    const unsigned long long key = key_of_pair((unsigned)(e >> 32), (unsigned)e);
    unsigned h = sym_slot(key) & mask;
    while (atomicCAS(s.hash + h, kSymEmpty, key) != kSymEmpty) h = (h + 1) & mask;
  }
  if (!barrier()) return kSymFailed;
  auto find = [&](unsigned long long key) -> unsigned {      // its slot, or ~0 when not listed
    unsigned h = sym_slot(key) & mask;
    for (;;) {
      const unsigned long long k = __ldcg(s.hash + h);
      if (k == key) return h;
      if (k == kSymEmpty) return ~0u;
      h = (h + 1) & mask;
    }
  };
  unsigned now = n;
  for (int p = 0;; ++p) {
    // a pair's level is stored as p + 1
    late += 2ull * now;
    unsigned rest = 0;
    for (unsigned i = tid; i < n; i += nt) {
      const unsigned long long e = __ldcg(s.list + i);
      const unsigned v = (unsigned)(e >> 32), src = (unsigned)e;
      const unsigned h = find(key_of_pair(v, src));
      if (__ldcg(s.hlev + h) != 255) continue;
      bool reached = false;
      for (int j = 0; j < d && !reached; ++j) {
        const unsigned u = (unsigned)__ldg(adj + (size_t)v * d + j);
        const unsigned f = find(key_of_pair(u, src));
        reached = f == ~0u || __ldcg(s.hlev + f) <= p;
      }
      if (reached) __stcg(s.hlev + h, (unsigned char)(p + 1));
      else ++rest;
    }
    rest = __reduce_add_sync(0xffffffffu, rest);
    if ((threadIdx.x & 31) == 0 && rest) atomicAdd(left + p, rest);
    if (!barrier()) return kSymFailed;
    const unsigned was = now;
    now = __ldcg(left + p);
    passes = p + 1;
    if (now == 0) return kSymResolved;
    if (now == was) return kSymStalled;
    if (p + 1 == max_passes) return kSymTooLong;
  }
}

template <int R>
__global__ void __launch_bounds__(kThreads, 1) apsp_sym_kernel(const ApspArgs a, const SymArgs s) {
  __shared__ int s_flag;
  __shared__ int s_go, s_early;                              // window 0's decisions
  __shared__ unsigned long long s_acc[kSymLevels + 8];       // this CTA's weighted |S_L|
  constexpr int W = 128 * R;
  const int N = a.N, d = a.d, nwin = (N + W - 1) / W;
  const long long warp_id = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5);
  const long long n_warps = (long long)gridDim.x * kWarps;
  const unsigned grid = gridDim.x;
  unsigned long long bar_target = 0;
  ApspCtrl* const ctrl = a.ctrl;
  const size_t cells = (size_t)N * R;
  unsigned nbuf = 4;
  auto buf = [&](unsigned q) -> uint4* { return a.buf0 + (q % nbuf) * cells; };
  auto barrier = [&]() -> bool {
    bar_target += grid;
    return grid_barrier(ctrl, bar_target, a.timeout_ns, &s_flag);
  };
  if (ld_volatile_i32(&ctrl->error) != 0) return;      // the ball kernel's checks
  if (threadIdx.x < kSymLevels + 8) s_acc[threadIdx.x] = 0ULL;
  __syncthreads();
  bool fallback = ld_volatile_i32(&ctrl->asym) != 0, stalled = false;
  int last = 0;                                        // k*
  unsigned early = 0u;                                 // levels made from one that is nearly full
  int sweeps = 0;
  unsigned q = 0;                                      // dense writes so far: the buffer in turn
  bool full = false;                                   // this thread has seen the list full
  if (!fallback) {
    const int l = min(W, N);
    // row v of window k at a stored level lies at level + tri_base(k) + v * R, from (k + 1) * W on
    auto tri_base = [&](int k) -> long long {
      return ((long long)k * N - (long long)W * ((long long)k * (k + 1) / 2) - (long long)(k + 1) * W) * R;
    };
    auto ball_base = [&](int k) -> long long { return (long long)k * (long long)cells; };
    auto rows3 = [&](int i) -> SymRows { return {s.ball + ball_base(i), s.ball + ball_base(i), 0}; };
    // ---- window 0, level by level ------------------------------------------------
    unsigned long long prev = 0;
    SymRows src = rows3(0);
    for (int L = kSymFirst;; ++L) {
      uint4* const dst = buf(q++);
      uint4* const hi = L - kSymFirst < s.stored ? s.tri + (size_t)(L - kSymFirst) * s.tri_cells + tri_base(0) : dst;
      unsigned cd = 0, co = 0;
      sym_sweep<R, false>(s, src, dst, hi, a.adj, N, d, a.vec4, 0, l, l, (early >> L) & 1u, warp_id,
                          n_warps, cd, co, full);
      ++sweeps;
      sym_add((unsigned long long)cd + co, s.cnt + kSymCnt0 + L);
      // the weighted count holds rows of the window's own block once, the others twice
      sym_add((unsigned long long)cd + 2ull * co, s_acc + L);
      if (!barrier()) return;
      if (threadIdx.x == 0) {
        const unsigned long long c = ld_acquire_u64(s.cnt + kSymCnt0 + L);
        const unsigned long long miss = (unsigned long long)N * l - c;
        const bool kept = L - kSymFirst < s.stored;
        s_go = miss * (unsigned)nwin / 2 <= (kept ? kSymTarget : kSymTargetLast) ? 1 : c == prev ? 2 : kept ? 0 : 3;
        // under 0.5 % of the bits unset: a 256-bit part is full more than once in four
        s_early = miss * 200 <= (unsigned long long)N * l;
        prev = c;
      }
      __syncthreads();
      const int go = s_go;
      if (s_early) early |= 2u << L;
      __syncthreads();
      src = {dst, hi, l};
      if (go == 0) continue;
      last = L;
      stalled = go == 2;
      fallback = go == 3;
      break;
    }
    if (!fallback && !stalled) {
      // The last sweep of window i: nobody waits for its rows, so it runs while
      // the barrier behind window i + 1's first level fills.  Its source must
      // stay alive until every CTA is past the barrier behind window i + 1's
      // second level, or its first if it has one only; by then that window has
      // written two buffers, and with three levels or more a third.
      q = (q - 1) % nbuf + 1;
      nbuf = last - kSymFirst >= 3 ? 4 : 3;
      auto finish = [&](int i, const SymRows from) {
        if (i == 0) {
          sym_list_window0<R>(s, from, N, l, warp_id, n_warps, full);
          return;
        }
        const int first = i * W, li = min(W, N - first);
        unsigned cd = 0, co = 0;
        sym_sweep<R, true>(s, from, nullptr, nullptr, a.adj, N, d, a.vec4, first, first + li, li, (early >> last) & 1u,
                           warp_id, n_warps, cd, co, full);
        sym_add((unsigned long long)cd + 2ull * co, s_acc + last);
      };
      SymRows done = src;                              // rows of window i - 1 one level below k* (window 0: at k*)
      for (int i = 1; i < nwin; ++i) {
        const int first = i * W, li = min(W, N - first), next = first + li;
        SymRows from = rows3(i);
        if (last > kSymFirst) {
          sym_transposes<R>(s.tri, tri_base, buf(q), i, li, warp_id, n_warps);
        } else {
          finish(i - 1, done);
        }
        for (int L = kSymFirst; L < last; ++L) {
          uint4* const dst = buf(q++);
          uint4* const level = s.tri + (size_t)(L - kSymFirst) * s.tri_cells;
          uint4* const hi = level + tri_base(i);
          unsigned cd = 0, co = 0;
          sym_sweep<R, false>(s, from, dst, hi, a.adj, N, d, a.vec4, first, next, li, (early >> L) & 1u,
                              warp_id, n_warps, cd, co, full);
          sym_add((unsigned long long)cd + 2ull * co, s_acc + L);
          grid_arrive(ctrl);
          if (L == kSymFirst) finish(i - 1, done);
          if (L + 1 < last) sym_transposes<R>(level + s.tri_cells, tri_base, buf(q), i, li, warp_id, n_warps);
          bar_target += grid;
          if (!grid_wait(ctrl, bar_target, a.timeout_ns, &s_flag)) return;
          from = {dst, hi, next};
        }
        done = from;
        sweeps += last - kSymFirst + 1;
      }
      finish(nwin - 1, done);
      __syncthreads();
      if (threadIdx.x < kSymLevels + 8 && s_acc[threadIdx.x])
        atomicAdd(s.cnt + kSymCntW + threadIdx.x, s_acc[threadIdx.x]);
      if (!barrier()) return;
      fallback = __ldcg(s.list_n) > kSymList;
    }
  }
  // ---- the listed pairs, level by level --------------------------------------------
  const unsigned n = stalled || fallback ? 0u : __ldcg(s.list_n);
  unsigned long long late = 0;                 // sum of the unreached pairs at the levels from k* on
  int diam = last;
  if (n) {
    int passes = 0;
    const int r = sym_resolve(s, s.list_n + 1, a.adj, d, n, kSymPasses, blockIdx.x * kThreads + threadIdx.x,
                              grid * kThreads, barrier, late, passes);
    if (r == kSymFailed) return;
    diam = last + passes;
    stalled = r == kSymStalled;
    fallback = r == kSymTooLong;
  }
  if (fallback) {   // the persistent kernel launched behind this one runs instead
    if (blockIdx.x == 0 && threadIdx.x == 0) ctrl->fallback = 1;
    return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const unsigned long long nn = (unsigned long long)N * N;
    // U_1, U_2 from the ball, U_3 .. U_{k*-1} from the weighted counters, the rest from the list
    unsigned long long sum = late;
    for (int L = last - 1; L >= 1; --L) {
      const unsigned long long u = nn - __ldcg(L <= 2 ? s.cnt + L - 1 : s.cnt + kSymCntW + L);
      sum += u;
      if (u == 0) diam = L;
    }
    ctrl->diam = stalled ? N + 1 : diam;
    ctrl->disconnected = stalled ? 1 : 0;
    ctrl->sum = (long long)sum;
    ctrl->levels = (long long)nwin * diam;
    ctrl->dense_levels = sweeps;
    ctrl->windows = nwin;
    __threadfence();
    ctrl->done = 1;
  }
}

}  // namespace ggb
