// Pruned exact search: the table kernel's enumeration with integer upper
// bounds that skip whole blocks of labelings which cannot beat an incumbent.
//
// Split the free rows into top rows (the Gray digits of a walk index), walk
// rows (the fw digits a thread walks) and low rows (the tabulated k digits).
// For any labeling, per message m and column l the column sum is
// P_ml + Q_ml, P over the fixed and top rows, Q over the rest, so
//     value <= sum_ml |P_ml| + max over the rest's labelings of sum_ml |Q_ml|
// and the second term is exactly the L_d norm (for LM: the marginal norm)
// of the rest rows alone, computed beforehand by the plain solver.  The
// search goes from short prefixes to whole high indices:
//   1. prefix_bound_kernel: for every walk, the bound with P over the top rows
//      and the rest = walk + low rows; walks whose bound is below the
//      incumbent are dropped, the others are appended to a list;
//   2. prefix_bound_kernel again: every listed prefix is extended by some walk
//      rows and bounded with the norm of the rows that remain, while the
//      listed ones hold many high indices, and at last by all of them, when
//      the rest is the low rows.  (One step from the walks to their high
//      indices took 2214 us for a 44 x 44 matrix whose 9037 listed walks hold
//      148 M of them; one more level leaves 5.6 M.)
//   3. prune_eval_kernel: the B labelings of each surviving high index, each
//      table shared by a few threads.  Survivors lie close together: evaluated
//      where they are found, 1075 of them kept one warp busy for 50 us.
// Only bounds strictly below the incumbent prune, so every labeling that
// attains the maximum is evaluated and the smallest Gray index among them is
// the one reported: the result equals the plain enumeration's.
//
// Bounds are formed in the kernel's representation: for d = 1 the register
// vector is the signed sum (for LM with column 0 shifted by K_H >= 0, so its
// absolute value is the shifted signed sum); for d = 2 the messages are H
// and T - H, for d = 3 H1, H2 and T - H1 - H2, where T is the column total of
// the rows in P (uploaded per level).
#pragma once
#include "table_kernel.cuh"

namespace ld {

struct PruneArgs {
  TableArgs t;                    // the table kernel's operands; fw = rows below a prefix, walk_begin ..
                                  // walk_end = the extensions to bound
  const uint32_t* ttop;           // WT words: column totals of the fixed + prefix rows (d >= 2)
  long long threshold;            // incumbent, in the kernel's value representation
  long long m_rest;               // norm of the rows below a prefix (representation-adjusted)
  const unsigned long long* src;  // the listed prefixes to extend (null: extension = prefix)
  unsigned long long expand;      // extensions of each, a power of the base
  unsigned long long run;         // consecutive extensions per thread, a power of the base up to it
  unsigned long long* list;       // surviving prefixes (evaluation: high indices)
  unsigned long long* list_count; // their number; then a bound's first block's start and its last one's
                                  // end (ns; all 0 before a bound)
  Slot* best;                     // evaluation: the best over its launches; then the high indices seen,
                                  // and the ns from the bounds' starts to the evaluations' ends
};

constexpr int kPruneThreads = 128;

// sum over the register vectors' lanes of |x| for d = 1, or of the message
// vectors' |.| for d = 2, 3 (T = column totals of the rows the vectors cover)
template <int D, int WB, int WA>
__device__ __forceinline__ long long prefix_abs(const uint32_t* H, const uint32_t* T) {
  using S = Shape<D, WB, WA>;
  static_assert(D != 3 || S::NR == 3, "pruned d = 3 shapes keep H1 + H2 in registers");
  uint32_t acc[2] = {0u, 0u};   // two chains: the launches have few warps
  if (D == 1) {
#pragma unroll
    for (int w = 0; w < S::WV; ++w) acc[w & 1] = wsad<WB>(w, H[w], 0u, acc[w & 1]);
  } else if (D == 2) {
#pragma unroll
    for (int w = 0; w < S::WV; ++w) {
      acc[0] = wsad<WB>(w, H[w], 0u, acc[0]);
      acc[1] = wsad<WB>(w, H[w], T[w], acc[1]);
    }
  } else {
#pragma unroll
    for (int w = 0; w < S::WV; ++w) {
      acc[0] = wsad<WB>(w, H[w], 0u, acc[0]);
      acc[1] = wsad<WB>(w, H[S::WV + w], 0u, acc[1]);
      acc[w & 1] = wsad<WB>(w, H[2 * S::WV + w], T[w], acc[w & 1]);
    }
  }
  return (long long)(acc[0] + acc[1]);
}

// H[vec] += row * m, m = -2 .. 2: without a branch on the label, which differs
// between the lanes of a warp, and with 16-byte loads (one 4-byte load per word
// and a branch per label made a step of 44 words 590 clocks per warp)
template <int D, int WB, int WA>
__device__ __forceinline__ void add_times(uint32_t* H, const uint32_t* row, int vec, int m) {
  using S = Shape<D, WB, WA>;
  const uint4* r = reinterpret_cast<const uint4*>(row);
#pragma unroll
  for (int q = 0; q < S::WT / 4; ++q) {
    const uint4 x = r[q];
    const uint32_t xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int w = 4 * q + c;
      if (w >= S::WV) continue;
      uint32_t& h = H[vec * S::WV + w];
      if (w < WB) {
        h += xs[c] * (uint32_t)m;
      } else {
        uint32_t y = m == 0 ? 0u : m == 2 || m == -2 ? wadd<WB>(w, xs[c], xs[c]) : xs[c];
        if (m < 0) y = wsub<WB>(w, 0u, y);
        h = wadd<WB>(w, h, y);
      }
    }
  }
}

// a row moves from label a to label b (a = -1: it gets its first label)
template <int D, int WB, int WA>
__device__ __forceinline__ void relabel(uint32_t* H, const uint32_t* row, int a, int b) {
  if constexpr (D == 1) {
    add_times<D, WB, WA>(H, row, 0, a < 0 ? (b ? 1 : -1) : (b ? 2 : -2));
  } else if constexpr (D == 2) {
    add_times<D, WB, WA>(H, row, 0, (b == 1) - (a == 1));
  } else {
    add_times<D, WB, WA>(H, row, 0, (b == 1) - (a == 1));
    add_times<D, WB, WA>(H, row, 1, (b == 2) - (a == 2));
    add_times<D, WB, WA>(H, row, 2, (b > 0) - (a > 0));
  }
}

// H over the fixed row and the top rows only (digits fw.. of the high index)
template <int D, int WB, int WA>
__device__ __forceinline__ void seed_top(uint32_t* H, const uint32_t* sA, const uint32_t* sH0,
                                         int k, int fw, int nh, unsigned long long h) {
  using S = Shape<D, WB, WA>;
#pragma unroll
  for (int w = 0; w < S::WV; ++w) H[w] = sH0[w];
#pragma unroll
  for (int v = 1; v < S::NR; ++v)
#pragma unroll
    for (int w = 0; w < S::WV; ++w) H[v * S::WV + w] = 0u;
  if constexpr (D <= 2) {
    const unsigned long long g = h ^ (h >> 1);
    for (int t = fw; t < nh; ++t) relabel<D, WB, WA>(H, sA + (k + t) * S::WT, -1, (int)((g >> t) & 1ull));
  } else {
    unsigned long long q = h;
    for (int t = 0; t < fw; ++t) q /= 3ull;
    for (int t = fw; t < nh; ++t) {
      const int r = (int)(q % 6ull);
      q /= 3ull;
      relabel<D, WB, WA>(H, sA + (k + t) * S::WT, -1, r < 3 ? r : 5 - r);
    }
  }
}

// stage rows, vectors and (for the scan) the table into shared memory
template <int D, int WB, int WA>
__device__ __forceinline__ void stage(const PruneArgs& args, uint32_t* smem, bool with_table) {
  using S = Shape<D, WB, WA>;
  constexpr int WT = S::WT;
  const TableArgs& ta = args.t;
  const int R = ta.R;
  uint32_t* sA = smem;
  uint32_t* sTot = sA + R * WT;
  uint32_t* sH0 = sTot + WT;
  uint32_t* sTb = sH0 + WT;
  uint32_t* sTtop = sTb + WT;
  for (int t = threadIdx.x; t < R * WT; t += blockDim.x) sA[t] = ta.A[t];
  for (int t = threadIdx.x; t < WT; t += blockDim.x) {
    sTot[t] = ta.tot[t];
    sH0[t] = ta.hinit[t];
    sTb[t] = ta.tbias ? ta.tbias[t] : 0u;
    sTtop[t] = args.ttop[t];
  }
  __syncthreads();
  if (!with_table) return;
  uint32_t* sT = smem + (((R * WT + 4 * WT) + 3) & ~3);
  const int k = ta.k, B = ta.B;
  for (int j = threadIdx.x; j < B; j += blockDim.x) {
    uint32_t L1[S::WV], L2[S::WV];
#pragma unroll
    for (int w = 0; w < S::WV; ++w) { L1[w] = D == 1 ? sTb[w] : 0u; L2[w] = 0u; }
    if (D <= 2) {
      const unsigned g = (unsigned)j ^ ((unsigned)j >> 1);
      for (int i = 0; i < k; ++i) {
        const int lab = (g >> i) & 1u;
        const uint32_t* row = sA + i * WT;
        if (D == 1) {
#pragma unroll
          for (int w = 0; w < S::WV; ++w) L1[w] = lab ? wsub<WB>(w, L1[w], row[w]) : wadd<WB>(w, L1[w], row[w]);
        } else if (lab) {
#pragma unroll
          for (int w = 0; w < S::WV; ++w) L1[w] = wadd<WB>(w, L1[w], row[w]);
        }
      }
    } else {
      unsigned q = (unsigned)j;
      for (int i = 0; i < k; ++i) {
        const unsigned r = q % 6u;
        const int lab = r < 3u ? (int)r : 5 - (int)r;
        q /= 3u;
        const uint32_t* row = sA + i * WT;
        if (lab == 1) {
#pragma unroll
          for (int w = 0; w < S::WV; ++w) L1[w] = wadd<WB>(w, L1[w], row[w]);
        } else if (lab == 2) {
#pragma unroll
          for (int w = 0; w < S::WV; ++w) L2[w] = wadd<WB>(w, L2[w], row[w]);
        }
      }
    }
    uint32_t* e = sT + j * S::NW;
#pragma unroll
    for (int w = 0; w < WT; ++w) {
      if (w < S::WV) {
        if (D == 1) {
          e[w] = L1[w];
        } else if (D == 2) {
          e[w] = wsub<WB>(w, 0u, L1[w]);
          e[WT + w] = wsub<WB>(w, sTot[w], L1[w]);
        } else {
          e[w] = wsub<WB>(w, 0u, L1[w]);
          e[WT + w] = wsub<WB>(w, 0u, L2[w]);
          e[2 * WT + w] = wsub<WB>(w, wsub<WB>(w, sTot[w], L1[w]), L2[w]);
        }
      } else {
#pragma unroll
        for (int v = 0; v < D; ++v) e[v * WT + w] = 0u;
      }
    }
  }
  __syncthreads();
}

__host__ __device__ inline int prune_smem_words(int D, int W, int R, int B, bool with_table) {
  int head = R * W + 4 * W;
  head = (head + 3) & ~3;
  return head + (with_table ? B * D * W : 0);
}

// Bound prefixes; list those that survive.  A thread takes runs of consecutive
// prefixes and visits each run in order: the labels of a prefix's rows are its
// reflected Gray code (binary for d <= 2, 3-ary for d = 3), so consecutive
// prefixes differ in one row, and the prefix vector is seeded once per run and
// then updated by one row move per prefix.  Runs are aligned powers of the
// base, so that the row that moves depends on the step alone and its words are
// read once for the warp.
template <int D, int WB, int WA>
__global__ void __launch_bounds__(kPruneThreads) prefix_bound_kernel(const PruneArgs args) {
  using S = Shape<D, WB, WA>;
  extern __shared__ __align__(16) uint32_t smem[];
  if (blockIdx.x == 0 && threadIdx.x == 0) args.list_count[1] = global_ns();
  stage<D, WB, WA>(args, smem, false);
  const TableArgs& ta = args.t;
  const int R = ta.R, k = ta.k, fw = ta.fw, nh = R - 1 - k;
  const uint32_t* sA = smem;
  const uint32_t* sH0 = smem + R * S::WT + S::WT;
  const uint32_t* sTtop = smem + R * S::WT + 3 * S::WT;
  const int lane = threadIdx.x & 31;
  const unsigned run = (unsigned)args.run;
  const unsigned long long E = args.expand;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x * run;
  uint32_t H[S::NR * S::WV];
  // d = 3 with label symmetry: a walk that holds no smallest index of a
  // class (walk_holds_class_min, table_kernel.cuh) is dropped as well
  const int P = D == 3 ? ta.sym_digits : 0;
  unsigned long long pw = 1ull;
  for (int t = 1; t < P; ++t) pw *= 3ull;
  // every lane of a warp runs the same number of iterations (ballots below)
  const unsigned long long base = ta.walk_begin + ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x - lane) * run;
  for (unsigned long long b0 = base; b0 < ta.walk_end; b0 += stride) {
    const unsigned long long v = b0 + (unsigned long long)lane * run;
    const bool on = v < ta.walk_end;
    unsigned long long w0 = on ? v : 0ull;
    if (args.src) {
      const unsigned long long slot = w0 / E;
      w0 = args.src[slot] * E + (w0 - slot * E);
    }
    seed_top<D, WB, WA>(H, sA, sH0, k, fw, nh, w0 * ta.walk_len);
    for (unsigned r = 0; r < run; ++r) {
      const unsigned long long wk = w0 + r;
      if (r) {
        int i;
        if constexpr (D <= 2) {
          i = __ffs((int)r) - 1;
          const int b = ((wk >> (i + 1)) & 1ull) == 0ull;
          relabel<D, WB, WA>(H, sA + (k + fw + i) * S::WT, b ^ 1, b);
        } else {
          // runs start at multiples of a power of 3, an odd number, so w0
          // adds its own parity to the digits above the changing one
          unsigned q = r;
          i = 0;
          while (q % 3u == 0u) { q /= 3u; ++i; }
          const int c = (int)(q % 3u);
          const int par = (int)(((unsigned)w0 ^ (q / 3u)) & 1u);
          const int b = par ? 2 - c : c, a = par ? 3 - c : c - 1;
          relabel<D, WB, WA>(H, sA + (k + fw + i) * S::WT, a, b);
        }
      }
      bool keep = on && prefix_abs<D, WB, WA>(H, sTtop) + args.m_rest >= args.threshold;
      if constexpr (D == 3) {
        if (P > 0 && keep) keep = walk_holds_class_min<3>(wk, P, pw);
      }
      const unsigned mask = __ballot_sync(0xffffffffu, keep);
      if (mask) {
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(args.list_count, (unsigned long long)__popc(mask));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (keep) args.list[at + __popc(mask & ((1u << lane) - 1u))] = wk;
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) atomicMax(args.list_count + 2, global_ns());
}

// Evaluate the listed high indices: a thread per high index and part of the
// table, as many parts (at most 32, at least four entries each) as there are
// threads for; the lanes of a warp share a part, so that an entry is read once
// for all of them.
template <int D, int WB, int WA>
__global__ void __launch_bounds__(kPruneThreads) prune_eval_kernel(const PruneArgs args) {
  using S = Shape<D, WB, WA>;
  constexpr int WT = S::WT, NW = S::NW;
  extern __shared__ __align__(16) uint32_t smem[];
  const TableArgs& ta = args.t;
  const unsigned long long n = *args.list_count;
  const unsigned long long warps = (unsigned long long)gridDim.x * (kPruneThreads / 32);
  const int B = ta.B, R = ta.R, k = ta.k, nh = R - 1 - k;
  unsigned P = 1u;
  while (P < 32u && 8 * (int)P <= B && ((n + 31) / 32) * (2 * P) <= warps) P *= 2u;
  long long bv = LLONG_MIN;
  unsigned long long bn = ULLONG_MAX;
  // a block without work stages nothing
  if (((unsigned long long)blockIdx.x * (kPruneThreads / 32)) / P * 32ull < n) {
    stage<D, WB, WA>(args, smem, true);
    const uint32_t* sA = smem;
    const uint32_t* sH0 = smem + R * WT + WT;
    const uint32_t* sT = smem + (((R * WT + 4 * WT) + 3) & ~3);
    const unsigned long long warp = (unsigned long long)blockIdx.x * (kPruneThreads / 32) + (threadIdx.x >> 5);
    const int part = (int)(warp % P), per = (B + (int)P - 1) / (int)P;
    const int j0 = part * per, j1 = j0 + per < B ? j0 + per : B;
    uint32_t H[S::NR * S::WV];
    int best = INT_MIN;
    unsigned long long best_h = 0ull, last_h = 0ull;
    if (warp < warps / P * P && j0 < j1) {
      for (unsigned long long i = warp / P * 32ull + (threadIdx.x & 31); i < n; i += warps / P * 32ull) {
        const unsigned long long h = args.list[i];
        seed_top<D, WB, WA>(H, sA, sH0, k, 0, nh, h);
        int m = INT_MIN;
        for (int j = j0; j < j1; ++j) m = max(m, entry_value<D, WB, WA>(H, sT + j * NW));
        if (m > best || (m == best && h < best_h)) { best = m; best_h = h; }
        last_h = h;
      }
    }
    if (best != INT_MIN) {   // the part's first position attaining it (read backwards for odd h)
      if (best_h != last_h) seed_top<D, WB, WA>(H, sA, sH0, k, 0, nh, best_h);
      const bool rev = (best_h & 1ull) != 0ull;
      int jbest = INT_MAX;
      for (int j = j0; j < j1; ++j)
        if (entry_value<D, WB, WA>(H, sT + j * NW) == best) jbest = min(jbest, rev ? B - 1 - j : j);
      bv = (long long)best - ta.value_offset;
      bn = best_h * (unsigned long long)B + (unsigned long long)jbest;
    }
  }
  if (grid_reduce(bv, bn, ta.red) && threadIdx.x == 0) {
    const Slot r = *ta.red.result;
    if (better(r.value, r.index, args.best->value, args.best->index)) *args.best = r;
    unsigned long long* seen = reinterpret_cast<unsigned long long*>(args.best + 1);
    seen[0] += n;
    seen[1] += global_ns() - args.list_count[1];
  }
}

}  // namespace ld
