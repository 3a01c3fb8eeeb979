// Table enumeration with two columns per 32-bit word (16-bit halves), for
// L_1, LM (d = 1), L_2 and L_3.
//
// The enumeration is the table kernel's (table_kernel.cuh: N = h * B + j, a
// shared-memory table of the low rows' partial sums, one row moved per step
// of a walk over the high indices).  What differs is how an entry is valued.
// With |x - y| = 2 max(x, y) - x - y,
//     sum_c |H_c - T_c| = 2 sum_c max(H_c, T_c) - sum_c H_c - sum_c T_c,
// and the last two sums belong to the high index and to the entry alone.  So
// a labeling costs, per two columns and message vector, one pair maximum
// (max.u16x2, ALU pipe) and one multiply-add by a run-time one that adds the
// pair to a packed accumulator (FMA pipe), where the 32-bit form costs two
// absolute-difference-accumulates on the ALU pipe.  Both pipes take a warp
// instruction every two clocks, so the bound is the issue slot: one per
// column instead of two ALU clocks per column.  (A plain add goes to the ALU
// pipe instead and measures 1.25x slower.)
//
// Fields.  Column c is stored with a bias beta_c that makes every value H_c
// or T_c can take non-negative; a word is field_hi * 65536 + field_lo, and
// adding or subtracting rows is ordinary 32-bit arithmetic on such words
// (a row's word is a_hi * 65536 + a_lo, borrow included), exact as long as
// both end states are in range.  The packed accumulator starts from the
// entry's seed word, which takes out the smallest value each half can have
// and half of the entry's own column sum; the host checks that both halves
// then end below 65536.  One dot product (dp2a) adds the halves:
//     Y = sum of fields + seed,   value = 2 Y - SH(h) + value_bias,
// SH(h) the column sum of the register vectors, kept in one extra word that
// moves with the rows.
//
// K high indices per thread share each table read.  S > 1: S adjacent lanes
// share a high index, lane g holding slice g of the columns (as in
// split_kernel.cuh, with its ring reduce-scatter over tiles of S entries).
#pragma once
#include "table_kernel.cuh"

namespace ld {

struct HalfArgs {
  TableArgs t;      // image, geometry, label symmetry, reduction (vectors: S slices of WT words)
  int Bp;           // table entries: B rounded up to a multiple of S
  int span;         // words of one slice's shared-memory region (bank padding included)
  int value_bias;   // added to 2 Y - SH
  uint32_t one;     // 1, opaque to the compiler: keeps the accumulation on the FMA pipe
};

// One slice: W words of two columns.  A vector (row, totals, initial H, bias)
// has WT words: the W data words, the slice's column sum (no bias), and, in
// the bias vector, the entries' seed base.
template <int D, int W>
struct Half {
  static constexpr int WV = W + 1;                  // register words of one vector (with its sum)
  static constexpr int WT = (W + 2 + 3) & ~3;       // stored words of one vector
  static constexpr int NR = D == 3 ? 3 : 1;         // register vectors: H, or H1, H2, H1 + H2
  static constexpr int NW = (1 + D * W + 3) & ~3;   // words of an entry: seed, then D x W
  static constexpr int SUM = (D == 3 ? 2 : 0) * WV + W;   // register word of the column sum
};

__host__ __device__ inline int half_row_words(int W) { return (W + 2 + 3) & ~3; }
__host__ __device__ inline int half_entry_words(int D, int W) { return (1 + D * W + 3) & ~3; }
// words of one slice region: R rows, totals, initial H, bias, then Bp entries
__host__ __device__ inline int half_region_words(int D, int W, int R, int Bp) {
  return (R + 3) * half_row_words(W) + Bp * half_entry_words(D, W);
}

// H[v] += row * m (m = 1, 0 or -1; rows are 16-byte aligned)
template <int D, int W>
__device__ __forceinline__ void half_add(uint32_t* H, const uint32_t* row, int v, uint32_t m) {
  const uint4* r = reinterpret_cast<const uint4*>(row);
#pragma unroll
  for (int q = 0; q < (W + 4) / 4; ++q) {
    const uint4 x = r[q];
    const uint32_t xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (4 * q + c <= W) H[v * (W + 1) + 4 * q + c] += xs[c] * m;
  }
}

// high row `row` moves from label a to label b
template <int D, int W>
__device__ __forceinline__ void half_move(uint32_t* H, const uint32_t* row, int a, int b) {
  if constexpr (D == 1) {
    half_add<D, W>(H, row, 0, b ? 2u : 0u - 2u);
  } else if constexpr (D == 2) {
    half_add<D, W>(H, row, 0, b ? 1u : 0u - 1u);
  } else {
    half_add<D, W>(H, row, 0, (uint32_t)(b == 1) - (uint32_t)(a == 1));
    half_add<D, W>(H, row, 1, (uint32_t)(b == 2) - (uint32_t)(a == 2));
    half_add<D, W>(H, row, 2, (uint32_t)(b != 0) - (uint32_t)(a != 0));
  }
}

// Register vectors of high index h: every vector starts from sH0 (the bias,
// for d = 1 with the fixed row).  Without branches on the label: the groups of
// a warp hold different high indices (with branches and word-wise loads a
// seed of 18 rows of 8 x 16 words took 10,000 clocks).
template <int D, int W>
__device__ __forceinline__ void half_seed(uint32_t* H, const uint32_t* sA, const uint32_t* sH0, int k, int nh,
                                          unsigned long long h) {
  using P = Half<D, W>;
#pragma unroll
  for (int v = 0; v < P::NR; ++v)
#pragma unroll
    for (int w = 0; w <= W; ++w) H[v * P::WV + w] = sH0[w];
  const uint32_t* row = sA + k * P::WT;
  if constexpr (D <= 2) {
    unsigned long long g = h ^ (h >> 1);
    for (int t = 0; t < nh; ++t, g >>= 1, row += P::WT) {
      const uint32_t lab = (uint32_t)(g & 1ull);
      half_add<D, W>(H, row, 0, D == 1 ? 2u * lab - 1u : lab);
    }
  } else {
    unsigned long long x = h;
    for (int t = 0; t < nh; ++t, row += P::WT) {
      const unsigned long long q = x / 3ull;
      const unsigned n = (unsigned)(x - 3ull * q), lab = (q & 1ull) ? 2u - n : n;
      x = q;
      half_add<D, W>(H, row, 0, lab == 1u);
      half_add<D, W>(H, row, 1, lab == 2u);
      half_add<D, W>(H, row, 2, lab != 0u);
    }
  }
}

// entry j (the Gray word of j over the k low rows) of one slice
template <int D, int W>
__device__ __forceinline__ void half_build_entry(int j, int k, const uint32_t* sA, const uint32_t* sTot,
                                                 const uint32_t* sTb, uint32_t* e) {
  using P = Half<D, W>;
  uint32_t L1[W + 1], L2[W + 1];
#pragma unroll
  for (int w = 0; w <= W; ++w) { L1[w] = 0u; L2[w] = 0u; }
  if constexpr (D <= 2) {
    const unsigned g = (unsigned)j ^ ((unsigned)j >> 1);
    for (int i = 0; i < k; ++i) {
      const int lab = (g >> i) & 1u;
      const uint32_t* row = sA + i * P::WT;
#pragma unroll
      for (int w = 0; w <= W; ++w) L1[w] += lab ? row[w] : (D == 1 ? 0u - row[w] : 0u);
    }
  } else {
    unsigned q = (unsigned)j;
    for (int i = 0; i < k; ++i) {
      const unsigned r = q % 6u;
      const int lab = r < 3u ? (int)r : 5 - (int)r;
      q /= 3u;
      const uint32_t* row = sA + i * P::WT;
#pragma unroll
      for (int w = 0; w <= W; ++w) {
        L1[w] += lab == 1 ? row[w] : 0u;
        L2[w] += lab == 2 ? row[w] : 0u;
      }
    }
  }
  // the entry's column sum over its vectors, halved (its parity is the same
  // for every entry), goes into the seed
  const int st = D == 1 ? (int)(sTb[W] - L1[W]) : (int)(sTot[W] - 2u * (L1[W] + L2[W]));
  e[0] = sTb[W + 1] - (uint32_t)(st >> 1);
#pragma unroll
  for (int w = 0; w < W; ++w) {
    e[1 + w] = sTb[w] - L1[w];
    if constexpr (D == 2) e[1 + W + w] = sTot[w] - L1[w];
    if constexpr (D == 3) {
      e[1 + W + w] = sTb[w] - L2[w];
      e[1 + 2 * W + w] = sTot[w] - L1[w] - L2[w];
    }
  }
#pragma unroll
  for (int w = 1 + D * W; w < P::NW; ++w) e[w] = 0u;
}

// acc[i] += the words 4q .. 4q+3 of an entry against register vectors i
template <int D, int W, int K>
__device__ __forceinline__ void half_acc4(const uint32_t (*H)[Half<D, W>::NR * (W + 1)], const uint4& x, int q,
                                          uint32_t* acc, uint32_t one) {
  const uint32_t xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int t = 4 * q + c - 1;
    if (t < 0) {
#pragma unroll
      for (int i = 0; i < K; ++i) acc[i] = xs[c];
    } else if (t < D * W) {
      const int r = (D == 3 ? t / W : 0) * (W + 1) + t % W;
#pragma unroll
      for (int i = 0; i < K; ++i) acc[i] = __vmaxu2(H[i][r], xs[c]) * one + acc[i];
    }
  }
}

// Y of one entry for K register vector sets
template <int D, int W, int K>
__device__ __forceinline__ void half_entry(const uint32_t (*H)[Half<D, W>::NR * (W + 1)], const uint32_t* e, int* y,
                                           uint32_t one) {
  uint32_t acc[K];
  const uint4* t = reinterpret_cast<const uint4*>(e);
#pragma unroll
  for (int q = 0; q < Half<D, W>::NW / 4; ++q) half_acc4<D, W, K>(H, t[q], q, acc, one);
#pragma unroll
  for (int i = 0; i < K; ++i) y[i] = (int)__dp2a_lo(acc[i], 0x0101u, 0u);
}

// full Y of entry j0 + g of a tile of S entries, for K register vector sets:
// partial sums of the slice, then the ring reduce-scatter within the group
template <int D, int W, int S, int K>
__device__ __forceinline__ void half_tile(const uint32_t (*H)[Half<D, W>::NR * (W + 1)], const uint32_t* sT, int j0,
                                          int g, unsigned gmask, int src, int* y, uint32_t one) {
  int p[S][K];
#pragma unroll
  for (int r = 0; r < S; ++r)
    half_entry<D, W, K>(H, sT + (j0 + ((g + r) & (S - 1))) * Half<D, W>::NW, p[r], one);
#pragma unroll
  for (int t = 1; t < S; ++t)
#pragma unroll
    for (int i = 0; i < K; ++i) p[S - 1 - t][i] += __shfl_sync(gmask, p[S - t][i], src, S);
#pragma unroll
  for (int i = 0; i < K; ++i) y[i] = p[0][i];
}

// max of Y over the table for K register vector sets (a lane's share of it
// when S > 1)
template <int D, int W, int S, int K>
__device__ __forceinline__ void half_scan(const uint32_t (*H)[Half<D, W>::NR * (W + 1)], const uint32_t* sT, int Bp,
                                          int g, unsigned gmask, int src, int* m, uint32_t one) {
#pragma unroll
  for (int i = 0; i < K; ++i) m[i] = INT_MIN;
  if constexpr (S > 1) {
    for (int j0 = 0; j0 < Bp; j0 += S) {
      int y[K];
      half_tile<D, W, S, K>(H, sT, j0, g, gmask, src, y, one);
#pragma unroll
      for (int i = 0; i < K; ++i) m[i] = max(m[i], y[i]);
    }
  } else {
    // two entries per step: independent accumulator chains
    int j = 0;
    for (; j + 2 <= Bp; j += 2) {
      int y[K], z[K];
      half_entry<D, W, K>(H, sT + j * Half<D, W>::NW, y, one);
      half_entry<D, W, K>(H, sT + (j + 1) * Half<D, W>::NW, z, one);
#pragma unroll
      for (int i = 0; i < K; ++i) m[i] = max(m[i], max(y[i], z[i]));
    }
    if (j < Bp) {
      int y[K];
      half_entry<D, W, K>(H, sT + j * Half<D, W>::NW, y, one);
#pragma unroll
      for (int i = 0; i < K; ++i) m[i] = max(m[i], y[i]);
    }
  }
}

// column sum of the register vectors against all table vectors (this slice's)
template <int D, int W>
__device__ __forceinline__ int half_sh(const uint32_t* H) {
  return D == 1 ? (int)H[Half<D, W>::SUM] : 2 * (int)H[Half<D, W>::SUM];
}

// Resident blocks of 128 threads: K x NR register vectors, about 56 other
// registers, the ring's partial sums and, for d >= 2, the longer entry loop's;
// 8 at most.  (With 44 instead of 56 the main loop spills.)
__host__ __device__ constexpr int half_min_blocks(int D, int W, int S, int K) {
  const int need = K * (D == 3 ? 3 : 1) * (W + 1) + 56 + (S > 1 ? S * K : 0) + (D >= 2 ? 8 * K : 0);
  return 512 / need > 8 ? 8 : (512 / need < 1 ? 1 : 512 / need);
}

template <int D, int W, int S, int K>
__global__ void __launch_bounds__(kTableThreads, half_min_blocks(D, W, S, K)) half_kernel(const HalfArgs ha) {
  using P = Half<D, W>;
  static_assert(D >= 1 && D <= 3 && (S == 1 || S == 2 || S == 4 || S == 8) && (K == 1 || K == 2), "");
  const TableArgs& args = ha.t;
  extern __shared__ __align__(16) uint32_t smem[];
  block_start();
  const int R = args.R, k = args.k, B = args.B, Bp = ha.Bp, span = ha.span;
  const uint32_t one = ha.one;
  const int nh = R - 1 - k;
  const int g = S > 1 ? (threadIdx.x & (S - 1)) : 0;
  const unsigned gmask = S > 1 ? ((1u << S) - 1u) << ((threadIdx.x & 31) & ~(S - 1)) : 0u;
  const int src = (g + S - 1) & (S - 1);
  uint32_t* sA = smem + g * span;
  uint32_t* sH0 = sA + (R + 1) * P::WT;
  uint32_t* sT = sA + (R + 3) * P::WT;

  // stage: rows, totals, initial H and bias, slice r of each to region r
  for (int t = threadIdx.x; t < (R + 3) * S * P::WT; t += blockDim.x) {
    const int i = t / (S * P::WT), u = t - i * (S * P::WT), r = u / P::WT, w = u - r * P::WT;
    const uint32_t* v = i < R ? args.A + (size_t)i * S * P::WT : i == R ? args.tot : i == R + 1 ? args.hinit : args.tbias;
    smem[r * span + i * P::WT + w] = v[u];
  }
  __syncthreads();
  // the table, one (entry, slice) per thread; entries B .. Bp-1 repeat entry 0
  for (int t = threadIdx.x; t < Bp * S; t += blockDim.x) {
    const int j = t / S, r = t - j * S;
    uint32_t* rb = smem + r * span;
    half_build_entry<D, W>(j < B ? j : 0, k, rb, rb + R * P::WT, rb + (R + 2) * P::WT,
                           rb + (R + 3) * P::WT + j * P::NW);
  }
  __syncthreads();

  const unsigned long long WL = args.walk_len;
  const bool by_rank = D >= 3 && args.sym_digits > 0;
  const unsigned long long it_begin = by_rank ? args.rank_begin : args.walk_begin;
  const unsigned long long it_end = by_rank ? args.rank_end : args.walk_end;
  uint32_t H[K][P::NR * P::WV];
  int best = INT_MIN;
  unsigned long long best_h = 0ull;
  // K walks in lockstep (a walk past the end repeats the first one)
  auto run = [&](unsigned long long first, unsigned long long step) {
    unsigned long long wk[K];
#pragma unroll
    for (int i = 0; i < K; ++i) {
      wk[i] = first + (unsigned long long)i * step;
      if (wk[i] >= it_end) wk[i] = first;
      if constexpr (D >= 3) {
        if (by_rank) wk[i] = walk_of_rank<D>(wk[i], args.sym_digits, args.sym_table);
      }
      half_seed<D, W>(H[i], sA, sH0, k, nh, wk[i] * WL);
    }
    for (unsigned long long u = 0; u < WL; ++u) {
      if (u) {
#pragma unroll
        for (int i = 0; i < K; ++i) {
          int row, a, b;
          high_step<D>(wk[i], wk[i] * WL + u, u, row, a, b);
          half_move<D, W>(H[i], sA + (k + row) * P::WT, a, b);
        }
      }
      int m[K];
      half_scan<D, W, S, K>(H, sT, Bp, g, gmask, src, m, one);
#pragma unroll
      for (int i = 0; i < K; ++i) {
        int sh = half_sh<D, W>(H[i]);
#pragma unroll
        for (int off = 1; off < S; off <<= 1) sh += __shfl_xor_sync(gmask, sh, off, S);
        const int v = 2 * m[i] - sh;
        const unsigned long long h = wk[i] * WL + u;
        if (v > best || (v == best && h < best_h)) { best = v; best_h = h; }
      }
    }
  };
  // walks: fetched by the warp, 32 / S groups x K at a time, from the launch's
  // counter, or a fixed share per group (table_kernel.cuh); all lanes of a
  // group take the same walks
  constexpr unsigned GW = 32u / S;
  const unsigned gl = (threadIdx.x & 31u) / S;
  if (args.red.work) {
    for (;;) {
      unsigned long long base = 0ull;
      if ((threadIdx.x & 31u) == 0u) base = atomicAdd(args.red.work, (unsigned long long)(GW * K));
      base = it_begin + __shfl_sync(0xffffffffu, base, 0);
      if (base >= it_end) break;
      if (base + gl < it_end) run(base + gl, GW);
      __syncwarp();
    }
  } else {
    const unsigned long long G = (unsigned long long)gridDim.x * blockDim.x / S;
    const unsigned long long gid = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) / S;
    for (unsigned long long it = it_begin + gid; it < it_end; it += K * G) run(it, G);
  }

  // the group's maximum and the smallest high index attaining it
#pragma unroll
  for (int off = 1; off < S; off <<= 1) {
    const int ob = __shfl_xor_sync(gmask, best, off, S);
    const unsigned long long oh = __shfl_xor_sync(gmask, best_h, off, S);
    if (ob > best || (ob == best && oh < best_h)) { best = ob; best_h = oh; }
  }
  // the first index attaining the block's best: the smallest Gray position
  // among the entries of its block at the maximum, a tile per group (the low
  // word is read backwards for odd h)
  long long bv = LLONG_MIN;
  unsigned long long bn = ULLONG_MAX;
  block_top(best, best_h);
  if (best != INT_MIN) {
    half_seed<D, W>(H[0], sA, sH0, k, nh, best_h);
    int sh = half_sh<D, W>(H[0]);
#pragma unroll
    for (int off = 1; off < S; off <<= 1) sh += __shfl_xor_sync(gmask, sh, off, S);
    const bool rev = (best_h & 1ull) != 0ull;
    int jbest = INT_MAX;
    for (int j0 = (int)threadIdx.x / S * S; j0 < Bp; j0 += blockDim.x) {
      int y[1];
      half_tile<D, W, S, 1>(H, sT, j0, g, gmask, src, y, one);
      const int je = j0 + g;
      if (je < B && 2 * y[0] - sh == best) jbest = min(jbest, rev ? B - 1 - je : je);
    }
    jbest = block_min(jbest);
    if (jbest != INT_MAX) bn = best_h * (unsigned long long)B + (unsigned long long)jbest;
    bv = (long long)best + ha.value_bias - args.value_offset;
  }
  grid_reduce(bv, bn, args.red);
}

}  // namespace ld
