// Batched persistent kernel over matrices in the two-columns-per-word form
// (half_kernel.cuh): the int32 batch classes of 8, 16, .., 64 columns, D = 1,
// 2, 3, when every value fits the 16-bit fields.  The queue, the chunks and
// the slots are those of batch_kernel.cuh.  For d <= 2 each thread walks two
// of the chunk's walks in lockstep, so that an entry is read once for both.
#include <utility>

#include "batch_kernel.cuh"
#include "half_kernel.cuh"
#include "registry.h"

namespace ld {
namespace {

template <int D, int W>
__global__ void __launch_bounds__(kBatchMaxThreads, half_min_blocks(D, W, 1, D <= 2 ? 2 : 1))
    batch_half_kernel(const BatchArgs args, uint32_t one) {
  using P = Half<D, W>;
  constexpr int K = D <= 2 ? 2 : 1;
  extern __shared__ __align__(16) uint32_t smem[];
  __shared__ int s_chunk;
  int loaded = -1;
  uint32_t H[K][P::NR * P::WV];
  for (;;) {
    if (threadIdx.x == 0) s_chunk = (int)atomicAdd(args.head, 1u);
    __syncthreads();
    const int c = s_chunk;
    __syncthreads();
    if (c >= args.nchunks) break;
    const BatchChunk ch = args.chunks[c];
    const BatchProblem pr = args.problems[ch.problem];
    const int R = pr.R, k = pr.k, B = pr.B, nh = R - 1 - k;
    uint32_t* sA = smem;
    uint32_t* sH0 = sA + (R + 1) * P::WT;
    uint32_t* sT = sA + (R + 3) * P::WT;
    if (ch.problem != loaded) {
      for (int t = threadIdx.x; t < R * P::WT; t += blockDim.x) sA[t] = pr.A[t];
      for (int t = threadIdx.x; t < P::WT; t += blockDim.x) {
        sA[R * P::WT + t] = pr.tot[t];
        sH0[t] = pr.hinit[t];
        sH0[P::WT + t] = pr.tbias[t];
      }
      __syncthreads();
      for (int j = threadIdx.x; j < B; j += blockDim.x)
        half_build_entry<D, W>(j, k, sA, sA + R * P::WT, sH0 + P::WT, sT + j * P::NW);
      __syncthreads();
      loaded = ch.problem;
    }
    const unsigned long long WL = pr.walk_len;
    int best = INT_MIN;
    unsigned long long best_h = 0ull;
    for (unsigned long long w0 = ch.walk_begin + threadIdx.x; w0 < ch.walk_end; w0 += K * blockDim.x) {
      if constexpr (D == 3) {   // walks holding no class minimum (table_kernel.cuh)
        if (pr.sym_digits > 0 && !walk_holds_class_min<3>(w0, pr.sym_digits, pr.sym_pw)) continue;
      }
      unsigned long long wk[K];
#pragma unroll
      for (int i = 0; i < K; ++i) {
        wk[i] = w0 + (unsigned long long)i * blockDim.x;
        if (wk[i] >= ch.walk_end) wk[i] = w0;     // a lone walk runs twice
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
        half_scan<D, W, 1, K>(H, sT, B, 0, 0u, 0, m, one);
#pragma unroll
        for (int i = 0; i < K; ++i) {
          const int v = 2 * m[i] - half_sh<D, W>(H[i]);
          const unsigned long long h = wk[i] * WL + u;
          if (v > best || (v == best && h < best_h)) { best = v; best_h = h; }
        }
      }
    }
    long long bv = LLONG_MIN;
    unsigned long long bn = ULLONG_MAX;
    block_top(best, best_h);
    if (best != INT_MIN) {
      half_seed<D, W>(H[0], sA, sH0, k, nh, best_h);
      const int sh = half_sh<D, W>(H[0]);
      const bool rev = (best_h & 1ull) != 0ull;
      int jbest = INT_MAX;
      for (int je = threadIdx.x; je < B; je += blockDim.x) {
        int y[1];
        half_entry<D, W, 1>(H, sT + je * P::NW, y, one);
        if (2 * y[0] - sh == best) jbest = min(jbest, rev ? B - 1 - je : je);
      }
      jbest = block_min(jbest);
      if (jbest != INT_MAX) bn = best_h * (unsigned long long)B + (unsigned long long)jbest;
      bv = (long long)best - pr.value_offset;   // the offset holds the value bias
    }
    if (threadIdx.x == 0) { args.chunk_results[c].value = bv; args.chunk_results[c].index = bn; }
  }
}

template <int D, int... I>
void fill(const void* (&t)[4][9], std::integer_sequence<int, I...>) {
  ((t[D][I + 1] = (const void*)&batch_half_kernel<D, 4 * (I + 1)>), ...);
}

}  // namespace

const void* batch_half_kernel_ptr(int D, int W) {
  static const void* tab[4][9] = {};
  static bool init = [] {
    fill<1>(tab, std::make_integer_sequence<int, 8>{});
    fill<2>(tab, std::make_integer_sequence<int, 8>{});
    fill<3>(tab, std::make_integer_sequence<int, 8>{});
    return true;
  }();
  (void)init;
  if (D < 1 || D > 3 || W < 4 || W > 32 || W % 4) return nullptr;
  return tab[D][W / 4];
}

}  // namespace ld
