// Single-row-move local search: polish starting labelings into an
// incumbent for the pruned search.
//
// One block per start.  It keeps the message column sums S_m (int64) and the
// labels in shared memory; in each round four lanes share a row and evaluate
// the gain of its moves (d = 1: flip the sign; d >= 2: move the row to another
// message), the block takes the largest gain (ties: smallest row, then
// smallest label) and applies it, until no move gains or the round limit is
// reached.  The last row keeps its fixed label (+1 / message 0), as in the
// enumeration.  Values are exact int64; a start's final value is the value of
// its final labeling.  The rounds are a serial chain, so their latency is the
// time: with a warp per start, a lane per row and rows that fell on four bank
// groups, 8 starts of 44 x 44 took 71 us, now 24.
#include <cuda_runtime.h>

#include <climits>
#include <cstdint>
#include <cstring>
#include <mutex>

#include "../abi/smem_limit.h"
#include "../host/ld_internal.h"
#include "../abi/device_guard.h"

namespace {

constexpr int kLsThreads = 256;   // at most: four lanes for each of up to 64 rows
constexpr int kLsMaxCols = 128;
constexpr int kLsMaxRows = 64;

struct LsArgs {
  const long long* A;     // R x C
  int R, C, d, marginal;
  const int* starts;      // n x (R-1) labels
  int n, max_rounds;
  long long* values;      // n
  int* labels;            // n x (R-1)
};

template <typename T>
__device__ __forceinline__ T ls_abs(T x) { return x < 0 ? -x : x; }

// Entries of a staged row: an odd multiple of 4, so that the four columns which
// each of several rows reads at once (four rows of 8 bytes, eight of 4) fall on
// distinct banks.
__host__ __device__ inline int ls_stride(int C) {
  const int p = (C + 3) & ~3;
  return p % 8 ? p : p + 4;
}

// T = int32 when four times the sum of all |entries| fits it (every column sum
// and gain then does), else int64.
template <typename T>
__global__ void __launch_bounds__(kLsThreads) local_search_kernel(const LsArgs a) {
  extern __shared__ long long smem[];
  T* sA = reinterpret_cast<T*>(smem);
  __shared__ T S[3][kLsMaxCols];
  __shared__ int lab[kLsMaxRows];
  __shared__ T sg[kLsThreads / 32];
  __shared__ int si[kLsThreads / 32], st[kLsThreads / 32];   // row; its labels, from * 4 + to
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int R = a.R, C = a.C, d = a.d, nm = d == 1 ? 1 : d, W = ls_stride(C);
  const int start = blockIdx.x;
  for (int t = threadIdx.x; t < R * C; t += blockDim.x) sA[t / C * W + t % C] = (T)a.A[t];
  for (int i = threadIdx.x; i < R; i += blockDim.x)
    lab[i] = i < R - 1 ? a.starts[(size_t)start * (R - 1) + i] : d == 1 ? 1 : 0;
  __syncthreads();
  for (int l = threadIdx.x; l < C; l += blockDim.x) {
    T s0 = 0, s1 = 0, s2 = 0;
    for (int i = 0; i < R; ++i) {
      const T x = sA[i * W + l];
      const int b = lab[i];
      if (d == 1) s0 += b ? x : -x;
      else { s0 += b == 0 ? x : 0; s1 += b == 1 ? x : 0; s2 += b == 2 ? x : 0; }
    }
    S[0][l] = s0; S[1][l] = s1; S[2][l] = s2;
  }
  __syncthreads();
  const int i = threadIdx.x >> 2, q = threadIdx.x & 3;
  const bool live = i < R - 1;
  const T* row = sA + (live ? i : 0) * W;
  int from = live ? lab[i] : 0;
  for (int round = 0; round < a.max_rounds; ++round) {
    T bg = 0;                   // best gain of this row (> 0 to count)
    int bi = INT_MAX, bt = 0;
    if (d == 1) {
      const T f = from ? -2 : 2;              // change of the column sum per unit of A
      T g = 0;
      if (live) {
#pragma unroll 4
        for (int l = q; l < C; l += 4) {
          const T s = S[0][l], ns = s + f * row[l];
          g += (a.marginal && l == 0) ? ns - s : ls_abs(ns) - ls_abs(s);
        }
      }
      g += __shfl_xor_sync(0xffffffffu, g, 1);
      g += __shfl_xor_sync(0xffffffffu, g, 2);
      if (g > 0) { bg = g; bi = i; bt = from * 4 + (from ^ 1); }
    } else {
      for (int t = 0; t < d; ++t) {
        T g = 0;
        if (live && t != from) {
#pragma unroll 4
          for (int l = q; l < C; l += 4) {
            const T x = row[l], sf = S[from][l], su = S[t][l];
            g += ls_abs(sf - x) + ls_abs(su + x) - ls_abs(sf) - ls_abs(su);
          }
        }
        g += __shfl_xor_sync(0xffffffffu, g, 1);
        g += __shfl_xor_sync(0xffffffffu, g, 2);
        if (g > bg) { bg = g; bi = i; bt = from * 4 + t; }
      }
    }
    // largest gain, then smallest row, then smallest label
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) {
      const T og = __shfl_xor_sync(0xffffffffu, bg, off);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
      const int ot = __shfl_xor_sync(0xffffffffu, bt, off);
      if (og > bg || (og == bg && oi < bi)) { bg = og; bi = oi; bt = ot; }
    }
    if (lane == 0) { sg[wid] = bg; si[wid] = bi; st[wid] = bt; }
    __syncthreads();
    bg = sg[0]; bi = si[0]; bt = st[0];
    for (int w = 1; w < nw; ++w)
      if (sg[w] > bg || (sg[w] == bg && si[w] < bi)) { bg = sg[w]; bi = si[w]; bt = st[w]; }
    if (bg <= 0) break;
    const int was = bt >> 2, to = bt & 3;
    if (i == bi) from = to;
    for (int l = threadIdx.x; l < C; l += blockDim.x) {
      const T x = sA[bi * W + l];
      if (d == 1) S[0][l] += to ? 2 * x : -2 * x;
      else { S[was][l] -= x; S[to][l] += x; }
    }
    __syncthreads();
  }
  if (live && q == 0) a.labels[(size_t)start * (R - 1) + i] = from;
  if (wid == 0) {
    long long v = 0;
    for (int l = lane; l < C; l += 32)
      for (int m = 0; m < nm; ++m) v += (d == 1 && a.marginal && l == 0) ? (long long)S[m][l] : ls_abs((long long)S[m][l]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (lane == 0) a.values[start] = v;
  }
}

#define LS_CUDA(call)                                                                \
  do {                                                                               \
    cudaError_t e_ = (call);                                                         \
    if (e_ != cudaSuccess) return ld_fail(LD_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
  } while (0)

// Per-device workspace kept between calls: one device arena, one pinned
// staging buffer (inputs out, results back in one copy each) and a stream.
struct LsWorkspace {
  char* dmem = nullptr;
  size_t dcap = 0;
  char* hmem = nullptr;
  size_t hcap = 0;
  cudaStream_t stream = nullptr;
};
std::mutex g_ls_mu[64];
LsWorkspace g_ls[64];

size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace

extern "C" ld_status ld_local_search(const int64_t* a, int32_t R, int32_t C, int32_t d, int32_t marginal,
                                     const int32_t* starts, int32_t n, int32_t max_rounds, int32_t device,
                                     int64_t* values, int32_t* labels) {
  ldsolve::ContextRestore ctx_restore;   // the caller's current context, back on return
  if (!a || !starts || !values || !labels || n < 1 || R < 2 || C < 1)
    return ld_fail(LD_ERR_ARG, "bad local-search arguments");
  if (d < 1 || d > 3 || C > kLsMaxCols || R > kLsMaxRows)
    return ld_fail(LD_ERR_LIMIT, "local search takes d <= 3, <= %d columns, <= %d rows", kLsMaxCols, kLsMaxRows);
  if (device < 0 || device >= 64) return ld_fail(LD_ERR_ARG, "device %d out of range", device);
  for (int64_t t = 0; t < (int64_t)n * (R - 1); ++t)
    if (starts[t] < 0 || starts[t] >= (d == 1 ? 2 : d)) return ld_fail(LD_ERR_ARG, "start label out of range");
  const size_t nl = (size_t)n * (R - 1);
  // inputs: matrix | starts; results: values | labels
  const size_t bA = up256(sizeof(long long) * (size_t)R * C), bS = up256(sizeof(int) * nl);
  const size_t bV = up256(sizeof(long long) * (size_t)n), bL = up256(sizeof(int) * nl);
  const size_t in_bytes = bA + bS, out_bytes = bV + bL, total = in_bytes + out_bytes;
  if (cudaSetDevice(device) != cudaSuccess) return ld_fail(LD_ERR_NODEV, "no device %d", device);
  std::lock_guard<std::mutex> lock(g_ls_mu[device]);
  LsWorkspace& w = g_ls[device];
  if (!w.stream) LS_CUDA(cudaStreamCreateWithFlags(&w.stream, cudaStreamNonBlocking));
  if (w.dcap < total) {
    if (w.dmem) { LS_CUDA(cudaStreamSynchronize(w.stream)); LS_CUDA(cudaFree(w.dmem)); w.dmem = nullptr; w.dcap = 0; }
    LS_CUDA(cudaMalloc(&w.dmem, total));
    w.dcap = total;
  }
  if (w.hcap < total) {
    if (w.hmem) { LS_CUDA(cudaStreamSynchronize(w.stream)); LS_CUDA(cudaFreeHost(w.hmem)); w.hmem = nullptr; w.hcap = 0; }
    LS_CUDA(cudaMallocHost(&w.hmem, total));
    w.hcap = total;
  }
  memcpy(w.hmem, a, sizeof(long long) * (size_t)R * C);
  memcpy(w.hmem + bA, starts, sizeof(int) * nl);
  LS_CUDA(cudaMemcpyAsync(w.dmem, w.hmem, in_bytes, cudaMemcpyHostToDevice, w.stream));
  LsArgs args{(const long long*)w.dmem, R, C, d, marginal, (const int*)(w.dmem + bA), n,
              max_rounds > 0 ? max_rounds : 4 * R, (long long*)(w.dmem + in_bytes),
              (int*)(w.dmem + in_bytes + bV)};
  unsigned long long sum = 0;        // saturated well above the int32 limit
  for (int64_t t = 0; t < (int64_t)R * C && sum < (1ull << 40); ++t) {
    const unsigned long long x = a[t] < 0 ? 0ull - (unsigned long long)a[t] : (unsigned long long)a[t];
    sum += x < (1ull << 40) ? x : 1ull << 40;
  }
  const bool narrow = sum < (1ull << 29);
  const size_t smem = (narrow ? 4 : 8) * (size_t)R * ls_stride(C);   // at most 64 rows x 132 columns = 66 KB
  if (ld_raise_smem_limit(narrow ? (const void*)local_search_kernel<int> : (const void*)local_search_kernel<long long>,
                          smem) != cudaSuccess)
    return ld_fail(LD_ERR_CUDA, "local search: cannot reserve %zu bytes of shared memory", smem);
  const int threads = (4 * (R - 1) + 31) & ~31;
  if (narrow) local_search_kernel<int><<<n, threads, smem, w.stream>>>(args);
  else local_search_kernel<long long><<<n, threads, smem, w.stream>>>(args);
  LS_CUDA(cudaGetLastError());
  LS_CUDA(cudaMemcpyAsync(w.hmem + in_bytes, w.dmem + in_bytes, out_bytes, cudaMemcpyDeviceToHost, w.stream));
  LS_CUDA(cudaStreamSynchronize(w.stream));
  memcpy(values, w.hmem + in_bytes, sizeof(long long) * (size_t)n);
  memcpy(labels, w.hmem + in_bytes + bV, sizeof(int) * nl);
  return LD_OK;
}
