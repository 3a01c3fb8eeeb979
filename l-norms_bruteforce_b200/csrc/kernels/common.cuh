// Device-side pieces shared by the enumeration kernels: packed integer lanes,
// the (value, Gray index) order, and the grid-wide reduction that turns
// per-thread maxima into the norm and the smallest Gray index attaining it
// (the reference's strict '>' inside a worker, L_CUDA.cu:80, and strict '<'
// across workers in index order, L_CUDA.cu:347).
#pragma once
#include <cstdint>
#include <climits>

namespace ld {

// One block's (or the final) candidate.
struct Slot {
  long long value;          // norm candidate (LLONG_MIN = none)
  unsigned long long index; // its Gray index (ULLONG_MAX = none)
};

// The result of a one-shot solve in pinned host memory, written by the kernel:
// a copy queued behind a small kernel took 8 us, a pair of timing events 6.
struct HostSlot {
  long long value;
  unsigned long long index;
  unsigned long long t0, t1;   // ns: the first block's start, the last one's end
};

// Scratch a launch reduces through.  `slots` holds one entry per block;
// `counter` and `gvalue` must be 0 / LLONG_MIN before the first launch and
// are restored by the last block of every launch.
struct Reduce {
  Slot* slots;
  unsigned int* counter;
  long long* gvalue;
  Slot* result;
  unsigned long long* work;   // walk counter the launch's warps fetch from (0 before
                              // the launch, reset by the last block), or null
};

// A one-shot solve's two further words of the scratch header, at these 64-bit
// words from `counter`: the first block's start time (ULLONG_MAX before the
// launch, re-armed likewise), and where the last block also writes the result
// and the times (null: nowhere; so the header's words must be zero elsewhere).
// Not members: with two pointers more the wide kernel's arguments were above
// 128 bytes, which the compiler handles differently, and its loops got other
// registers (24 x 300, d = 1: 48 instead of 63 and 2.12 ms instead of 1.86; 17
// x 2048, d = 2: 683 us instead of 593 even at 128 bytes).
constexpr int kStartWord = 5, kHostWord = 6;
__device__ __forceinline__ unsigned long long* start_word(const Reduce& R) {
  return reinterpret_cast<unsigned long long*>(R.counter) + kStartWord;
}
__device__ __forceinline__ HostSlot* host_slot(const Reduce& R) {
  return reinterpret_cast<HostSlot*>(reinterpret_cast<unsigned long long*>(R.counter)[kHostWord]);
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// The block's start time, kept by thread 0 for grid_reduce.
__device__ __forceinline__ unsigned long long& block_clock() {
  __shared__ unsigned long long t;
  return t;
}

// First thing in a kernel that may reduce into a HostSlot.
__device__ __forceinline__ void block_start() {
  if (threadIdx.x == 0) block_clock() = global_ns();
}

// ---- packed integer lanes ----------------------------------------------
// PK columns share one 32-bit word as independent signed lanes of 32/PK
// bits.  The host picks PK from an exact bound on every partial column sum,
// so lane arithmetic never wraps.  Only 32-bit and 8x4-bit lanes exist:
// vabsdiff4 runs at the rate of a 32-bit absolute difference on sm_100a and
// covers four columns, while the 16x2-bit form measured about seven times
// slower than two 32-bit ones.
template <int PK> struct Lanes;

template <> struct Lanes<1> {
  __device__ __forceinline__ static uint32_t add(uint32_t a, uint32_t b) { return a + b; }
  __device__ __forceinline__ static uint32_t sub(uint32_t a, uint32_t b) { return a - b; }
  // c + |a - b|, a and b signed 32-bit
  __device__ __forceinline__ static uint32_t sad(uint32_t a, uint32_t b, uint32_t c) {
    return __sad((int)a, (int)b, c);
  }
};

template <> struct Lanes<4> {
  __device__ __forceinline__ static uint32_t add(uint32_t a, uint32_t b) { return __vadd4(a, b); }
  __device__ __forceinline__ static uint32_t sub(uint32_t a, uint32_t b) { return __vsub4(a, b); }
  // c + sum over the 4 bytes of |a.b_i - b.b_i|, bytes signed 8-bit
  __device__ __forceinline__ static uint32_t sad(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("vabsdiff4.u32.s32.s32.add %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
  }
};

// ---- candidate order ----------------------------------------------------
__device__ __forceinline__ bool better(long long v, unsigned long long n,
                                       long long bv, unsigned long long bn) {
  return v > bv || (v == bv && n < bn);
}

__device__ __forceinline__ void warp_best(long long& v, unsigned long long& n) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    long long ov = __shfl_xor_sync(0xffffffffu, v, off);
    unsigned long long on = __shfl_xor_sync(0xffffffffu, n, off);
    if (better(ov, on, v, n)) { v = ov; n = on; }
  }
}

// The block's largest v and the smallest h that attains it, to every thread
// (h is arbitrary where v is INT_MIN everywhere).  The first index attaining
// the best is then found by the whole block in the one block of h, instead of
// by every thread in its own: with few high indices per thread that scan of a
// table by single threads was up to a third of a solve (d = 1: 31 x 40 905 ->
// 834 us, 22 x 19 24 -> 18, 19 x 251 50 -> 37).
__device__ __forceinline__ void block_top(int& v, unsigned long long& h) {
  __shared__ int s_top[32];
  __shared__ unsigned long long s_toph[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
  const int m = __reduce_max_sync(0xffffffffu, v);
  const unsigned hi = __reduce_min_sync(0xffffffffu, v == m ? (unsigned)(h >> 32) : 0xffffffffu);
  const unsigned lo = __reduce_min_sync(0xffffffffu, v == m && (unsigned)(h >> 32) == hi ? (unsigned)h : 0xffffffffu);
  if (lane == 0) { s_top[wid] = m; s_toph[wid] = ((unsigned long long)hi << 32) | lo; }
  __syncthreads();
  v = s_top[0];
  h = s_toph[0];
  for (int w = 1; w < nwarps; ++w)
    if (s_top[w] > v || (s_top[w] == v && s_toph[w] < h)) { v = s_top[w]; h = s_toph[w]; }
}

// The block's smallest j, to every thread.
__device__ __forceinline__ int block_min(int j) {
  __shared__ int s_min[32];
  const int nwarps = (blockDim.x + 31) >> 5;
  j = __reduce_min_sync(0xffffffffu, j);
  if ((threadIdx.x & 31) == 0) s_min[threadIdx.x >> 5] = j;
  __syncthreads();
  for (int w = 0; w < nwarps; ++w) j = min(j, s_min[w]);
  return j;
}

// Block-wide best, then one atomicMax per block on the value and a slot
// write; the last block to finish picks the smallest index among the slots
// that reach the maximum and re-arms the scratch for the next launch.
// Must be called by every thread of the block; true in the last block to
// finish (which has written the result).
__device__ __forceinline__ bool grid_reduce(long long v, unsigned long long n, const Reduce& R) {
  __shared__ long long s_v[32];
  __shared__ unsigned long long s_n[32];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
  warp_best(v, n);
  if (lane == 0) { s_v[wid] = v; s_n[wid] = n; }
  __syncthreads();
  if (wid == 0) {
    v = lane < nwarps ? s_v[lane] : LLONG_MIN;
    n = lane < nwarps ? s_n[lane] : ULLONG_MAX;
    warp_best(v, n);
    if (lane == 0) {
      R.slots[blockIdx.x].value = v;
      R.slots[blockIdx.x].index = n;
      if (v != LLONG_MIN) atomicMax(R.gvalue, v);
      if (host_slot(R)) atomicMin(start_word(R), block_clock());
      __threadfence();
      unsigned int done = atomicAdd(R.counter, 1u);
      s_last = (done == gridDim.x - 1);
    }
  }
  __syncthreads();
  if (!s_last) return false;
  __threadfence();
  const long long gmax = *((volatile long long*)R.gvalue);
  unsigned long long bn = ULLONG_MAX;
  for (unsigned int b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
    long long sv = __ldcg(&R.slots[b].value);
    unsigned long long sn = __ldcg(&R.slots[b].index);
    if (sv == gmax && sn < bn) bn = sn;
  }
  long long vv = gmax;
  warp_best(vv, bn);
  __syncthreads();
  if (lane == 0) { s_v[wid] = vv; s_n[wid] = bn; }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long best = ULLONG_MAX;
    for (int w = 0; w < nwarps; ++w) if (s_n[w] < best) best = s_n[w];
    R.result->value = gmax;
    R.result->index = best;
    if (HostSlot* host = host_slot(R)) *host = HostSlot{gmax, best, atomicExch(start_word(R), ULLONG_MAX), global_ns()};
    *R.gvalue = LLONG_MIN;
    *R.counter = 0u;
    if (R.work) *R.work = 0ull;   // every block has finished fetching walks
    __threadfence();
  }
  return true;
}

}  // namespace ld
