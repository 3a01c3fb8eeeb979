// Enumeration on the tensor cores, for matrices with small entries (d <= 4).
//
// As in table_kernel.cuh the Gray index is N = h * B + j, and a labeling's
// value is a sum over (vector, column) pairs p of |H_p(h) - T_p(j)|.  For
// integers, with t_p the smallest value T_p takes,
//     |H - T| = |H - t| + (T - t) - 2 sum_{t < u <= T} [H >= u],
// and the last sum is a scalar product of the bits [H >= u] (features of h)
// with the bits [T >= u] (features of j).  So the values of 128 high indices
// against all B low labelings are one integer matrix product
//     acc(h, j) = 128 ((C_j - parity) / 2 - sum_f bit_f(h) weight_f(j)),
//     value = base(h) + parity + acc / 64,
// C_j and base(h) the parts that depend on j or h alone: exact in 32-bit
// accumulators.  Thresholds u that no reachable H separates share a feature
// (its weight counts them), those outside H's range need none; a +-1 or
// -1/0/1 matrix needs about as many features per column as there are low
// rows, 5 to 9.  Per 32 labelings and SM quarter the product costs (features /
// 61) clocks, the 8-bit table kernel 2.3 for four columns: 34 x 37 with
// marginals (256 features) 4.2 against 22 clocks.
//
// One persistent CTA per SM, 18 warps:
//   warps 8-15 (producers, two sets of four)  walk the high indices: H as
//       bytes, one row moved per tile of 128 high indices (128 walks in
//       lockstep), and write the feature bytes of the tile into the set's two
//       shared-memory chunks in the tensor core's core-matrix layout.  Four
//       lanes share a high index, each with a quarter of the pairs, so that a
//       warp's store is one 128-byte core matrix; a feature word is one byte
//       select, one add (the sum's top bit is the comparison) and one mask.
//       The sets take their own groups of 128 walks and their tiles are
//       multiplied in turn, because a tile's production is a chain of waits
//       and shared-memory round trips (1700 clocks at 256 features).  Word
//       counts are compile-time, so that a tile is straight code.
//   warps 16, 17            tcgen05.mma kind::i8 of one set each, 128 x B x 32
//       per instruction: A (u8 feature bytes) from the chunks, B (s8 weights of
//       all B low labelings, built once) resident in shared memory.  B = 256
//       takes 134 clocks (7800 products per clock and SM); 128 columns would
//       take 98, so the low rows are as many as give up to 256 labelings.  One
//       warp for both sets spent 500 clocks per tile between them in waits and
//       the commit.
//   warps 0-7 (epilogue, four per set)  a set's accumulators (256 columns of
//       TMEM) while the other set's tile is multiplied: maximum over j, and the
//       smallest high index attaining the thread's maximum.
// The block position of the maximum is found once, by the last CTA.
//
// Every wait is bounded (wait_polls); one that runs out makes all warps leave,
// TMEM is given back when the products in flight are done, and the result is
// LLONG_MAX (the host's LD_ERR_TIMEOUT).
#pragma once
#include "table_kernel.cuh"

namespace ld {

constexpr int kTcThreads = 32 * 18;
// Steps of a chunk (a set has two): the whole tile while the weights and four
// tiles fit in shared memory, else 10 or 12.  A commit costs the tensor pipe
// about 200 clocks beside 134 per product of two steps: with chunks of four
// steps they took most of the time.
__host__ __device__ constexpr int tc_chunk_steps(int steps) {
  return steps <= 16 ? steps : steps == 22 || steps == 24 ? 12 : 10;
}
constexpr int kTcMaxWords = 8;           // H words per lane and high index (WH)
constexpr int kTcMaxSteps = 30;
struct TcArgs {
  // image (32-bit words); a pair vector has 4 WH words, word (i, w) at 4 i + w
  const uint32_t* hinit;     // H bytes with every high row at label 0
  const uint32_t* tinit;     // T - t bytes with every low row at label 0
  const uint32_t* tmin;      // t, in H's byte offset
  const uint32_t* always;    // thresholds below every H, per pair (bytes)
  const uint32_t* once;      // 0xff where a pair has its only, or first, byte
  const uint32_t* delta;     // [row][label step l -> l + 1]: change of H (high rows) or T (low rows)
  const uint4* prog;         // [two steps][w]: byte selector and addend of two feature words
  const uint2* feat;         // [step][w]: first threshold - 1 and threshold count of four features (bytes, T - t)
  const uint32_t* consts;    // places (byte of the table row) of the j-only part, 127 at most in each
  const int* raw;            // R x C entries, row R-1 fixed
  int R, C, d, marginal;
  int k, B, N;               // low rows, low labelings, table rows (a multiple of 64)
  int labels;                // label steps per row: max(1, d - 1)
  int parity, nconst;
  int fw;                    // digits of a walk
  unsigned long long walk_len, it_begin, it_end;   // walks (by rank when sym_digits > 0)
  int sym_digits;
  int sym_words;                              // 64-bit completion counts
  const unsigned long long* sym_table;
  long long value_offset;
  unsigned wait_polls;                        // of every wait but the last, for the products in flight
  Reduce red;
};
constexpr unsigned kTcWaitPolls = 1u << 20;   // of up to about 3 us

__host__ __device__ inline size_t tc_align(size_t x) { return (x + 127) & ~(size_t)127; }

// dynamic shared memory, bytes: weights, ring, then the small arrays
struct TcSmem { size_t ring, delta, prog, init, sym, total; };
__host__ __device__ inline TcSmem tc_smem(int N, int steps, int rows, int labels, int WH, int sym_words) {
  TcSmem s;
  s.ring = tc_align((size_t)N * steps * 16);
  s.delta = s.ring + (size_t)4 * tc_chunk_steps(steps) * 2048;
  s.prog = s.delta + tc_align((size_t)rows * labels * WH * 16);
  s.init = s.prog + tc_align((size_t)steps * 4 * 8);
  s.sym = s.init + tc_align((size_t)WH * 16 * 3);
  s.total = s.sym + tc_align((size_t)sym_words * 8);
  return s;
}

namespace tc {

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// K-major operand without swizzle: 8-row x 16-byte core matrices, 128 bytes
// apart along K, `rows8` bytes apart per 8 rows
__device__ __forceinline__ uint64_t operand(uint32_t addr, uint32_t rows8) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | (uint64_t)(128u >> 4) << 16 |
         (uint64_t)((rows8 >> 4) & 0x3FFFu) << 32 | (uint64_t)1 << 46;
}
// kind::i8: s32 accumulators, A unsigned, B signed bytes, M = 128
__device__ __forceinline__ uint32_t instruction(int N) {
  return (2u << 4) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((128u >> 4) << 24);
}
__device__ __forceinline__ void bar_init(uint64_t* b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count));
}
__device__ __forceinline__ void bar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory");
}
// completes the barrier when the MMAs issued so far are done
__device__ __forceinline__ void commit(uint64_t* b) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(b)));
}
// Waits for a phase; false when it ran out or another warp gave up.  All
// lanes of a warp call it together.  (With one lane polling, or a time limit
// on the blocking poll, the enumeration measured 6 to 40 % slower; polling two
// barriers at once by half of the lanes each, 40 %.)
__device__ __forceinline__ bool bar_wait(uint64_t* b, unsigned phase, int* abort, unsigned polls) {
  const uint32_t a = smem_addr(b);
  for (unsigned n = 0; n < polls; ++n) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(a), "r"(phase) : "memory");
    if (__all_sync(0xffffffffu, done)) return true;
    if (__any_sync(0xffffffffu, *(volatile int*)abort)) return false;
  }
  *(volatile int*)abort = 1;
  return false;
}
// one lane of a converged warp
__device__ __forceinline__ bool elect() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0u;
}
__device__ __forceinline__ void load32(uint32_t addr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
      "%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr));
}
__device__ __forceinline__ void load_done() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// generic shared-memory writes -> visible to the tensor core
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ int byte_of(uint32_t w, int b) { return (int)((w >> (8 * b)) & 0xffu); }

// label of row `t` (t-th digit) in the reflected base-D code of x (D = 2 for d <= 2)
template <int D>
__device__ __forceinline__ int digit_label(unsigned long long x, int t) {
  for (int i = 0; i < t; ++i) x /= (unsigned long long)D;
  const int r = (int)(x % (2ull * D));
  return r < D ? r : 2 * D - 1 - r;
}

}  // namespace tc

// H word of step s when S steps are spread over WH words
__host__ __device__ constexpr int tc_word_of_step(int s, int WH, int S) { return s * WH / S; }

// D: digits of the code (2 for d <= 2); WH: H words per lane and high index;
// S: steps, a step being 16 feature bytes of a high index (one word per lane).
template <int D, int WH, int S>
__global__ void __launch_bounds__(kTcThreads, 1) tc_kernel(const TcArgs a) {
  constexpr int kSteps = S;
  constexpr int kCS = tc_chunk_steps(kSteps), kChunks = (kSteps + kCS - 1) / kCS;
  constexpr int kSets = 2, kThreads = kTcThreads;
  extern __shared__ __align__(1024) unsigned char tc_mem[];
  block_start();
  // Per set: two chunks, one accumulator buffer, and four slots for the bases
  // of its tiles (their four partial sums per row) and its walks.  A base slot
  // is written when the tile's first chunk is taken: then the products of the
  // tile before last are done, so the epilogue is past the one before that.  A
  // group's walks are written one tile earlier, with the chunks of the tile
  // before taken: the epilogue is then past tile T - 4, whose group (of one
  // tile) had the slot.  It reads all three before it releases the tile.
  __shared__ __align__(8) uint64_t chunk_full[kSets][2], chunk_empty[kSets][2];
  __shared__ __align__(8) uint64_t slot_full[kSets][4], acc_full[kSets], acc_empty[kSets], drained;
  __shared__ unsigned long long s_high[kSets][4][128], s_next[kSets];   // first high index of a group's walks
  __shared__ unsigned long long s_label[kSets][128];                     // labels of their high rows, two bits each (32 rows; d <= 2: one)
  __shared__ __align__(8) uint2 s_base[kSets][4][128];                    // four 16-bit partial sums
  __shared__ unsigned s_where[kSets][4];                                 // group and offset of a tile
  __shared__ int s_end[kSets], s_go[kSets];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort, s_first;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const TcSmem L = tc_smem(a.N, kSteps, a.R - 1, a.labels, WH, a.sym_words);
  unsigned char* sB = tc_mem;
  unsigned char* sRing = tc_mem + L.ring;
  uint32_t* sDelta = reinterpret_cast<uint32_t*>(tc_mem + L.delta);
  uint4* sProg = reinterpret_cast<uint4*>(tc_mem + L.prog);
  uint32_t* sInit = reinterpret_cast<uint32_t*>(tc_mem + L.init);   // hinit, tmin, once
  unsigned long long* sSym = reinterpret_cast<unsigned long long*>(tc_mem + L.sym);

  if (warp == 16) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_addr(&s_tmem)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int g = 0; g < kSets; ++g) {
      for (int i = 0; i < 2; ++i) {
        tc::bar_init(&chunk_full[g][i], 4);
        tc::bar_init(&chunk_empty[g][i], 1);
      }
      for (int i = 0; i < 4; ++i) tc::bar_init(&slot_full[g][i], 4);
      tc::bar_init(&acc_full[g], 1);
      tc::bar_init(&acc_empty[g], 4);
      s_end[g] = 0;
    }
    tc::bar_init(&drained, kSets);
    s_abort = 0;
    s_first = INT_MAX;
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  for (int t = tid; t < (a.R - 1) * a.labels * WH * 4; t += kThreads) sDelta[t] = a.delta[t];
  for (int t = tid; t < kSteps * 2; t += kThreads) sProg[t] = a.prog[t];
  for (int t = tid; t < WH * 4; t += kThreads) {
    sInit[t] = a.hinit[t];
    sInit[WH * 4 + t] = a.tmin[t];
    sInit[WH * 8 + t] = a.once[t];
  }
  for (int t = tid; t < a.sym_words; t += kThreads) sSym[t] = a.sym_table[t];
  __syncthreads();

  // Weights of table row j (rows B .. N-1 repeat labeling 0), half of the steps
  // per thread, four features at a time: clamp(T - first + 1, 0, count),
  // negated.  The tables it reads wait in the ring.  (One thread per row,
  // feature by feature from global memory: 22 us at 224 features, 47 at 480.)
  {
    uint2* sFeat = reinterpret_cast<uint2*>(sRing);
    uint32_t* sT = reinterpret_cast<uint32_t*>(sRing + kSteps * 32);   // tinit, always
    for (int t = tid; t < kSteps * 4; t += kThreads) sFeat[t] = a.feat[t];
    for (int t = tid; t < WH * 4; t += kThreads) { sT[t] = a.tinit[t]; sT[WH * 4 + t] = a.always[t]; }
    __syncthreads();
    const int j = tid >> 1;
    if (j < a.N) {
      unsigned long long lab = 0ull;                 // two bits per low row
      unsigned q = j < a.B ? (unsigned)j : 0u;
      for (int r = 0; r < a.k; ++r) {
        const unsigned x = q % (2u * D);
        lab |= (unsigned long long)(x < (unsigned)D ? x : 2u * D - 1u - x) << (2 * r);
        q /= (unsigned)D;
      }
      auto t_words = [&](int i, uint32_t (&tw)[4]) {
#pragma unroll
        for (int w = 0; w < 4; ++w) tw[w] = sT[4 * i + w];
        for (int r = 0; r < a.k; ++r) {
          const int up = (int)(lab >> (2 * r)) & 3;
          for (int l = 0; l < up; ++l)
#pragma unroll
            for (int w = 0; w < 4; ++w) tw[w] += sDelta[(r * a.labels + l) * WH * 4 + 4 * i + w];
        }
      };
      unsigned char* row = sB + (size_t)(j >> 3) * kSteps * 128 + (j & 7) * 16;
      uint32_t tw[4] = {0u, 0u, 0u, 0u};
      const int s0 = (tid & 1) ? kSteps / 2 : 0, s1 = (tid & 1) ? kSteps : kSteps / 2;
      for (int s = s0; s < s1; ++s) {
        if (s == s0 || tc_word_of_step(s, WH, S) != tc_word_of_step(s - 1, WH, S)) t_words(tc_word_of_step(s, WH, S), tw);
        uint32_t out[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const uint2 f = sFeat[4 * s + w];
          const uint4 pg = sProg[(s / 2) * 4 + w];
          const uint32_t t = __byte_perm(tw[w], 0u, s % 2 == 0 ? pg.x : pg.z);
          out[w] = __vsub4(0u, __vminu4(__vsubus4(t, f.x), f.y));
        }
        *reinterpret_cast<uint4*>(row + s * 128) = make_uint4(out[0], out[1], out[2], out[3]);
      }
      int cj = -a.parity;                            // the j-only part
      for (int i = tid & 1; i < WH; i += 2) {
        t_words(i, tw);
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const uint32_t t = tw[w] & sInit[WH * 8 + 4 * i + w];
          cj += (int)__dp4a(t, 0x01010101u, 0u) - 2 * (int)__dp4a(__vminu4(t, sT[WH * 4 + 4 * i + w]), 0x01010101u, 0u);
        }
      }
      cj += (tid & 1) ? a.parity : 0;                // counted once
      const unsigned pair = 3u << (tid & 30);
      cj = (cj + __shfl_xor_sync(pair, cj, 1)) / 2;  // even: the parity is taken out
      __syncwarp(pair);
      for (int n = tid & 1; n < a.nconst; n += 2) {
        const int at = (int)__ldg(a.consts + n), v = max(min(cj < 0 ? -cj - 127 * n : cj - 127 * n, 127), 0);
        row[(at >> 4) * 128 + (at & 15)] = (unsigned char)(cj < 0 ? -v : v);
      }
    }
  }
  tc::fence_async();
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = s_tmem;
  long long best_value = LLONG_MIN;
  unsigned long long best_high = ULLONG_MAX;

  if (warp >= 8 && warp < 16) {
    // ---- producers
    constexpr int Q = 4;                             // high indices per lane
    const int set = (warp - 8) >> 2, pw = warp & 3, w = lane & 3, pt = tid & 127;
    const int row0 = 32 * pw + (lane >> 2);          // rows row0 + 8 q
    const unsigned WL = (unsigned)a.walk_len;
    unsigned char* ring = sRing + (size_t)set * 2 * (2048 * kCS) + pw * (Q * 128 * kCS) + lane * 4;
    uint32_t H[Q][WH];
    unsigned tile = 0, chunk = 0, group = 0;         // of this set
    bool ok = true;
    auto take = [&] {
      if (chunk >= 2) ok = tc::bar_wait(&chunk_empty[set][chunk & 1u], (chunk / 2 - 1) & 1u, &s_abort, a.wait_polls) && ok;
    };
    auto hand = [&] {
      __syncwarp();
      if (lane == 0) tc::bar_arrive(&chunk_full[set][chunk & 1u]);
      ++chunk;
    };
    auto sync = [&] { asm volatile("bar.sync %0, 128;" ::"r"(1 + set) : "memory"); };
    // the next 128 walks are asked for one group ahead
    if (pt == 0) s_next[set] = atomicAdd(a.red.work, 128ull);
    sync();
    unsigned long long next = s_next[set];
    sync();
    while (ok) {
      const unsigned long long first = a.it_begin + next;
      if (first >= a.it_end) {                        // out of walks: tell the others
        take();
        if (lane == 0) { s_end[set] = (int)tile + 1; tc::bar_arrive(&slot_full[set][tile & 3u]); }
        hand();
        break;
      }
      unsigned long long ahead = 0;
      if (pt == 0) ahead = atomicAdd(a.red.work, 128ull);
      unsigned long long* high = s_high[set][group & 3u];
      {                                               // one walk per thread
        unsigned long long it = min(first + (unsigned long long)pt, a.it_end - 1);
        if constexpr (D >= 3) {
          if (a.sym_digits > 0) it = walk_of_rank<D, false>(it, a.sym_digits, sSym);
        }
        unsigned long long x = it * a.walk_len, lab = 0ull;
        high[pt] = x;
        if constexpr (D == 2) {
          lab = x ^ (x >> 1);
        } else {
          for (int r = 0; r < a.R - 1 - a.k; ++r) {
            const unsigned long long q = x / (unsigned long long)D;
            const unsigned n = (unsigned)(x - q * (unsigned long long)D);
            lab |= (unsigned long long)((q & 1ull) ? D - 1 - n : n) << (2 * r);
            x = q;
          }
        }
        s_label[set][pt] = lab;
      }
      sync();
      unsigned odd = 0;                               // parities of the walk numbers
      {
        unsigned long long x[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          x[q] = s_label[set][row0 + 8 * q];
          odd |= (unsigned)((high[row0 + 8 * q] / a.walk_len) & 1ull) << q;
#pragma unroll
          for (int i = 0; i < WH; ++i) H[q][i] = sInit[4 * i + w];
        }
        for (int r = a.k; r < a.R - 1; ++r) {
          const uint32_t* dr = sDelta + r * a.labels * WH * 4 + w;
#pragma unroll
          for (int l = 0; l < D - 1; ++l) {
            uint32_t v[WH];
#pragma unroll
            for (int i = 0; i < WH; ++i) v[i] = dr[l * WH * 4 + 4 * i];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
              const uint32_t up = (uint32_t)(x[q] & (D == 2 ? 1ull : 3ull)) > (uint32_t)l ? 1u : 0u;
#pragma unroll
              for (int i = 0; i < WH; ++i) H[q][i] += v[i] * up;
            }
          }
#pragma unroll
          for (int q = 0; q < Q; ++q) x[q] >>= D == 2 ? 1 : 2;
        }
      }
      for (unsigned u = 0; u < WL && ok; ++u, ++tile) {
        if (u) {
          // digit i0 (the lowest nonzero one of u) goes from c - 1 to c, read
          // mirrored when the number formed by the digits above it is odd;
          // the walk number is part of it for odd D, else only above a walk's
          // last digit
          int i0, c;
          unsigned above;
          if constexpr (D == 2) {
            i0 = __ffs((int)u) - 1;
            c = 1;
            above = u >> (i0 + 1);
          } else {
            unsigned v = u;
            i0 = 0;
            while (v % D == 0u) { v /= D; ++i0; }
            c = (int)(v % D);
            above = v / D;
          }
          const unsigned walks = (D & 1) || i0 == a.fw - 1 ? odd : 0u;
#pragma unroll
          for (int q = 0; q < Q; ++q) {
            const bool mirrored = ((above ^ (walks >> q)) & 1u) != 0u;
            const uint32_t sgn = mirrored ? 0xffffffffu : 1u;
            const int step = mirrored ? D - 1 - c : c - 1;     // label step between the two labels
            const uint32_t* dr = sDelta + ((a.k + i0) * a.labels + (D == 2 ? 0 : step)) * WH * 4 + w;
#pragma unroll
            for (int i = 0; i < WH; ++i) H[q][i] += dr[4 * i] * sgn;
          }
        }
        // base(h), a quarter per lane, and the feature bytes, chunk by chunk
        take();
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          uint32_t s = 0u;
#pragma unroll
          for (int i = 0; i < WH; ++i)
            asm("vabsdiff4.u32.u32.u32.add %0, %1, %2, %3;"
                : "=r"(s) : "r"(H[q][i] & sInit[WH * 8 + 4 * i + w]), "r"(sInit[WH * 4 + 4 * i + w]), "r"(s));
          reinterpret_cast<uint16_t*>(s_base[set][tile & 3u])[4 * (row0 + 8 * q) + w] = (uint16_t)s;
        }
        if (lane == 0) s_where[set][tile & 3u] = (group & 3u) << 30 | u;
        __syncwarp();
        if (lane == 0) tc::bar_arrive(&slot_full[set][tile & 3u]);
        unsigned char* dst = nullptr;
        uint4 pg = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int s = 0; s < kSteps; ++s) {
          if (s % kCS == 0) {
            if (s > 0) take();
            dst = ring + (chunk & 1u) * (2048 * kCS);
          }
          if (s % 2 == 0) pg = sProg[2 * s + w];
#pragma unroll
          for (int q = 0; q < Q; ++q) {
            const uint32_t h = __byte_perm(H[q][tc_word_of_step(s, WH, S)], 0u, s % 2 == 0 ? pg.x : pg.z);
            *reinterpret_cast<uint32_t*>(dst + q * (128 * kCS) + (s % kCS) * 128) =
                (h + (s % 2 == 0 ? pg.y : pg.w)) & 0x80808080u;
          }
          if (s % kCS == kCS - 1 || s == kSteps - 1) { tc::fence_async(); hand(); }
        }
      }
      // one thread looks at the flag, so that a set's warps leave together
      if (pt == 0) { s_next[set] = ahead; s_go[set] = *(volatile int*)&s_abort == 0; }
      sync();
      next = s_next[set];
      ok = s_go[set] != 0;
      ++group;
      sync();
    }
  } else if (warp >= 16) {
    // ---- matrix products of one set (the warp stays converged, one lane issues)
    const int g = warp - 16;
    const uint32_t idesc = tc::instruction(a.N), acc = tmem + g * 256u;
    const uint64_t db0 = tc::operand(tc::smem_addr(sB), kSteps * 128);
    const uint64_t da0 = tc::operand(tc::smem_addr(sRing) + g * 2 * (2048 * kCS), 128 * kCS);
    unsigned chunk = 0;
    bool ok = true;
    for (unsigned tile = 0; ok; ++tile) {
#pragma unroll
      for (int n = 0; n < kChunks; ++n, ++chunk) {
        const unsigned c = chunk & 1u;
        ok = tc::bar_wait(&chunk_full[g][c], (chunk / 2) & 1u, &s_abort, a.wait_polls);
        if (!ok) break;
        if (n == 0) {
          if (tile >= 1) ok = tc::bar_wait(&acc_empty[g], (tile - 1) & 1u, &s_abort, a.wait_polls);
          if (!ok) break;
          if ((unsigned)*(volatile int*)&s_end[g] == tile + 1u) {
            // the set's last, empty tile: the epilogue waits for it as for others
            // (and is past the one before, whose release is another phase)
            const unsigned last = tile * kChunks + kChunks - 1;
            if (lane == 0) tc::bar_arrive(kChunks <= 2 ? &chunk_empty[g][last & 1u] : &acc_full[g]);
            ok = false;
            break;
          }
        }
        tc::fence_after();
        if (tc::elect()) {
          const uint64_t da = da0 + (uint64_t)(c * (2048 * kCS / 16));
#pragma unroll
          for (int s = 0; s < kCS; s += 2)
            if (n * kCS + s < kSteps)
              asm volatile(
                  "{\n\t.reg .pred p;\n\t"
                  "setp.ne.b32 p, %4, 0;\n\t"
                  "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
                  ::"r"(acc), "l"(da + s * (128 / 16)), "l"(db0 + (n * kCS + s) * (128 / 16)), "r"(idesc),
                    "r"(n + s > 0 ? 1u : 0u));
          tc::commit(&chunk_empty[g][c]);            // kChunks <= 2: the last one also hands the accumulators over
          if (kChunks > 2 && n == kChunks - 1) tc::commit(&acc_full[g]);
        }
        __syncwarp();
      }
    }
    // nothing is in flight when TMEM is given back
    if (tc::elect()) tc::commit(&drained);
    __syncwarp();
    int never = 0;
    tc::bar_wait(&drained, 0u, &never, kTcWaitPolls);
  } else {
    // ---- epilogue: row tid % 128 of a set's tiles
    const int row = tid & 127, g = warp >> 2;
    const uint32_t addr = tmem + g * 256u + ((uint32_t)((warp & 3) * 32) << 16);
    int best = INT_MIN;
    for (unsigned tile = 0;; ++tile) {
      // the bases, then the release of the tile's last chunk: its products are
      // complete (with three chunks a tile that release could be two phases of
      // its barrier away, which one parity bit does not tell apart)
      const unsigned slot = tile & 3u, last = tile * kChunks + kChunks - 1;
      if (!tc::bar_wait(&slot_full[g][slot], (tile / 4) & 1u, &s_abort, a.wait_polls)) break;
      const uint2 part = s_base[g][slot][row];
      const unsigned where = s_where[g][slot];
      const unsigned long long high = s_high[g][where >> 30][row];
      const bool end = (unsigned)*(volatile int*)&s_end[g] == tile + 1u;
      if (!(kChunks <= 2 ? tc::bar_wait(&chunk_empty[g][last & 1u], (last / 2) & 1u, &s_abort, a.wait_polls)
                         : tc::bar_wait(&acc_full[g], tile & 1u, &s_abort, a.wait_polls)) || end)
        break;
      tc::fence_after();
      int m0 = INT_MIN, m1 = INT_MIN, m2 = INT_MIN, m3 = INT_MIN;
      for (int c = 0; c < a.N; c += 64) {
        uint32_t x[32], y[32];
        tc::load32(addr + (uint32_t)c, x);
        tc::load32(addr + (uint32_t)c + 32u, y);
        tc::load_done();
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          m0 = max(max(m0, (int)x[i]), (int)x[i + 1]);
          m1 = max(max(m1, (int)x[i + 2]), (int)x[i + 3]);
          m2 = max(max(m2, (int)y[i]), (int)y[i + 1]);
          m3 = max(max(m3, (int)y[i + 2]), (int)y[i + 3]);
        }
      }
      tc::fence_before();
      __syncwarp();
      if (lane == 0) tc::bar_arrive(&acc_empty[g]);
      const int v = (int)__dp2a_lo(part.x, 0x0101u, __dp2a_lo(part.y, 0x0101u, 0u)) +
                    (max(max(m0, m1), max(m2, m3)) >> 6);
      if (v >= best) {
        // rows past the last walk repeat it, at its indices
        const unsigned long long h = high + (where & 0x3fffffffu);
        if (v > best || h < best_high) { best = v; best_high = h; }
      }
    }
    if (best != INT_MIN) best_value = (long long)best + a.parity - a.value_offset;
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  if (s_abort) { best_value = LLONG_MAX; best_high = 0ull; }
  if (warp == 16) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));

  // (value, smallest high index) of the launch; the last CTA turns the index
  // into the smallest Gray index of that block of B labelings
  if (!grid_reduce(best_value, best_high, a.red)) return;
  __syncthreads();
  const long long gmax = *(volatile long long*)&a.red.result->value;
  const unsigned long long gh = *(volatile unsigned long long*)&a.red.result->index;
  if (gh == ULLONG_MAX || gmax == LLONG_MAX) return;
  // the entries in shared memory, then the high rows' sums per message and
  // column (d = 1: one signed sum), then two threads per low labeling, each
  // over half of the columns
  const int msgs = a.d, nh = a.R - 1 - a.k;
  int* sRaw = reinterpret_cast<int*>(tc_mem);
  int* sS = sRaw + a.R * a.C;
  int* sLab = sS + msgs * a.C;
  for (int t = tid; t < a.R * a.C; t += kThreads) sRaw[t] = a.raw[t];
  for (int t = tid; t < nh; t += kThreads) sLab[t] = tc::digit_label<D>(gh, t);
  __syncthreads();
  for (int t = tid; t < msgs * a.C; t += kThreads) {
    const int m = t / a.C, c = t - m * a.C;
    int s = m == 0 ? sRaw[(a.R - 1) * a.C + c] : 0;
    for (int r = 0; r < nh; ++r) {
      const int v = sRaw[(a.k + r) * a.C + c], lab = sLab[r];
      s += a.d == 1 ? (lab ? v : -v) : (lab == m ? v : 0);
    }
    sS[t] = s;
  }
  __syncthreads();
  if (tid < 512) {
    const int j = tid >> 1;
    unsigned long long lab = 0ull;
    unsigned q = (unsigned)j;
    for (int r = 0; r < a.k; ++r) {
      const unsigned x = q % (2u * D);
      lab |= (unsigned long long)(x < (unsigned)D ? x : 2u * D - 1u - x) << (2 * r);
      q /= (unsigned)D;
    }
    int v = 0;
    for (int c = tid & 1; c < a.C; c += 2) {
      int s[4] = {0, 0, 0, 0};
      for (int r = 0; r < a.k; ++r) {
        const int e = sRaw[r * a.C + c], l = (int)(lab >> (2 * r)) & 3;
        if (a.d == 1) s[0] += l ? e : -e;
        else {
#pragma unroll
          for (int m = 0; m < 4; ++m) s[m] += l == m ? e : 0;
        }
      }
#pragma unroll
      for (int m = 0; m < 4; ++m)
        if (m < msgs) {
          const int x = s[m] + sS[m * a.C + c];
          v += (a.marginal && c == 0) ? x : abs(x);
        }
    }
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    if (j < a.B && (long long)v == gmax) {
      int pos;
      if constexpr (D >= 4) pos = block_pos_of_entry<D>(j, a.k, (int)(gh & 1ull));
      else pos = (gh & 1ull) ? a.B - 1 - j : j;
      atomicMin(&s_first, pos);
    }
  }
  __syncthreads();
  if (tid == 0) {
    const unsigned long long n = gh * (unsigned long long)a.B + (unsigned long long)s_first;
    a.red.result->index = n;
    if (HostSlot* host = host_slot(a.red)) { host->index = n; host->t1 = global_ns(); }
  }
}

}  // namespace ld
