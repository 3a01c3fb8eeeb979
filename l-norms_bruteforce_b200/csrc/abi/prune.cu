// Pruned exact search (prune_kernel.cuh).  Exactly the plain enumeration's
// result; the incumbent only decides how much is skipped.
#include <cuda_runtime.h>

#include <algorithm>
#include <cinttypes>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "smem_limit.h"
#include "solver_internal.h"
#include "../kernels/registry.h"
#include "../kernels/table_kernel.cuh"

using namespace ldsolve;

#include "../kernels/prune_kernel.cuh"
#include "device_guard.h"

namespace {

// value of one labeling (labels of rows 0..R-2), int64
long long labeling_value(const int64_t* a, int R, int C, int d, int marginal, const int32_t* lab) {
  const int nm = d == 1 ? 1 : d;
  std::vector<long long> s((size_t)nm * C, 0);
  for (int l = 0; l < C; ++l) s[l] = a[(size_t)(R - 1) * C + l];
  for (int i = 0; i < R - 1; ++i)
    for (int l = 0; l < C; ++l) {
      const long long x = a[(size_t)i * C + l];
      if (d == 1) s[l] += lab[i] ? x : -x;
      else s[(size_t)lab[i] * C + l] += x;
    }
  long long v = 0;
  for (int m = 0; m < nm; ++m)
    for (int l = 0; l < C; ++l) {
      const long long x = s[(size_t)m * C + l];
      v += (d == 1 && marginal && l == 0) ? x : (x < 0 ? -x : x);
    }
  return v;
}

// Capacities of the two prefix lists (8 bytes each; the first also holds
// every walk).
constexpr unsigned long long kListA = 1ull << 21, kListB = 1ull << 22;
// Listed prefixes that hold more high indices than this are extended by a part
// of their rows first: such a level costs about 80 us (the norm of the rows
// left, a launch, a wait for the count), bounding 2^23 high indices 150.
constexpr unsigned long long kLevelHighs = 1ull << 23;

// The norm of rows [0, r) alone (every labeling of them), for the bounds:
// the plain solver on those rows plus a zero fixed row.  Falls back to the
// always-valid sum of absolute entries when the submatrix is too large to
// enumerate quickly.
ld_status rest_norm(const int64_t* a, int C, int d, int marginal, int r, int device, long long* out) {
  if (r <= 0) { *out = 0; return LD_OK; }
  const int base = d <= 2 ? 2 : d;
  if ((double)r * std::log2((double)base) > 34.0) {
    long long s = 0;
    for (int i = 0; i < r; ++i)
      for (int l = 0; l < C; ++l) { const int64_t x = a[(size_t)i * C + l]; s += x < 0 ? -x : x; }
    *out = s;
    return LD_OK;
  }
  std::vector<int64_t> sub((size_t)(r + 1) * C, 0);
  memcpy(sub.data(), a, sizeof(int64_t) * (size_t)r * C);
  ld_options o;
  ld_options_init(&o);
  o.device = device;
  ld_result res;
  ld_status st = ld_solve_reduced(sub.data(), r + 1, C, d, marginal, &o, &res, nullptr);
  if (st != LD_OK) return st;
  *out = res.value;
  return LD_OK;
}

}  // namespace

extern "C" ld_status ld_solve_pruned(const int64_t* a, int32_t R, int32_t C, int32_t d, int32_t marginal,
                                     const ld_options* opt, const int32_t* incumbent_labels,
                                     ld_result* res, int32_t* strategy, ld_prune_stats* stats) {
  ldsolve::ContextRestore ctx_restore;   // the caller's current context, back on return
  if (!a || !res || R < 1 || C < 1) return ld_fail(LD_ERR_ARG, "bad arguments");
  ld_options o;
  if (opt) o = *opt; else ld_options_init(&o);
  ld_prune_stats ps;
  memset(&ps, 0, sizeof ps);
  ps.incumbent = LLONG_MIN;
  if (incumbent_labels && R > 1) {
    for (int i = 0; i < R - 1; ++i)
      if (incumbent_labels[i] < 0 || incumbent_labels[i] >= (d == 1 ? 2 : d))
        return ld_fail(LD_ERR_ARG, "incumbent label %d of row %d out of range", incumbent_labels[i], i);
    ps.incumbent = labeling_value(a, R, C, d, marginal, incumbent_labels);
  }
  auto plain = [&]() -> ld_status {
    ld_status s = ld_solve_reduced(a, R, C, d, marginal, &o, res, strategy);
    ps.pruned = 0;
    if (stats) *stats = ps;
    return s;
  };
  if (d > 3 || R < 3 || C > LD_MAX_COLS || R > ld_max_rows_for(d)) return plain();
  DeviceInfo di;
  ld_status st = device_info(o.device, &di);
  if (st != LD_OK) return st;
  const Bounds bnd = compute_bounds(a, R, C, marginal);
  if (bnd.overflow || bnd.total + (marginal ? bnd.K : 0) > (long long)INT32_MAX) return plain();

  // table configuration with a pruned-kernel instance: the largest k whose
  // table fits 48 KB
  const int base = d <= 2 ? 2 : d, F = R - 1;
  Choice ch;
  const void* kb = nullptr;
  const void* ke = nullptr;
  int k = -1;
  for (int kk = std::min(F - 1, 10); kk >= 0 && k < 0; --kk) {
    const unsigned long long B = ipow(base, kk);
    if (B > 1024) continue;
    Choice c;
    if (!table_config(a, R, C, d, marginal, kk, 0, &c)) continue;
    // round to an instantiated shape
    if (d == 1 && !(c.WB <= 2 && c.WA <= 16)) {
      if (C > 64) continue;
      c.order.clear();
      for (int l = 0; l < C; ++l) c.order.push_back(l);
      c.WB = round4(C); c.WA = 0; c.lane_bits = 32;
    } else if (d >= 2) {
      if (c.WA > 0) c.WA = round4(c.WA); else c.WB = round4(c.WB);
    }
    c.WT = round4(c.WB + c.WA);
    const void* b1; const void* b2;
    ld::prune_kernel_ptrs(d, c.WB, c.WA, &b1, &b2);
    if (!b1 || B * (unsigned long long)(d * c.WT) * 4ull > 48ull * 1024ull) continue;
    ch = c; kb = b1; ke = b2; k = kk;
  }
  if (k < 0) return plain();
  const int nh = F - k;
  // walk rows: every walk gets one bound in the first launch, so at most
  // about 2^21 walks; the surviving ones are extended over all threads, so
  // long walks cost nothing extra there
  int fw = std::min(nh, 5);
  while (fw < nh && (double)(nh - fw) * std::log2((double)base) > 21.0) ++fw;
  const unsigned long long walk_len = ipow(base, fw), walks = ipow(base, nh - fw);
  const int B = (int)ipow(base, k);
  ps.low_rows = k; ps.walk_rows = fw;
  ps.walks_total = walks;
  ps.highs_total = walks * walk_len;
  ps.block = (uint64_t)B;

  // bounds of the rest rows, in the kernel's representation
  long long m_low = 0, m_walk = 0, kl = 0, kh = 0;
  st = rest_norm(a, C, d, marginal, k + fw, o.device, &m_walk);
  if (st != LD_OK) return st;
  if (d == 1 && marginal) {
    for (int i = 0; i < R; ++i) { const int64_t v = a[(size_t)i * C]; (i < k ? kl : kh) += v < 0 ? -v : v; }
    m_walk += kl;
  }
  const long long offset = kh + kl;
  const long long thr = ps.incumbent == LLONG_MIN ? LLONG_MIN : ps.incumbent + offset;

  // image: header | tot | h0 | tb | the prefix rows' totals | rows
  const int WT = ch.WT;
  std::vector<int64_t> tot(C, 0), h0(C, 0), tb(C, 0);
  for (int i = 0; i < R; ++i)
    for (int l = 0; l < C; ++l) tot[l] += a[(size_t)i * C + l];
  if (d == 1) {
    for (int l = 0; l < C; ++l) h0[l] = a[(size_t)(R - 1) * C + l];
    if (marginal) { h0[0] += kh; tb[0] = -kl; }
  }
  // totals of the fixed row and the rows above the lowest `rows`, packed
  auto pack_totals = [&](int rows, uint32_t* out) {
    std::vector<int64_t> t(C, 0);
    for (int i = rows; i < R; ++i)
      for (int l = 0; l < C; ++l) t[l] += a[(size_t)i * C + l];
    pack_row(t.data(), ch, out);
  };
  const size_t offBest = 64, offTot = 256, offH0 = 512, offTb = 768, offTtop = 1024, offA = 1280;
  const size_t upload = offA + (size_t)R * WT * 4;
  std::vector<char> image(upload, 0);
  const long long gmin = LLONG_MIN;
  memcpy(image.data() + 8, &gmin, sizeof gmin);
  const ld::Slot none{LLONG_MIN, ULLONG_MAX};
  memcpy(image.data() + offBest, &none, sizeof none);   // then the high indices kept, and the time
  pack_row(tot.data(), ch, (uint32_t*)(image.data() + offTot));
  pack_row(h0.data(), ch, (uint32_t*)(image.data() + offH0));
  pack_row(tb.data(), ch, (uint32_t*)(image.data() + offTb));
  pack_totals(k + fw, (uint32_t*)(image.data() + offTtop));
  for (int i = 0; i < R; ++i) pack_row(a + (size_t)i * C, ch, (uint32_t*)(image.data() + offA) + (size_t)i * WT);

  const size_t smem_b = (size_t)ld::prune_smem_words(d, WT, R, B, false) * 4;
  const size_t smem_e = (size_t)ld::prune_smem_words(d, WT, R, B, true) * 4;
  int bps_b = 0, bps_e = 0;
  if (cudaSetDevice(o.device) != cudaSuccess ||
      ld_raise_smem_limit(kb, smem_b) != cudaSuccess || ld_raise_smem_limit(ke, smem_e) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps_b, kb, ld::kPruneThreads, smem_b) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps_e, ke, ld::kPruneThreads, smem_e) != cudaSuccess ||
      bps_b < 1 || bps_e < 1)
    return ld_fail(LD_ERR_CUDA, "pruned kernels do not fit an SM");
  const unsigned long long full_b = (unsigned long long)di.sms * bps_b, blocks_e = (unsigned long long)di.sms * bps_e;
  // list A: the walks, then every other level's survivors; list B: the levels
  // between, or the surviving high indices of one launch
  const unsigned long long capA = std::max(walks, std::min<unsigned long long>(ps.highs_total, kListA));
  const unsigned long long capB = std::min<unsigned long long>(ps.highs_total, kListB);
  const size_t off_slots = align256(upload);
  const size_t off_a = off_slots + align256(blocks_e * sizeof(ld::Slot));
  const size_t off_b = off_a + align256(capA * 8);
  const size_t off_cnt = off_b + align256(capB * 8);
  const size_t dbytes = off_cnt + 256;
  if (o.device < 0 || o.device >= 64) return ld_fail(LD_ERR_ARG, "device %d out of range", o.device);
  std::lock_guard<std::mutex> lock(g_pws_mu[o.device]);
  Resources* r = &g_pws[o.device];
  // the workspace keeps the stream it was created with: the caller's, or its own
  if (r->device >= 0 && (cudaStream_t)o.stream != (r->own_stream ? nullptr : r->stream)) resources_release(r);
  st = resources_acquire(r, o.device, (cudaStream_t)o.stream, dbytes, 256);
  if (st != LD_OK) return st;
  char* dmem = (char*)r->dmem;
  cudaStream_t s = r->stream;
  struct Best { ld::Slot slot; unsigned long long kept, ns; };
  struct Bounded { unsigned long long count, t0, t1; };   // PruneArgs::list_count
  Best* out_h = (Best*)r->hstage;
  Bounded* out_b = (Bounded*)((char*)r->hstage + 64);
  float ms_b = 0.f, ms_s = 0.f;
  auto fail = [&](const char* what, cudaError_t e) {
    cudaStreamSynchronize(s);
    return ld_fail(LD_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  };
  unsigned long long visited = 0, h2d = upload, d2h = sizeof(Best);
  cudaError_t e;
  if ((e = cudaMemcpyAsync(dmem, image.data(), upload, cudaMemcpyHostToDevice, s)) != cudaSuccess) return fail("upload", e);
  {
    ld::PruneArgs args;
    ld::TableArgs& t = args.t;
    t.A = (const uint32_t*)(dmem + offA);
    t.tot = (const uint32_t*)(dmem + offTot);
    t.hinit = (const uint32_t*)(dmem + offH0);
    t.tbias = (const uint32_t*)(dmem + offTb);
    t.R = R; t.k = k; t.B = B; t.fw = fw;
    t.walk_len = walk_len;
    // d = 3: the walk bound also drops walks that hold no class minimum
    t.sym_digits = (d == 3 && !o.enumerate_all && nh - fw > 0) ? nh - fw : 0;
    t.sym_table = nullptr; t.rank_begin = t.rank_end = 0;
    t.value_offset = offset;
    t.pack16 = 0;
    t.red.counter = (unsigned int*)(dmem + 0);
    t.red.gvalue = (long long*)(dmem + 8);
    t.red.result = (ld::Slot*)(dmem + 16);
    t.red.slots = (ld::Slot*)(dmem + off_slots);
    t.red.work = nullptr;
    args.ttop = (const uint32_t*)(dmem + offTtop);
    args.threshold = thr;
    args.list_count = (unsigned long long*)(dmem + off_cnt);
    args.best = (ld::Slot*)(dmem + offBest);
    void* params[] = {&args};
    // Bound the extensions [begin, end) of the listed prefixes.  Runs of up to
    // `expand` of them: long ones share the seed of rows x words, but half of
    // the threads should have one.
    auto bound = [&](unsigned long long begin, unsigned long long end) -> cudaError_t {
      const unsigned long long total = end - begin;
      unsigned long long run = 1;
      while (run * base <= args.expand && run * base <= 4096 && total / run > full_b * (ld::kPruneThreads / 2))
        run *= base;
      args.run = run;
      t.walk_begin = begin; t.walk_end = end;
      const unsigned long long need = ((total + run - 1) / run + ld::kPruneThreads - 1) / ld::kPruneThreads;
      cudaError_t x = cudaMemsetAsync(args.list_count, 0, sizeof(Bounded), s);
      if (x != cudaSuccess) return x;
      return cudaLaunchKernel(kb, dim3((unsigned)std::min(full_b, need)), dim3(ld::kPruneThreads), params, smem_b, s);
    };
    unsigned long long* lists[2] = {(unsigned long long*)(dmem + off_a), (unsigned long long*)(dmem + off_b)};
    const unsigned long long caps[2] = {capA, capB};
    int cur = 0;                       // the list that holds the survivors
    args.src = nullptr; args.expand = walks; args.list = lists[0]; args.m_rest = m_walk;
    if ((e = bound(0, walks)) != cudaSuccess) return fail("walk bound launch", e);
    if ((e = cudaMemcpyAsync(out_b, args.list_count, sizeof(Bounded), cudaMemcpyDeviceToHost, s)) != cudaSuccess)
      return fail("survivors", e);
    // the low rows' norm, meanwhile
    if ((st = rest_norm(a, C, d, marginal, k, o.device, &m_low)) != LD_OK) { cudaStreamSynchronize(s); return st; }
    m_low += kl;
    if ((e = cudaSetDevice(o.device)) != cudaSuccess || (e = cudaStreamSynchronize(s)) != cudaSuccess)
      return fail("walk bound", e);
    unsigned long long n = out_b->count;
    ps.walks_kept = n;
    ms_b = (float)(out_b->t1 - out_b->t0) * 1e-6f;
    d2h += sizeof(Bounded);
    // When more than a quarter of the walks survive their bound the search
    // would do most of the plain enumeration's work at a lower rate: run the
    // plain enumeration instead (same result).
    if (o.prune_policy == 0 && n * 4ull > walks) {
      ps.bound_ms = ms_b;
      return plain();
    }
    t.sym_digits = 0;
    std::vector<uint32_t> tw(WT);
    for (int left = fw; left > 0;) {
      // extend by all the rows left, or by a part of them: about half, as many
      // as the other list takes
      int more = left;
      if ((double)n * (double)ipow(base, left) > (double)kLevelHighs) {
        int m = 0;
        while (2 * m < left && n * ipow(base, m + 1) <= std::min(kListA, caps[cur ^ 1])) ++m;
        if (m >= 2) more = m;
      }
      left -= more;
      args.m_rest = m_low;
      if (left > 0) {
        if ((st = rest_norm(a, C, d, marginal, k + left, o.device, &args.m_rest)) != LD_OK) return st;
        args.m_rest += kl;
        if ((e = cudaSetDevice(o.device)) != cudaSuccess) return fail("device", e);
      }
      if (d >= 2) {
        pack_totals(k + left, tw.data());
        if ((e = cudaMemcpyAsync(dmem + offTtop, tw.data(), WT * 4, cudaMemcpyHostToDevice, s)) != cudaSuccess ||
            (e = cudaStreamSynchronize(s)) != cudaSuccess)
          return fail("totals", e);
        h2d += WT * 4;
      }
      args.src = lists[cur];
      args.list = lists[cur ^ 1];
      args.expand = ipow(base, more);
      t.fw = left;
      t.walk_len = ipow(base, left);
      const unsigned long long total = n * args.expand;
      if (left > 0) {
        if ((e = bound(0, total)) != cudaSuccess) return fail("level launch", e);
        if ((e = cudaMemcpyAsync(out_b, args.list_count, sizeof(Bounded), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
            (e = cudaStreamSynchronize(s)) != cudaSuccess)
          return fail("level bound", e);
        n = out_b->count;
        ms_s += (float)(out_b->t1 - out_b->t0) * 1e-6f;
        cur ^= 1;
        d2h += sizeof(Bounded);
        continue;
      }
      // whole high indices: as many at once as the list can hold, a power of
      // the base (runs do not straddle the launches)
      visited = total;
      unsigned long long seg = 1;
      while (seg * base <= caps[cur ^ 1]) seg *= base;
      for (unsigned long long v = 0; v < total; v += seg) {
        if ((e = bound(v, std::min(total, v + seg))) != cudaSuccess) return fail("scan launch", e);
        if ((e = cudaLaunchKernel(ke, dim3((unsigned)blocks_e), dim3(ld::kPruneThreads), params, smem_e, s)) != cudaSuccess)
          return fail("evaluation launch", e);
      }
    }
  }
  if ((e = cudaMemcpyAsync(out_h, dmem + offBest, sizeof(Best), cudaMemcpyDeviceToHost, s)) != cudaSuccess)
    return fail("result", e);
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return fail("solve", e);
  ms_s += (float)out_h->ns * 1e-6f;
  const ld::Slot out = out_h->slot;
  const unsigned long long kept = out_h->kept;
  if (ps.incumbent != LLONG_MIN && out.value < ps.incumbent)
    return ld_fail(LD_ERR_CUDA, "internal: pruned result %lld below the incumbent %lld", (long long)out.value,
                   (long long)ps.incumbent);
  memset(res, 0, sizeof *res);
  res->value = out.value;
  res->gray_index = out.index;
  res->labelings = ld_labelings(R, d);
  res->kernel_ms = ms_b + ms_s;
  res->kernel_kind = LD_KERNEL_TABLE;
  res->lane_bits = ch.lane_bits;
  res->h2d_bytes = h2d;
  res->d2h_bytes = d2h;
  res->evaluated = kept * (unsigned long long)B;   // high indices whose block was scanned
  if (strategy) ld_gray_labels(out.index, R, d, strategy);
  ps.pruned = 1;
  ps.highs_kept = kept;
  ps.highs_visited = visited;
  ps.bound_ms = ms_b;
  ps.scan_ms = ms_s;
  if (stats) *stats = ps;
  return LD_OK;
}

