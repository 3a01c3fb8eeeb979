#include "tc_layout.h"

#include <algorithm>
#include <numeric>

#include "../kernels/registry.h"
#include "../kernels/tc_kernel.cuh"

namespace ldsolve {
namespace {

// One (vector, column) pair: H starts at h0 and changes by step(v, l) x entry
// when a high row goes from label l to l + 1; T starts at t0 and changes by
// the opposite for a low row.
struct Pair {
  int col = 0;
  int coef[10] = {};                 // per label step
  int64_t h0 = 0, t0 = 0;
  int64_t h_lo = 0, h_hi = 0, h_step = 0, t_lo = 0, t_hi = 0;
  int64_t origin = 0;                // H bytes hold H - origin
  int features = 0, feature0 = 0;    // how many, and the first one's place
  int always = 0;                    // thresholds 1 .. always (T - t_lo) are below every H
};

// Thresholds first .. first + count - 1 (T - t_lo), compared at H >= at (H byte).
struct Feature { int first, count, at; };

}  // namespace

int tc_low_rows(int d, int R) {
  const int base = d <= 2 ? 2 : d;
  int k = 0;
  for (long long b = base; b <= 256 && k + 1 < R; b *= base) ++k;
  return k;
}

bool tc_layout(const int64_t* a, int R, int C, int d, int marginal, int k, TcLayout* out) {
  const int V = d;                   // table vectors per column
  const int L = std::max(1, d - 1);
  const int P = V * C;
  if (d < 1 || d > 4 || P > 16 * ld::kTcMaxWords) return false;
  if (d >= 3 && R - 1 - k > 32) return false;   // the kernel holds a walk's labels in 64 bits, two for each high row
  std::vector<Pair> pairs;
  std::vector<Feature> feats;
  pairs.reserve(P);
  feats.reserve(16 * ld::kTcMaxSteps + 256);
  int64_t c_lo = 0, c_hi = 0, parity = 0;   // range and parity of the j-only part
  for (int v = 0; v < V; ++v)
    for (int c = 0; c < C; ++c) {
      Pair p;
      p.col = c;
      int64_t low = 0, high = 0, tot = 0, abs_high = 0, abs_low = 0;
      for (int i = 0; i < R; ++i) {
        const int64_t x = a[(size_t)i * C + c];
        if (x > 127 || x < -127) return false;
        tot += x;
        if (i < k) { low += x; abs_low += std::llabs(x); }
        else if (i < R - 1) { high += x; abs_high += std::llabs(x); }
      }
      if (d == 1) {
        const int64_t fixed = a[(size_t)(R - 1) * C + c];
        const bool lm = marginal && c == 0;             // the shift that makes column 0's term its own sum
        p.coef[0] = 2;
        p.h0 = fixed - high + (lm ? abs_high + std::llabs(fixed) : 0);
        p.t0 = low - (lm ? abs_low : 0);
      } else if (d == 2) {
        p.coef[0] = 1;
        p.t0 = v == 0 ? 0 : tot;
      } else if (v < d - 1) {                           // rows labelled v + 1
        for (int l = 0; l < L; ++l) p.coef[l] = l == v ? 1 : l == v + 1 ? -1 : 0;
      } else {                                          // rows with any label but 0
        p.coef[0] = 1;
        p.t0 = tot;
      }
      p.h_lo = p.h_hi = p.h0;
      p.t_lo = p.t_hi = p.t0;
      for (int i = 0; i < R - 1; ++i) {
        const int64_t x = a[(size_t)i * C + c];
        int64_t s = 0, lo = 0, hi = 0;
        for (int l = 0; l < L; ++l) {
          s += p.coef[l] * x;
          lo = std::min(lo, s);
          hi = std::max(hi, s);
          const int64_t step = std::llabs(p.coef[l] * x);
          if (i >= k && step != 0 && p.h_step != 1) p.h_step = std::gcd(p.h_step, step);
        }
        if (i < k) { p.t_lo -= hi; p.t_hi -= lo; }
        else { p.h_lo += lo; p.h_hi += hi; }
      }
      p.origin = std::min(p.h_lo, p.t_lo);
      if (std::max(p.h_hi, p.t_lo) - p.origin > 255 || p.t_hi - p.t_lo > 255) return false;
      p.feature0 = (int)feats.size();
      // thresholds u in (t_lo, t_hi], grouped by the smallest H that reaches them
      for (int64_t u = p.t_lo + 1; u <= p.t_hi; ++u) {
        const int t = (int)(u - p.t_lo);
        if (u <= p.h_lo) { p.always = t; continue; }
        if (u > p.h_hi) break;                           // no H reaches it (nor any above)
        const int64_t rep = p.h_step > 0 ? p.h_lo + (u - p.h_lo + p.h_step - 1) / p.h_step * p.h_step : p.h_hi + 1;
        if (rep > p.h_hi) break;
        const int at = (int)(rep - p.origin);
        if (p.features > 0 && feats.back().at == at) {
          if (++feats.back().count > 127) return false;   // a weight is a signed byte
          continue;
        }
        // H - at + 128 must stay in a byte
        if (at > 128 || p.h_hi - rep > 127 || p.h_lo - rep < -128) return false;
        feats.push_back({t, 1, at});
        ++p.features;
      }
      if (feats.size() > 16 * (size_t)ld::kTcMaxSteps) return false;
      c_lo -= p.always;
      c_hi += p.t_hi - p.t_lo;
      parity += p.t0 - p.t_lo;
      pairs.push_back(p);
    }
  const int par = (int)(parity & 1);
  // the j-only part halved, in signed bytes
  const int nconst = (int)std::max<int64_t>(1, (std::max(c_hi, 1 - c_lo) / 2 + 126) / 127);
  // H words: 4 WH bins of four bytes; bin (i, w) takes four features per step
  // of its word.  Pairs go in order into the open bin; one whose features do
  // not fit continues in the next bin with a second byte.  The fewest steps
  // that hold all features, then the fewest words whose bytes suffice.  The
  // constant's bytes fill what is left of the bins.
  int room[ld::kTcMaxWords];                          // features of a word's bins
  auto rooms = [&](int S, int WH) {
    std::fill(room, room + WH, 0);
    for (int s = 0; s < S; ++s) room[ld::tc_word_of_step(s, WH, S)] += 4;
  };
  // calls put(bin, pair, features so far, features put there) until all are placed
  auto place = [&](int WH, auto&& put) {
    int at = 0, used = 0, left = room[0];
    for (int q = 0; q < P; ++q) {
      int f = 0;
      do {
        while (used == 4 || (f < pairs[q].features && left == 0)) {
          if (++at == 4 * WH) return false;
          used = 0;
          left = room[at / 4];
        }
        const int n = std::min(left, pairs[q].features - f);
        put(at, q, f, n);
        ++used;
        f += n;
        left -= n;
      } while (f < pairs[q].features);
    }
    return true;
  };
  out->steps = 0;
  const int need = (int)feats.size() + nconst;
  for (int S = std::max(2, ((need + 15) / 16 + 1) & ~1); S <= ld::kTcMaxSteps && !out->steps; S += 2)
    for (int WH = std::max(1, (P + 15) / 16); WH <= ld::kTcMaxWords; ++WH) {
      if (!ld::tc_kernel_ptr(d <= 2 ? 2 : d, WH, S)) continue;
      rooms(S, WH);
      if (!place(WH, [](int, int, int, int) {})) continue;   // 16 S >= need: the constant has room
      out->steps = S;
      out->WH = WH;
      break;
    }
  const int base = d <= 2 ? 2 : d;
  int B = 1;
  for (int i = 0; i < k; ++i) B *= base;
  out->N = (B + 63) / 64 * 64;
  out->labels = L;
  out->parity = par;
  if (out->steps == 0 || out->N > 256) return false;
  const int WH = out->WH, WP = 4 * WH, S = out->steps;
  rooms(S, WH);
  out->hinit.assign(WP, 0u);
  out->tinit.assign(WP, 0u);
  out->tmin.assign(WP, 0u);
  out->always.assign(WP, 0u);
  out->once.assign(WP, 0u);
  out->delta.assign((size_t)(R - 1) * L * WP, 0u);
  out->prog.assign((size_t)out->steps * 8, 0u);
  out->feat.assign((size_t)out->steps * 8, 0u);
  out->consts.clear();
  int first_step[ld::kTcMaxWords + 1];
  for (int s = S - 1; s >= 0; --s) first_step[ld::tc_word_of_step(s, WH, S)] = s;
  std::vector<int> bytes(WP, 0), filled(WP, 0);       // of each bin (i, w), at 4 i + w
  // the next free feature place of a bin: byte b of word w in step s
  auto next = [&](int at, int* s, int* b) {
    *s = first_step[at / 4] + filled[at] / 4;
    *b = filled[at]++ % 4;
    return out->prog.data() + ((size_t)(*s / 2) * 4 + at % 4) * 4 + (*s % 2) * 2;   // selector, addend
  };
  place(WH, [&](int at, int q, int f0, int n) {
    const Pair& p = pairs[q];
    const int byte = bytes[at]++, sh = 8 * byte;
    out->hinit[at] |= (uint32_t)(p.h0 - p.origin) << sh;
    out->tinit[at] |= (uint32_t)(p.t0 - p.t_lo) << sh;
    if (f0 == 0) {                                    // what is counted once per pair
      out->once[at] |= 0xffu << sh;
      out->tmin[at] |= (uint32_t)(p.t_lo - p.origin) << sh;
      out->always[at] |= (uint32_t)p.always << sh;
    }
    for (int r = 0; r < R - 1; ++r)
      for (int l = 0; l < L; ++l) {
        const int64_t x = p.coef[l] * a[(size_t)r * C + p.col];
        out->delta[((size_t)r * L + l) * WP + at] += (uint32_t)(r < k ? -x : x) << sh;
      }
    for (int f = f0; f < f0 + n; ++f) {
      int s, b;
      uint32_t* prog = next(at, &s, &b);
      const Feature& x = feats[p.feature0 + f];
      prog[0] |= (uint32_t)byte << (4 * b);
      prog[1] |= (uint32_t)(128 - x.at) << (8 * b);
      uint32_t* feat = out->feat.data() + ((size_t)s * 4 + at % 4) * 2;   // first threshold - 1, count
      feat[0] |= (uint32_t)(x.first - 1) << (8 * b);
      feat[1] |= (uint32_t)x.count << (8 * b);
    }
  });
  for (int at = 0, left = nconst; at < WP; ++at)
    while (filled[at] < room[at / 4]) {
      int s, b;
      uint32_t* prog = next(at, &s, &b);
      prog[0] |= 4u << (4 * b);                       // the zero byte
      if (left-- <= 0) continue;
      prog[1] |= 128u << (8 * b);                     // always set
      out->consts.push_back((uint32_t)(16 * s + 4 * (at % 4) + b));
    }
  out->raw.resize((size_t)R * C);
  for (size_t t = 0; t < out->raw.size(); ++t) out->raw[t] = (int32_t)a[t];
  return true;
}

}  // namespace ldsolve
