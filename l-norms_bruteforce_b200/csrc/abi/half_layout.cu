#include "half_layout.h"

#include <algorithm>

#include "../kernels/half_kernel.cuh"

namespace ldsolve {

int half_vector_words(int W, int S) { return S * ld::half_row_words(W); }

void half_pack(const int64_t* v, const int64_t* bias, int C, int W, int S, uint32_t* out) {
  const int WT = ld::half_row_words(W);
  std::fill(out, out + S * WT, 0u);
  for (int c = 0; c < C; ++c) {
    const int g = c / (2 * W), f = c - g * 2 * W;
    const int64_t x = v[c] + (bias ? bias[c] : 0);
    out[g * WT + f / 2] += (f & 1) ? (uint32_t)x << 16 : (uint32_t)x;
    out[g * WT + W] += (uint32_t)v[c];
  }
}

HalfSums::HalfSums(const int64_t* a, int R, int C, int d, int marginal, int k0, int k1)
    : C(C), d(d), marginal(marginal), k0(k0), tot(C, 0), pos(C, 0), neg(C, 0), low_pos((size_t)(k1 - k0 + 1) * C),
      low_neg((size_t)(k1 - k0 + 1) * C) {
  for (int i = 0; i < R && fields; ++i) {
    const int64_t* row = a + (size_t)i * C;
    if (i >= k0 && i <= k1) low(i);
    for (int c = 0; c < C; ++c) {
      const int64_t v = row[c];
      if (v > 65535 || v < -65535) fields = false;
      tot[c] += v;
      if (d == 1 || i < R - 1) (v < 0 ? neg : pos)[c] += v < 0 ? -v : v;
    }
  }
  if (R <= k1) low(R);
}

void HalfSums::low(int k) {
  std::copy(pos.begin(), pos.end(), low_pos.begin() + (size_t)(k - k0) * C);
  std::copy(neg.begin(), neg.end(), low_neg.begin() + (size_t)(k - k0) * C);
}

bool half_layout(const HalfSums& sums, int k, int W, int S, HalfLayout* out) {
  const int C = sums.C, d = sums.d, marginal = sums.marginal;
  const int64_t* low_pos = sums.low_pos.data() + (size_t)(k - sums.k0) * C;
  const int64_t* low_neg = sums.low_neg.data() + (size_t)(k - sums.k0) * C;
  if (2 * W * S < C || !sums.fields) return false;
  out->W = W;
  out->S = S;
  out->beta.assign(C, 0);
  out->seed.assign(S, 0u);
  out->value_bias = 0;
  for (int g = 0; g < S; ++g) {
    // per half: the smallest sum of its fields, and how far the sum can rise
    int64_t low[2] = {0, 0}, range[2] = {0, 0};
    int64_t beta_sum = 0, st_min = 0, st_max = 0, st_any = 0;
    const int c0 = g * 2 * W, c1 = std::min(C, c0 + 2 * W);
    for (int c = c0; c < c1; ++c) {
      // negative / positive parts of the high and low rows
      const int64_t lp = low_pos[c], ln = low_neg[c], hp = sums.pos[c] - lp, hn = sums.neg[c] - ln;
      const int64_t low_sum = lp - ln, tot = sums.tot[c];
      // ranges of the register vectors and of the table vectors compared with them
      int64_t h_lo[3], h_hi[3], t_lo[3], t_hi[3];
      const int nv = d == 1 ? 1 : d;
      if (d == 1) {
        const int64_t hb = hn + hp, lb = ln + lp, lm = (marginal && c == 0) ? 1 : 0;   // LM shift K_H, K_L
        h_lo[0] = lm ? 0 : -hb; h_hi[0] = lm ? 2 * hb : hb;
        t_lo[0] = lm ? -2 * lb : -lb; t_hi[0] = lm ? 0 : lb;
        st_any += low_sum - (lm ? lb : 0);
      } else {
        for (int v = 0; v < nv; ++v) { h_lo[v] = -hn; h_hi[v] = hp; t_lo[v] = -lp; t_hi[v] = ln; }
        t_lo[nv - 1] = tot - lp; t_hi[nv - 1] = tot + ln;
        st_any += tot;
      }
      int64_t beta = 0;
      for (int v = 0; v < nv; ++v) beta = std::max(beta, -std::min(h_lo[v], t_lo[v]));
      out->beta[c] = beta;
      const int half = (c - c0) & 1;
      for (int v = 0; v < nv; ++v) {
        if (beta + std::max(h_hi[v], t_hi[v]) > 65535) return false;
        const int64_t m = std::max(h_lo[v], t_lo[v]);          // the maximum is never below
        low[half] += beta + m;
        range[half] += std::max(h_hi[v], t_hi[v]) - m;
        st_min += t_lo[v];
        st_max += t_hi[v];
      }
      beta_sum += beta * nv;
    }
    // the seed's own share, q - floor(st / 2) in [0, q - floor(st_min / 2)], goes to the low half
    const int64_t q = st_max >> 1;
    if (range[0] + q - (st_min >> 1) > 65535 || range[1] > 65535) return false;
    out->seed[g] = (uint32_t)(q - low[0]) - ((uint32_t)low[1] << 16);
    out->value_bias += (int)(2 * (low[0] + low[1] - q - beta_sum) - (st_any & 1));
  }
  return true;
}

bool half_layout(const int64_t* a, int R, int C, int d, int marginal, int k, int W, int S, HalfLayout* out) {
  return half_layout(HalfSums(a, R, C, d, marginal, k, k), k, W, S, out);
}

}  // namespace ldsolve
