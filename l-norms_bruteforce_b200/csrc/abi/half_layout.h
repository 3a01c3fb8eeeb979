// Host side of the two-columns-per-word kernels (half_kernel.cuh): which
// matrices they take, the columns' biases, the entries' seeds, and packing.
#pragma once
#include <cstdint>
#include <vector>

namespace ldsolve {

// One matrix at k low rows, S slices of W words (2 W columns each).
struct HalfLayout {
  int W = 0, S = 1;
  std::vector<int64_t> beta;      // per column: added to every stored H and T value
  std::vector<uint32_t> seed;     // per slice: seed base of its entries
  int value_bias = 0;             // value = 2 Y - SH + value_bias (- the LM shift)
};

// A matrix's column sums by sign: of all rows a labeling moves (d = 1: the fixed
// row too), and of the low ones alone for k = k0 .. k1 of them (at most R).
struct HalfSums {
  HalfSums(const int64_t* a, int R, int C, int d, int marginal, int k0, int k1);
  int C, d, marginal, k0;
  bool fields = true;                             // every entry fits a 16-bit field
  std::vector<int64_t> tot, pos, neg;             // signed over all rows; positive, negative parts
  std::vector<int64_t> low_pos, low_neg;          // (k - k0) x C + c
 private:
  void low(int k);
};

// Fills *out, or returns false when a column's values do not fit a 16-bit
// field or a half of the packed accumulator could pass 65535.
bool half_layout(const HalfSums& sums, int k, int W, int S, HalfLayout* out);
bool half_layout(const int64_t* a, int R, int C, int d, int marginal, int k, int W, int S, HalfLayout* out);

// Words of one stored vector over all slices: S x half_row_words(W).
int half_vector_words(int W, int S);

// Pack C column values into the slices' data words (column 2 (g W + w) in the
// low half of word w of slice g, the next one in the high half) and their
// column sums; `bias` (may be null) is added to the fields, not to the sums.
void half_pack(const int64_t* v, const int64_t* bias, int C, int W, int S, uint32_t* out);

}  // namespace ldsolve
