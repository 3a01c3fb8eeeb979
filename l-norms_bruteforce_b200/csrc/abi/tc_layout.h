// Host side of the tensor-core enumeration (tc_kernel.cuh): the (vector,
// column) pairs of a matrix, the thresholds that separate its high rows'
// sums, and the words the kernel reads.
#pragma once
#include <cstdint>
#include <vector>

namespace ldsolve {

struct TcLayout {
  int WH = 0;                    // H words per lane
  int steps = 0;                 // steps of 16 features, even
  int N = 0;                     // table rows: B rounded up to a multiple of 64
  int labels = 1;                // label steps per row
  int parity = 0;
  // images, in the order of TcArgs
  std::vector<uint32_t> hinit, tinit, tmin, always, once, delta, prog, feat, consts;
  std::vector<int32_t> raw;
};

// Low rows of the tensor-core form: as many as give at most 256 labelings.
int tc_low_rows(int d, int R);

// Fills *out for k low rows; false when the entries are too large for byte
// sums or the features too many for shared memory.
bool tc_layout(const int64_t* a, int R, int C, int d, int marginal, int k, TcLayout* out);

}  // namespace ldsolve
