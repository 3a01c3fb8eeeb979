// half_kernel<1, W, S, K> for S = 2, 4 (W = 4, 8, .., 32) and S = 8 (W = 4 .. 16).
#include "half_inst.cuh"
namespace ld {
void half_register_d1_split(HalfKernelTab& t) {
  inst::fill_half<1, 2, 1, 4>(t, std::make_integer_sequence<int, 8>{});
  inst::fill_half<1, 2, 2, 4>(t, std::make_integer_sequence<int, 8>{});
  inst::fill_half<1, 4, 1, 4>(t, std::make_integer_sequence<int, 8>{});
  inst::fill_half<1, 4, 2, 4>(t, std::make_integer_sequence<int, 8>{});
  inst::fill_half<1, 8, 1, 4>(t, std::make_integer_sequence<int, 4>{});
  inst::fill_half<1, 8, 2, 4>(t, std::make_integer_sequence<int, 4>{});
}
}  // namespace ld
