// half_kernel<3, W, S, K> for S = 2, 4, 8 (W = 4, 8, 12, 16).
#include "half_inst.cuh"
namespace ld {
void half_register_d3_split(HalfKernelTab& t) {
  using Seq = std::make_integer_sequence<int, 4>;
  inst::fill_half<3, 2, 1, 4>(t, Seq{});
  inst::fill_half<3, 2, 2, 4>(t, Seq{});
  inst::fill_half<3, 4, 1, 4>(t, Seq{});
  inst::fill_half<3, 4, 2, 4>(t, Seq{});
  inst::fill_half<3, 8, 1, 4>(t, Seq{});
  inst::fill_half<3, 8, 2, 4>(t, Seq{});
}
}  // namespace ld
