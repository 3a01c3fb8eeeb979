// half_kernel<1, W, 1, K>: W = 2, 4, .., 32 words, one or two high indices per thread.
#include "half_inst.cuh"
namespace ld {
void half_register_d1(HalfKernelTab& t) {
  inst::fill_half<1, 1, 1, 2>(t, std::make_integer_sequence<int, 16>{});
  inst::fill_half<1, 1, 2, 2>(t, std::make_integer_sequence<int, 16>{});
}
}  // namespace ld
