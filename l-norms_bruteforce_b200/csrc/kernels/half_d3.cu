// half_kernel<3, W, 1, K>: W = 2, 4, .., 32 words; two high indices per thread up to 10.
#include "half_inst.cuh"
namespace ld {
void half_register_d3(HalfKernelTab& t) {
  inst::fill_half<3, 1, 1, 2>(t, std::make_integer_sequence<int, 16>{});
  inst::fill_half<3, 1, 2, 2>(t, std::make_integer_sequence<int, 5>{});
}
}  // namespace ld
