// tc_kernel<3, WH, S>: WH = 1..8 H words, S = 2, 4, .., 30 steps
// (at least one and at most twelve per word).
#include "tc_inst.cuh"
namespace ld {
void tc_register_d3(TcKernelTab& t) { inst::fill_tc<3>(t, std::make_integer_sequence<int, kTcMaxWords * kTcMaxSteps / 2>{}); }
}  // namespace ld
