// Fills the tc_kernel lookup (registry.h) with instances.
#pragma once
#include <utility>

#include "registry.h"
#include "tc_kernel.cuh"

namespace ld {
namespace inst {

template <int D, int WH, int S>
constexpr const void* tc_kp() {
  if constexpr (S < WH || S > 12 * WH) return nullptr;
  else return (const void*)&tc_kernel<D, WH, S>;
}
template <int D, int... I>
void fill_tc(TcKernelTab& t, std::integer_sequence<int, I...>) {
  ((t[D - 2][I / (kTcMaxSteps / 2)][I % (kTcMaxSteps / 2)] =
        tc_kp<D, I / (kTcMaxSteps / 2) + 1, 2 * (I % (kTcMaxSteps / 2)) + 2>()), ...);
}

}  // namespace inst
}  // namespace ld
