// Helpers that fill the half_kernel lookup (registry.h) with instances.
#pragma once
#include <utility>

#include "half_kernel.cuh"
#include "registry.h"

namespace ld {
namespace inst {

constexpr int log2_of(int s) { return s == 1 ? 0 : s == 2 ? 1 : s == 4 ? 2 : 3; }
// W = STEP (i + 1) for i in I...
template <int D, int S, int K, int STEP, int... I>
void fill_half(HalfKernelTab& t, std::integer_sequence<int, I...>) {
  ((t[D][STEP * (I + 1)][log2_of(S)][K - 1] = (const void*)&half_kernel<D, STEP * (I + 1), S, K>), ...);
}

}  // namespace inst
}  // namespace ld
