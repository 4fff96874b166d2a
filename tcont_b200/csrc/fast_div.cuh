// fast_div.cuh -- device side of FastDiv (kernels.hpp).
#pragma once

#include "kernels.hpp"

namespace tcontb {

__device__ __forceinline__ uint32_t fast_div(uint32_t n, const FastDiv& f) { return (__umulhi(n, f.mul) + n) >> f.shr; }

}  // namespace tcontb
