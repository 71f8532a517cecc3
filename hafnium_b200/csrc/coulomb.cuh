#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <mutex>

#include "jk.cuh"

namespace hf {

// The Coulomb build of one cluster in one pass over B (coulomb.cu). Applies when
// coulomb_fused_work_doubles(p) > 0 (the slices of J and D fit the registers of
// one CTA per SM: n up to about 1100); work holds that many doubles, zeroed once
// when it is allocated.
size_t coulomb_fused_work_doubles(const JkPlan& p);

// J = scale * sum_q (B_q . D) B_q, J full n x n. The grid's CTAs wait on one another,
// bounded by wait_ns; past it *err (device-visible, 0 before) becomes 1 and J is
// undefined. A small grid is one thread-block cluster; a larger one is cooperative
// (coulomb_fused_cooperative): hold cooperative_mutex(device) from its launch to its
// completion, since two such grids in flight could each hold SMs that the other waits for.
bool coulomb_fused_cooperative(const JkPlan& p);
cudaError_t coulomb_build_fused(const JkPlan& p, const double* D, double scale, double* J, double* work, int* err,
                                uint64_t wait_ns, cudaStream_t stream);

std::mutex& cooperative_mutex(int device);

}  // namespace hf
