#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <mutex>

#include "jk.cuh"

namespace hf {

// The Coulomb build of one cluster in one pass over B (coulomb.cu). Applies when
// coulomb_fused_work_doubles(p) > 0 (the slices of J and D fit the registers of
// one CTA per SM: n up to about 1100); work holds that many doubles.
size_t coulomb_fused_work_doubles(const JkPlan& p);

// What a workspace of the one-pass build holds: packets of builds of this shape with
// tags below `next`, or, with next == 0, anything (a build of another shape, or with
// next == 0, zeroes the packets first). Whoever allocates the workspace or writes
// something else to it sets next to 0.
struct PacketSpace {
    int64_t n = 0;
    int naux = 0;
    uint32_t next = 0;
};

// J = scale * sum_q (B_q . D) B_q, J full n x n. The grid's CTAs wait on one another,
// bounded by wait_ns; past it *err (device-visible, 0 before) becomes 1 and J is
// undefined (stall: a self-test in which one CTA's first packets are not sent). A small grid is one thread-block cluster; a larger one is cooperative
// (coulomb_fused_cooperative): hold cooperative_mutex(device) from its launch to its
// completion, since two such grids in flight could each hold SMs that the other waits for.
bool coulomb_fused_cooperative(const JkPlan& p);
cudaError_t coulomb_build_fused(const JkPlan& p, const double* D, double scale, double* J, double* work,
                                PacketSpace& held, int* err, uint64_t wait_ns, int stall, cudaStream_t stream);

std::mutex& cooperative_mutex(int device);

}  // namespace hf
