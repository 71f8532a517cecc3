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

// The turn of a cooperative grid on a device. Two such grids in flight could each hold SMs
// that the other waits for, so a grid's stream first waits for the grid launched before
// it; the host waits for neither. Under a lock held until a build had ended, a build also
// waited for whatever another caller's stream still had to do, and eight threads' builds
// took 44 us each at (H2O)4 and 75 at (H2O)8; now 34 and 53, in two passes 34 and 58.
// Left, at the latest by the destructor, when the stream has been waited for.
class CooperativeTurn {
   public:
    explicit CooperativeTurn(int device) : device_(device) {}
    ~CooperativeTurn() { leave(); }
    CooperativeTurn(const CooperativeTurn&) = delete;
    CooperativeTurn& operator=(const CooperativeTurn&) = delete;
    // Runs launch() in turn on `stream`. The next turn's stream waits for all work that is
    // on this one by then, or, with an event, for `mark`, recorded right after the launch.
    template <class Launch>
    cudaError_t enter(cudaStream_t stream, cudaEvent_t mark, Launch launch) {
        std::unique_lock<std::mutex> lock(mutex());
        cudaError_t e = follow(stream);
        if (e == cudaSuccess) e = launch();
        if (e == cudaSuccess) e = take(stream, mark);
        return e;
    }
    void leave();

   private:
    std::mutex& mutex();
    cudaError_t follow(cudaStream_t stream);
    cudaError_t take(cudaStream_t stream, cudaEvent_t mark);
    int device_;
    uint64_t number_ = 0;  // 0: not entered
};

// J = scale * sum_q (B_q . D) B_q, J full n x n. The grid's CTAs wait on one another,
// bounded by wait_ns; past it *err (device-visible, 0 before) becomes 1 and J is
// undefined (stall: a self-test in which the CTAs' packets carry tags that none waits
// for). A small grid is one thread-block cluster; a larger one is cooperative and takes
// its turn (mark: CooperativeTurn::enter).
bool coulomb_fused_cooperative(const JkPlan& p);
cudaError_t coulomb_build_fused(const JkPlan& p, const double* D, double scale, double* J, double* work,
                                PacketSpace& held, int* err, uint64_t wait_ns, int stall, CooperativeTurn& turn,
                                cudaEvent_t mark, cudaStream_t stream);

}  // namespace hf
