// Many steps in one launch on one lattice shape (ShapeSquare2); see mj_steps_impl.cuh.
#include "mj_steps_impl.cuh"

namespace mj {
mj_status launch_steps_square2(mj_plan* p, const StepsJob* job, const DynCoef& C, int* warps, bool& fits,
                         cudaStream_t s) {
    return launch_steps_shape<ShapeSquare2>(p, job, C, warps, fits, s);
}
}  // namespace mj
