// The plain FP64 step with the rounding of every operation of the
// reference's expressions: the forward of the differentiated step
// (shield_mp_step_ieee).
//
// A window of steps is differentiated at the states the forward leaves, and
// those decide branches by the sign of a rounding residue: where a process
// uses a species up, q - (factor a + factor b) leaves 0 or +-1e-20, and the
// next step's fix_negative borrows from another species if it is negative.
// With the plain form's exp, log and powers (good to 0.5 to 1.3 units in the
// last place, as CUDA's are, but not to the reference's last place) such signs, and
// with them 2e-3 of the norm of a 4-step window's rain gradient (C24 L79), came
// out differently. The step's own outputs do not see this: plain and IEEE
// forms agree to 1e-14.
//
// Division is the branch-free quotient of mp_math.cuh, which rounds as IEEE
// division does for the finite normal divisors and quotients of the step.
#define SHIELD_IEEE
#include "mp_kernel.cuh"
#include "mp_launch.h"

namespace shield {

cudaError_t mp_launch_ieee(const MpArgs& A, cudaStream_t st) { return launch_shapes<false, false>(A, st); }

}  // namespace shield
