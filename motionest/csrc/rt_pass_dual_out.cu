#include "rt_pass.cuh"

namespace me {
template int launch_rt_mode<PM_DUAL_OUT>(PassArgs&, const RtPlan&, cudaStream_t);
}  // namespace me
