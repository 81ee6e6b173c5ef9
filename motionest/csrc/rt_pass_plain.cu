#include "rt_pass.cuh"

namespace me {
template int launch_rt_mode<PM_FWD>(PassArgs&, const RtPlan&, cudaStream_t);
template int launch_rt_mode<PM_INV>(PassArgs&, const RtPlan&, cudaStream_t);
}  // namespace me
