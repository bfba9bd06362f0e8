// ptd_flow_nonlin.cu -- the one-launch 2D step of the NONLIN model (ptd_flow.cuh).
#include "ptd_flow.cuh"

namespace ptd {

const void* flow_kernel_nonlin(int rows) { return flow_kernel_of<NONLIN>(rows); }

}  // namespace ptd
