// ptd_flow_lin.cu -- the one-launch 2D step of the LIN model (ptd_flow.cuh).
#include "ptd_flow.cuh"

namespace ptd {

const void* flow_kernel_lin(int rows) { return flow_kernel_of<LIN>(rows); }

}  // namespace ptd
