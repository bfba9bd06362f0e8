// ptd_flow_linstep.cu -- the one-launch 2D step of the LINSTEP model (ptd_flow.cuh).
#include "ptd_flow.cuh"

namespace ptd {

const void* flow_kernel_linstep(int rows) { return flow_kernel_of<LINSTEP>(rows); }

}  // namespace ptd
