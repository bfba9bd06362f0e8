// ptd_flow_linstep.cu -- the flow kernels of the LINSTEP model (ptd_flow.cuh, ptd_flow3.cuh).
#include "ptd_flow3.cuh"

namespace ptd {

const void* flow_kernel_linstep(int rows, int planes, int warps)
{
    return planes ? flow3_kernel_of<LINSTEP>(rows, planes, warps) : flow_kernel_of<LINSTEP>(rows);
}

}  // namespace ptd
