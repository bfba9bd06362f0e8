// ptd_flow_lin.cu -- the flow kernels of the LIN model (ptd_flow.cuh, ptd_flow3.cuh).
#include "ptd_flow3.cuh"

namespace ptd {

const void* flow_kernel_lin(int rows, int planes, int warps)
{
    return planes ? flow3_kernel_of<LIN>(rows, planes, warps) : flow_kernel_of<LIN>(rows);
}

}  // namespace ptd
