// ptd_flow_nonlin.cu -- the flow kernels of the NONLIN model (ptd_flow.cuh, ptd_flow3.cuh).
#include "ptd_flow3.cuh"

namespace ptd {

const void* flow_kernel_nonlin(int rows, int planes, int warps)
{
    return planes ? flow3_kernel_of<NONLIN>(rows, planes, warps) : flow_kernel_of<NONLIN>(rows);
}

}  // namespace ptd
