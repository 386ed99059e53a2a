// FP32 instantiations of the line kernels' LN_IP operator (nkb_line_kernel.cuh).
#include "nkb_line_kernel.cuh"

namespace nkb
{
template int LineSwitch<LN_IP, float>(nkb_op *, const nkb_op *, const LineArgs<float> *, cudaStream_t);
} // namespace nkb
