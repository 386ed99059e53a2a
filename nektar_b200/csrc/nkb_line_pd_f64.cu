// FP64 instantiations of the line kernels' LN_PD operator (nkb_line_kernel.cuh).
#include "nkb_line_kernel.cuh"

namespace nkb
{
template int LineSwitch<LN_PD, double>(nkb_op *, const nkb_op *, const LineArgs<double> *, cudaStream_t);
} // namespace nkb
