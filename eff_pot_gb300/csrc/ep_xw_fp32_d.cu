// ep_xw_fp32_d.cu - X pass kernels, part d of the half-line lengths, for float fields.
#include "ep_xw.cuh"
EP_XW_PART(xw_part_d, EP_XW_LENGTHS_D)
template const XWKernels* xw_part_d<float>(int);
