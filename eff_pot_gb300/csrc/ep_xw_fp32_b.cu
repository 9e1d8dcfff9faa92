// ep_xw_fp32_b.cu - X pass kernels, part b of the half-line lengths, for float fields.
#include "ep_xw.cuh"
EP_XW_PART(xw_part_b, EP_XW_LENGTHS_B)
template const XWKernels* xw_part_b<float>(int);
