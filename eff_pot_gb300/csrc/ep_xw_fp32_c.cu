// ep_xw_fp32_c.cu - X pass kernels, part c of the half-line lengths, for float fields.
#include "ep_xw.cuh"
EP_XW_PART(xw_part_c, EP_XW_LENGTHS_C)
template const XWKernels* xw_part_c<float>(int);
