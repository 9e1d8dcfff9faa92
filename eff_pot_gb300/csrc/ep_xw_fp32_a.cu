// ep_xw_fp32_a.cu - X pass kernels, part a of the half-line lengths, for float fields.
#include "ep_xw.cuh"
EP_XW_PART(xw_part_a, EP_XW_LENGTHS_A)
template const XWKernels* xw_part_a<float>(int);
