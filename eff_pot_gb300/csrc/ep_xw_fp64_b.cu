// ep_xw_fp64_b.cu - X pass kernels, part b of the half-line lengths, for double fields.
#include "ep_xw.cuh"
EP_XW_PART(xw_part_b, EP_XW_LENGTHS_B)
template const XWKernels* xw_part_b<double>(int);
