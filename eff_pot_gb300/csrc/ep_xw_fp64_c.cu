// ep_xw_fp64_c.cu - X pass kernels, part c of the half-line lengths, for double fields.
#include "ep_xw.cuh"
EP_XW_PART(xw_part_c, EP_XW_LENGTHS_C)
template const XWKernels* xw_part_c<double>(int);
