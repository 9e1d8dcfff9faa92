// ep_xw_fp64_a.cu - X pass kernels, part a of the half-line lengths, for double fields.
#include "ep_xw.cuh"
EP_XW_PART(xw_part_a, EP_XW_LENGTHS_A)
template const XWKernels* xw_part_a<double>(int);
