// ep_xw_dd_b.cu - X pass kernels, part b of the half-line lengths, for dfloat fields.
#include "ep_xw.cuh"
EP_XW_PART(xw_part_b, EP_XW_LENGTHS_B)
template const XWKernels* xw_part_b<dfloat>(int);
