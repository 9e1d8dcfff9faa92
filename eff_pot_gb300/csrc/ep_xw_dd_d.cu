// ep_xw_dd_d.cu - X pass kernels, part d of the half-line lengths, for dfloat fields.
#include "ep_xw.cuh"
EP_XW_PART(xw_part_d, EP_XW_LENGTHS_D)
template const XWKernels* xw_part_d<dfloat>(int);
