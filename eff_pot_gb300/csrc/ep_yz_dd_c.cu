// ep_yz_dd_c.cu - Y and Z pass kernels, part c of the lengths, for dfloat fields.
#include "ep_yz.cuh"
EP_YZ_PART(yz_part_c, EP_YZ_LENGTHS_C)
template const YZKernels* yz_part_c<dfloat>(int);
