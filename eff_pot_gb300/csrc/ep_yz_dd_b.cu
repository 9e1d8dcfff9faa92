// ep_yz_dd_b.cu - Y and Z pass kernels, part b of the lengths, for dfloat fields.
#include "ep_yz.cuh"
EP_YZ_PART(yz_part_b, EP_YZ_LENGTHS_B)
template const YZKernels* yz_part_b<dfloat>(int);
