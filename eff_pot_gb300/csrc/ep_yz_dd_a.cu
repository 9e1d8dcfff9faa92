// ep_yz_dd_a.cu - Y and Z pass kernels, part a of the lengths, for dfloat fields.
#include "ep_yz.cuh"
EP_YZ_PART(yz_part_a, EP_YZ_LENGTHS_A)
template const YZKernels* yz_part_a<dfloat>(int);
