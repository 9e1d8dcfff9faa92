// ep_yz_fp64_d.cu - Y and Z pass kernels, part d of the lengths, for double fields.
#include "ep_yz.cuh"
EP_YZ_PART(yz_part_d, EP_YZ_LENGTHS_D)
template const YZKernels* yz_part_d<double>(int);
