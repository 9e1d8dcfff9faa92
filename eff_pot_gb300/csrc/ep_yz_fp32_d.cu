// ep_yz_fp32_d.cu - Y and Z pass kernels, part d of the lengths, for float fields.
#include "ep_yz.cuh"
EP_YZ_PART(yz_part_d, EP_YZ_LENGTHS_D)
template const YZKernels* yz_part_d<float>(int);
