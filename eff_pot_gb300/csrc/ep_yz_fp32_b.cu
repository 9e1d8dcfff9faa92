// ep_yz_fp32_b.cu - Y and Z pass kernels, part b of the lengths, for float fields.
#include "ep_yz.cuh"
EP_YZ_PART(yz_part_b, EP_YZ_LENGTHS_B)
template const YZKernels* yz_part_b<float>(int);
