// ep_yz_fp32_a.cu - Y and Z pass kernels, part a of the lengths, for float fields.
#include "ep_yz.cuh"
EP_YZ_PART(yz_part_a, EP_YZ_LENGTHS_A)
template const YZKernels* yz_part_a<float>(int);
