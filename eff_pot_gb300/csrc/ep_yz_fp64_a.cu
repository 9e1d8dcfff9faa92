// ep_yz_fp64_a.cu - Y and Z pass kernels, part a of the lengths, for double fields.
#include "ep_yz.cuh"
EP_YZ_PART(yz_part_a, EP_YZ_LENGTHS_A)
template const YZKernels* yz_part_a<double>(int);
