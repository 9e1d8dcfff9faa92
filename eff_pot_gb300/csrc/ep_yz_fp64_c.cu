// ep_yz_fp64_c.cu - Y and Z pass kernels, part c of the lengths, for double fields.
#include "ep_yz.cuh"
EP_YZ_PART(yz_part_c, EP_YZ_LENGTHS_C)
template const YZKernels* yz_part_c<double>(int);
