// sort_argsort_middle.cu -- awkward_argsort for the 16-bit integers and int32
// (segmented sort kernels: sort_impl.cuh).
#include "sort_impl.cuh"

GB_ARGSORT_ALL(int16, int16_t)
GB_ARGSORT_ALL(uint16, uint16_t)
GB_ARGSORT_ALL(int32, int32_t)
