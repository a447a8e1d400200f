// sort_argsort_narrow.cu -- awkward_argsort for bool and the 8-bit integers
// (segmented sort kernels: sort_impl.cuh).
#include "sort_impl.cuh"

GB_ARGSORT_ALL(bool, bool)
GB_ARGSORT_ALL(int8, int8_t)
GB_ARGSORT_ALL(uint8, uint8_t)
