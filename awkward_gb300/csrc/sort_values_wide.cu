// sort_values_wide.cu -- awkward_sort for the 64-bit integers and floating
// point (segmented sort kernels: sort_impl.cuh).
#include "sort_impl.cuh"

GB_SORT(int64, int64_t)
GB_SORT(uint64, uint64_t)
GB_SORT(float32, float)
GB_SORT(float64, double)
