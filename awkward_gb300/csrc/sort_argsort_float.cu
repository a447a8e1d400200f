// sort_argsort_float.cu -- awkward_argsort for floating point (segmented sort
// kernels: sort_impl.cuh).
#include "sort_impl.cuh"

GB_ARGSORT_ALL(float32, float)
GB_ARGSORT_ALL(float64, double)
