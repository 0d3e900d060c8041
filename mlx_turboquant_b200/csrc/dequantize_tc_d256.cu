// The tensor-core dequantize kernels of head_dim 256.
#include "dequantize_tc.cuh"

TQ_DEQUANTIZE_KERNELS(256)
