// Register-engine pair-solve kernels, FP32 fields, shape group 1.
#define GATO_FAST_T float
#define GATO_FAST_G 1
#define GATO_FAST_SHAPES GATO_FAST_SHAPES_1
#include "fast_inst.cuh"
