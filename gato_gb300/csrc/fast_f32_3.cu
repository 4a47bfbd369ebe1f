// Register-engine pair-solve kernels, FP32 fields, shape group 3.
#define GATO_FAST_T float
#define GATO_FAST_G 3
#define GATO_FAST_SHAPES GATO_FAST_SHAPES_3
#include "fast_inst.cuh"
