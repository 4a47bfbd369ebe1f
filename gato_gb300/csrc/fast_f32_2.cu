// Register-engine pair-solve kernels, FP32 fields, shape group 2.
#define GATO_FAST_T float
#define GATO_FAST_G 2
#define GATO_FAST_SHAPES GATO_FAST_SHAPES_2
#include "fast_inst.cuh"
