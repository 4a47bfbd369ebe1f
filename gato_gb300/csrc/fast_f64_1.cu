// Register-engine pair-solve kernels, FP64 fields, shape group 1.
#define GATO_FAST_T double
#define GATO_FAST_G 1
#define GATO_FAST_FE
#define GATO_FAST_SHAPES GATO_FAST_SHAPES_1
#include "fast_inst.cuh"
