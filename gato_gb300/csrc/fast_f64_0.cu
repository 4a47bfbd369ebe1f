// Register-engine pair-solve kernels, FP64 fields, shape group 0.
#define GATO_FAST_T double
#define GATO_FAST_G 0
#define GATO_FAST_FE
#define GATO_FAST_SHAPES GATO_FAST_SHAPES_0
#include "fast_inst.cuh"
