// Register-engine pair-solve kernels, FP64 fields, shape group 2.
#define GATO_FAST_T double
#define GATO_FAST_G 2
#define GATO_FAST_FE
#define GATO_FAST_SHAPES GATO_FAST_SHAPES_2
#include "fast_inst.cuh"
