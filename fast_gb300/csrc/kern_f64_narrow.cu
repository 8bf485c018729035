// Pure FP64 CG on 32 x 16 tiles.
#define FAST_TAU_TX 32
#include "kern_f64.cu"
