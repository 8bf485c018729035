// The residual replacement of MIXED CG on 32 x 16 tiles.
#define FAST_TAU_TX 32
#include "kern_misc.cu"
