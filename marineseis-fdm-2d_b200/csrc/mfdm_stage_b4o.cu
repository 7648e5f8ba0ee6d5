// The stage kernels built for five blocks per SM, accumulating once a step.
#define MFDM_STAGE_NS b4o
#define MFDM_STAGE_BLOCKS 5
#define MFDM_STAGE_ONCE true
#include "mfdm_stage.cu"
