// The stage kernels built for two blocks per SM: every register the general paths want.
#define MFDM_STAGE_NS b2
#define MFDM_STAGE_BLOCKS 2
#define MFDM_STAGE_ONCE false
#include "mfdm_stage.cu"
