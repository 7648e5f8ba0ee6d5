// The stage kernels built for five blocks per SM (48 registers): the interior body streams with the
// most loads in flight; the strip and row paths spill.
#define MFDM_STAGE_NS b4
#define MFDM_STAGE_BLOCKS 5
#define MFDM_STAGE_ONCE false
#include "mfdm_stage.cu"
