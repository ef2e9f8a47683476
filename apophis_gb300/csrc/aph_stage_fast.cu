// Batched stage kernel, fast arithmetic mode, for the reconstruction APH_STAGE_RECON.
#define APH_EXACT 0
#define APH_NS aph_fast
#include "aph_stage.cuh"
