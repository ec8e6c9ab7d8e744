// Level-step kernels, D3Q27 in FP64 storage.
#include "level_step.cuh"

ILBM_STEP_INSTANCE(27, ILBM_STORAGE_F64)
