// Level-step kernels, D3Q19 in FP64 storage.
#include "level_step.cuh"

ILBM_STEP_INSTANCE(19, ILBM_STORAGE_F64)
