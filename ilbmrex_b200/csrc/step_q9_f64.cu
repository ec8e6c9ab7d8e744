// Level-step kernels, D2Q9 in FP64 storage.
#include "level_step.cuh"

ILBM_STEP_INSTANCE(9, ILBM_STORAGE_F64)
