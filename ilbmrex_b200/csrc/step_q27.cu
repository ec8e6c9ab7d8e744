// Level-step kernels, D3Q27 in the 4- and 2-byte storage forms.
#include "level_step.cuh"

ILBM_STEP_INSTANCE(27, ILBM_STORAGE_F32_SHIFT)
ILBM_STEP_INSTANCE(27, ILBM_STORAGE_F16_SCALED)
