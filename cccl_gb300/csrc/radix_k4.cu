// Plain-path kernels for 4-byte keys (integer and floating-point key kinds).
#include "radix_instances.cuh"

GB300_ALL_VALUES(4, gb300::FP_NONE, i)
GB300_ONESWEEP_FIRST(4)
GB300_ALL_VALUES(4, gb300::FP_ONESWEEP, f)
GB300_SINGLE_TILE_DESC_FP(4)
GB300_FINISH_ALL(4, gb300::FP_NONE, i)
GB300_FINISH_ALL(4, gb300::FP_ONESWEEP, f)
