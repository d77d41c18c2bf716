// Plain-path kernels for 8-byte keys (integer and floating-point key kinds).
#include "radix_instances.cuh"

GB300_ALL_VALUES(8, gb300::FP_NONE, i)
GB300_ONESWEEP_FIRST(8)
GB300_ALL_VALUES(8, gb300::FP_ONESWEEP, f)
GB300_SINGLE_TILE_DESC_FP(8)
GB300_FINISH_ALL(8, gb300::FP_NONE, i)
GB300_FINISH_ALL(8, gb300::FP_ONESWEEP, f)
