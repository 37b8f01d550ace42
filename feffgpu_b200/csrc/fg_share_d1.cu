// The shared-matrix form: precision double, initial-state class 1.
#include "fg_shared.cuh"
FG_SHARE_INSTANCE(double, 1)
