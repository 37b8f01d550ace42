// The shared-matrix form: precision double, initial-state class 3.
#include "fg_shared.cuh"
FG_SHARE_INSTANCE(double, 3)
