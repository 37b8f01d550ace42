// The shared-matrix form: precision double, initial-state class 2.
#include "fg_shared.cuh"
FG_SHARE_INSTANCE(double, 2)
