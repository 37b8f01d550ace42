// The shared-matrix form: precision float, initial-state class 1.
#include "fg_shared.cuh"
FG_SHARE_INSTANCE(float, 1)
