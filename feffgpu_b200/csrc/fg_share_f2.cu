// The shared-matrix form: precision float, initial-state class 2.
#include "fg_shared.cuh"
FG_SHARE_INSTANCE(float, 2)
