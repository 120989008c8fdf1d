// Signed 8-bit operands.
#include "dense_launch_impl.cuh"

FLUXB_DENSE_INSTANCE(256, 2, 6, 2);
FLUXB_DENSE_INSTANCE(128, 2, 8, 2);
FLUXB_DENSE_INSTANCE(128, 2, 6);
