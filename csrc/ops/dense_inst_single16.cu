// Single CTAs, 16-bit inputs.
#include "dense_launch_impl.cuh"

FLUXB_DENSE_INSTANCE(256, 0, 4);
FLUXB_DENSE_INSTANCE(192, 0, 4);
FLUXB_DENSE_INSTANCE(128, 0, 6);
