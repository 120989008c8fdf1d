// CTA pairs, fp8 inputs.
#include "dense_launch_impl.cuh"

FLUXB_DENSE_INSTANCE(256, 1, 6, 2);
FLUXB_DENSE_INSTANCE(192, 1, 6, 2);
FLUXB_DENSE_INSTANCE(128, 1, 8, 2);
