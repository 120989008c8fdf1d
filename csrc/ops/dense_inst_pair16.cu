// CTA pairs, 16-bit inputs.
#include "dense_launch_impl.cuh"

FLUXB_DENSE_INSTANCE(256, 0, 6, 2);
FLUXB_DENSE_INSTANCE(192, 0, 6, 2);
FLUXB_DENSE_INSTANCE(128, 0, 8, 2);
