// Single CTAs with the staging rings of the all-gather / all-to-all push.
#include "dense_launch_impl.cuh"

FLUXB_DENSE_INSTANCE(128, 0, 6, 1, 16384);
FLUXB_DENSE_INSTANCE(128, 2, 6, 1, 16384);
FLUXB_DENSE_INSTANCE(128, 1, 6, 1, 16384);
