// CTA pairs on 512 x 256 tiles.
#include "dense_launch_impl.cuh"

FLUXB_DENSE_INSTANCE(256, 0, 4, 2, 0, fluxb::kBsNone, 2);
FLUXB_DENSE_INSTANCE(256, 1, 4, 2, 0, fluxb::kBsNone, 2);
