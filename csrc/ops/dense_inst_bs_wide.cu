// Block-scaled fp8, 128 x 256 tiles.
#include "dense_launch_impl.cuh"

FLUXB_DENSE_INSTANCE(256, 1, 3, 1, 32768, fluxb::kBsAny);
FLUXB_DENSE_INSTANCE(256, 1, 4, 1, 0, fluxb::kBsSquare);
FLUXB_DENSE_INSTANCE(256, 1, 4, 1, 0, fluxb::kBsColumn);
FLUXB_DENSE_INSTANCE(256, 1, 4, 1, 0, fluxb::kBsAny);
