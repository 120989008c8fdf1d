// CTA pairs with the staging rings of the all-gather / all-to-all push.
#include "dense_launch_impl.cuh"

FLUXB_DENSE_INSTANCE(256, 0, 4, 2, 16384, fluxb::kBsNone, 2);
FLUXB_DENSE_INSTANCE(256, 1, 4, 2, 16384, fluxb::kBsNone, 2);
FLUXB_DENSE_INSTANCE(256, 0, 6, 2, 16384);
FLUXB_DENSE_INSTANCE(256, 2, 6, 2, 16384);
FLUXB_DENSE_INSTANCE(256, 1, 6, 2, 16384);
