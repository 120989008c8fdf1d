// Block-scaled fp8, 128-column tiles (single CTAs and CTA pairs).
#include "dense_launch_impl.cuh"

FLUXB_DENSE_INSTANCE(128, 1, 5, 2, 32768, fluxb::kBsAny);
FLUXB_DENSE_INSTANCE(128, 1, 6, 2, 0, fluxb::kBsAny);
FLUXB_DENSE_INSTANCE(128, 1, 4, 1, 32768, fluxb::kBsAny);
FLUXB_DENSE_INSTANCE(128, 1, 5, 1, 0, fluxb::kBsAny);
