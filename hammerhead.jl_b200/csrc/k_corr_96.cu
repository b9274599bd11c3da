// Fused window correlation, 96-point FFTs (windows of 48 and 96 px).
#include "hh_corr_fused.cuh"

namespace hh {
HH_CORR_SIZE(96)
}  // namespace hh
