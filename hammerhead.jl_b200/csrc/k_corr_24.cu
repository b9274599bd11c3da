// Fused window correlation, 24-point FFTs (windows of 12 and 24 px).
#include "hh_corr_fused.cuh"

namespace hh {
HH_CORR_SIZE(24)
}  // namespace hh
