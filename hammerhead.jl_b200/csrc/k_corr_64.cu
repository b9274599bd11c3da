// Fused window correlation, 64-point FFTs (windows of 32 and 64 px).
#include "hh_corr_fused.cuh"

namespace hh {
HH_CORR_SIZE(64)
}  // namespace hh
