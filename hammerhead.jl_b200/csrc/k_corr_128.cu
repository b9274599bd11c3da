// Fused window correlation, 128-point FFTs (windows of 64 and 128 px).
#include "hh_corr_fused.cuh"

namespace hh {
HH_CORR_SIZE(128)
}  // namespace hh
