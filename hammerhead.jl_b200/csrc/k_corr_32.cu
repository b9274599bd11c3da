// Fused window correlation, 32-point FFTs (windows of 16 and 32 px).
#include "hh_corr_fused.cuh"

namespace hh {
HH_CORR_SIZE(32)
}  // namespace hh
