// Fused window correlation, 16-point FFTs (windows of 8 and 16 px).
#include "hh_corr_fused.cuh"

namespace hh {
HH_CORR_SIZE(16)
}  // namespace hh
