// Fused window correlation, 48-point FFTs (windows of 24 and 48 px).
#include "hh_corr_fused.cuh"

namespace hh {
HH_CORR_SIZE(48)
}  // namespace hh
