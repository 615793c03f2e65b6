// plane_rx.cuh kernels for dim 2 in FP32.
#include "sweep_rx.inl"

namespace pscfg {

RX2_INSTANCES(float)

}  // namespace pscfg
