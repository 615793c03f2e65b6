// plane_rx.cuh kernels for dim 3 in FP32.
#include "sweep_rx.inl"

namespace pscfg {

RX3_INSTANCES(float)

}  // namespace pscfg
