// plane_rx.cuh kernels in FP32.
#include "sweep_rx.inl"

namespace pscfg {

RX_INSTANCES(float)

}  // namespace pscfg
