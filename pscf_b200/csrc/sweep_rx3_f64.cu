// plane_rx.cuh kernels for dim 3 in FP64.
#include "sweep_rx.inl"

namespace pscfg {

RX3_INSTANCES(double)

}  // namespace pscfg
