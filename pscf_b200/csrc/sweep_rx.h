// sweep_rx.h -- host side of the plane_rx.cuh kernels: which shapes they
// take, and their launches.  Every launch function returns the number of
// kernels it queued on `st` (0: the shape has no such kernels).
#pragma once
#include "plane_rx.cuh"

namespace pscfg {

struct RxPlan {
    bool plane = false;       // x-y planes (dim 2 and 3)
    bool line = false;        // z lines (dim 3)
    RxShape sh;
    RzShape z;
    int n3 = 1;
    RxTables tb[2];           // FP64, FP32
    RzCols zc[2];
};

// Fills sh, z and the column table (of one type) of a grid; false: a length
// without radices.
bool rx_shape(int dim, const int n[3], RxPlan &p, RxCol *cols, bool f32);

// dim 2: steps [t0, t1) of every field
template <typename T> int rx2_sweep(const RxPlan &p, cudaStream_t st, const SweepField<T> *f, int nf, int t0, int t1);
template <typename T> int rx2_stress(const RxPlan &p, cudaStream_t st, const StressJob<T> *jobs, int njobs, int maxs);

// dim 3: the first transforms of step t, one step, the stress slice sums
template <typename T> bool rx3_fits(const RxPlan &p);
template <typename T> int rx3_planes(const RxPlan &p, int nf);   // planes per CTA of the x-y kernels
template <typename T> int rx3_first(const RxPlan &p, cudaStream_t st, const SweepField<T> *f, int nf, int t);
template <typename T> int rx3_half(const RxPlan &p, cudaStream_t st, const SweepField<T> *f, int nf);   // k3v_half, and the z pass before it
template <typename T> int rx3_step(const RxPlan &p, cudaStream_t st, const SweepField<T> *f, int nf, int t);
template <typename T> int rx3_stress_tiles(const RxPlan &p);
template <typename T>
int rx3_stress(const RxPlan &p, cudaStream_t st, const StressJob<T> *jobs, int njobs, int s0, int cnt, int cs, cx<T> *spec,
               double *part);

}  // namespace pscfg
