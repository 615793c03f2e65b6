// kernels1.cuh -- 1-D sweeps of up to 128 points with the whole contour
// step as one dense matrix.
//
// Within a block, step_exp (src/step_mod.f90:146-176) is the fixed linear
// map q <- A q with
//   A = (4 E2 C2 E1 C2 E2 - E1 C1 E1) / 3,
// E1 = diag exp(-w ds/2), E2 = diag exp(-w ds/4) and C1, C2 the circulant
// matrices of the k-space filters, c[d] = (1/N) sum_k ek(k) cos(2 pi k d/N).
// On a line this short the six transforms of a step are nothing but latency
// (a dozen barriers for 64 points), while A is N^2 <= 16384 numbers that fit
// the registers of one CTA.  So a CTA forms A once per block (N^3
// multiply-adds through shared memory) and then walks the contour with one
// matrix-vector product and one barrier per step.
//
// The product is taken about the row's own value,
//   (A q)_i = (A 1)_i q_i + sum_j A_ij (q_j - q_i),
// and A 1 from centred circulants, (C x)_i = x_i + sum_j c[i - j] (x_j - x_i)
// (C 1 = ek(0) = 1): a constant q in a uniform field then stays that constant
// to the last bit, as it does through exact transforms, and the rounding of
// A's entries acts on differences only.
#pragma once
#include "kernels.cuh"

namespace pscfg {

// Four lanes per row, lane l holding the columns 8 j + 2 l and 8 j + 2 l + 1
// (16-byte reads of q, four consecutive chunks per step, the same for every
// row of a warp).  All arithmetic in FP64, also for FP32 slabs.
// Bound: the serial chain of a step (shared-memory read, NMAX/16 dependent
// multiply-adds, two shuffles, write, barrier).  64 points, 100 steps of a
// diblock: 70 us, the two blocks' matrices included, against 1132 us with
// k_sweep_plane; 192 fields: 97 us against 1166.
// grid = nfields, 4 NMAX threads.
template <typename T, int NMAX>
__global__ void __launch_bounds__(4 * NMAX) k1_sweep_dense(const SweepField<T> *fields, int n, int t0, int t1,
                                                           const cx<double> *__restrict__ tw)
{
    constexpr int J = NMAX / 8;
    const SweepField<T> &f = fields[blockIdx.x];
    __shared__ __align__(16) double qs[2][NMAX];
    __shared__ double c1[2 * NMAX], c2[2 * NMAX], e1[NMAX], e2[NMAX], x2[NMAX];
    int blk, src, dst;
    if (!step_slices(f, t0, blk, src, dst)) return;
    const int row = threadIdx.x >> 2, l = threadIdx.x & 3;
    if (threadIdx.x < NMAX) {
        const T *q = src_slice(f, src, n);
        qs[0][threadIdx.x] = threadIdx.x < n ? (double)q[threadIdx.x] : 0.0;
        qs[1][threadIdx.x] = 0.0;
    }
    // (C x)_row of a shared vector, in all four lanes of the row
    auto centred = [&](const double *c, const double *x) {
        const int i = row < n ? row : 0;
        double s = 0.0;
        for (int j = l; j < n; j += 4) s += c[i - j + n] * (x[j] - x[i]);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        return x[i] + s;
    };
    double a[2 * J], a1 = 0.0;
    int cur = -1, p = 0;
    for (int t = t0; t < t1; t++) {
        if (!step_slices(f, t, blk, src, dst)) break;
        if (blk != cur) {
            cur = blk;
            __syncthreads();
            // circulants, twice in a row so that c[i - j + n] needs no modulus
            for (int i = threadIdx.x; i < n; i += blockDim.x) {
                const int d = min(i, n - i);   // c[n - d] = c[d] to the last bit
                double s1 = 0.0, s2 = 0.0;
                for (int k = 0; k <= n / 2; k++) {
                    const double w = (k == 0 || 2 * k == n) ? 1.0 : 2.0;
                    const double c = w * tw[(k * d) % n].x;
                    s1 += c * (double)f.ek1[blk][k];
                    s2 += c * (double)f.ek2[blk][k];
                }
                c1[i] = c1[i + n] = s1 / n;
                c2[i] = c2[i + n] = s2 / n;
                e1[i] = (double)f.eo1[blk][i];
                e2[i] = (double)f.eo2[blk][i];
            }
            __syncthreads();
            const int i = row < n ? row : 0;
#pragma unroll
            for (int j = 0; j < 2 * J; j++) a[j] = 0.0;
            // c2[m - col] of an odd column is what the even one before it had
            // at m - 1: one shared-memory read for two multiply-adds
            double co[J];
#pragma unroll
            for (int j = 0; j < J; j++) co[j] = c2[max(n - 1 - (8 * j + 2 * l), 0)];
            for (int m = 0; m < n; m++) {
                const double x = c2[i - m + n] * e1[m];
#pragma unroll
                for (int j = 0; j < J; j++) {
                    const double ce = c2[m - min(8 * j + 2 * l, n - 1) + n];
                    a[2 * j] += x * ce;
                    a[2 * j + 1] += x * co[j];
                    co[j] = ce;
                }
            }
#pragma unroll
            for (int j = 0; j < 2 * J; j++) {
                const int cj = 8 * (j >> 1) + 2 * l + (j & 1), col = min(cj, n - 1);
                a[j] = cj >= n ? 0.0 : (4.0 * (e2[i] * e2[col] * a[j]) - e1[i] * e1[col] * c1[i - col + n]) / 3.0;
            }
            const double h = e1[i] * centred(c2, e2);
            if (l == 0 && row < n) x2[row] = h;
            __syncthreads();
            a1 = (4.0 * (e2[i] * centred(c2, x2)) - e1[i] * centred(c1, e1)) / 3.0;
        }
        __syncthreads();
        double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
        const double qi = qs[p][row < n ? row : 0];
#pragma unroll
        for (int j = 0; j < J; j++) {
            const double2 q = *(const double2 *)&qs[p][8 * j + 2 * l];
            if (j & 1) {
                s2 = fma(a[2 * j], q.x - qi, s2);
                s3 = fma(a[2 * j + 1], q.y - qi, s3);
            } else {
                s0 = fma(a[2 * j], q.x - qi, s0);
                s1 = fma(a[2 * j + 1], q.y - qi, s1);
            }
        }
        double s = (s0 + s1) + (s2 + s3);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s = fma(a1, qi, s);
        p ^= 1;
        if (l == 0 && row < n) {
            const T v = (T)s;
            qs[p][row] = (double)v;
            dst_slice(f, dst, n)[row] = v;
        }
    }
}

// Whether a launch of nf fields of n points, `steps` contour steps in `blocks`
// blocks altogether, is faster with k1_sweep_dense than with k_sweep_plane:
// a block's matrix costs as much as 5 to 50 dense steps, which long blocks pay
// back and chains of short blocks, or short checkpoint segments, do not.  The
// times are microseconds per field and, beyond what runs side by side (dense:
// per SM, by the registers a CTA takes; plane: 10 warps an SM), grow with the
// fields.  Sweeps measured, plane / dense: 2 fields, 8 blocks of 2 steps: 64
// points 211 / 109, 128 points 215 / 479; 2 blocks of 50: 1169 / 81, 1198 /
// 230; 1200 fields, 8 blocks of 2: 425 / 841, 536 / 4408; 2 of 50: 1472 /
// 583, 2179 / 2119.
inline bool k1_dense_pays(int n, int nf, long steps, long blocks)
{
    const double build = n <= 64 ? 2.0 + n / 6.0 : 0.46 * n, dense_step = n <= 64 ? 0.55 : 1.15;
    const double plane_step = n <= 32 ? 9.0 : 11.5;
    const double per_sm = (nf + 147) / 148;
    const double fd = per_sm * (n <= 32 ? 0.27 : n <= 64 ? 0.62 : 1.0), fp = nf * (n <= 64 ? 1 : 2) / 1480.0;
    return (blocks * build + steps * dense_step) * (fd > 1 ? fd : 1) < steps * plane_step * (fp > 1 ? fp : 1);
}

}  // namespace pscfg
