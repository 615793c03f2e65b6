// sweep_rx.inl -- launches of the plane_rx.cuh kernels for one type,
// included by the sweep_rx*.cu units (one per dimension and type).
#include <algorithm>

#include "../../include/pscf_gpu.h"
#include "launch_util.h"
#include "sweep_rx.h"

namespace pscfg {

template <typename T> static int prec_of() { return sizeof(T) == 8 ? 0 : 1; }

static const int RX_NT = 288;            // threads of the run-time shaped plane kernels (most)
static const size_t SMEM_MOST = 226 * 1024;
static const int RX_SMS = 148;

static bool small10(const RxShape &s) { return s.P1 <= 8 && s.Q1 <= 10 && s.P2 <= 8 && s.Q2 <= 10; }

// threads of a CTA whose largest pass has `items`, in whole rounds
static int rx_threads(int items, int most = RX_NT)
{
    const int rounds = (items + most - 1) / most;
    const int per = (items + rounds - 1) / rounds;
    return std::max(32, std::min(most, (per + 31) / 32 * 32));
}

// planes per CTA: as many as keep the row pass within one round of the
// threads, fewer where the launch would not fill two CTAs on every SM
static int rx_ppc(int items, int n3, int nf, size_t plane_bytes)
{
    int p = std::max(1, std::min(n3, RX_NT / std::max(items, 1)));
    while (p > 1 && (p * plane_bytes > 100 * 1024 || (long)nf * ((n3 + p - 1) / p) < 296)) p--;
    return p;
}

#define RX_LAUNCH(kernel, grid, block, smem, st, ...)                        \
    do {                                                                     \
        if (allow_dyn_smem((const void *)kernel) != cudaSuccess) return -1;  \
        kernel<<<grid, block, smem, st>>>(__VA_ARGS__);                      \
        if (cudaPeekAtLastError() != cudaSuccess) return -1;                 \
    } while (0)

// A field's sweep by two CTAs while both have an SM of their own, by one CTA
// with its tables in shared memory while there is one per SM, else by two
// CTAs sharing each SM.  64 x 64, 100 steps, sweep alone: 1 instance (2
// fields) 1.05 / 1.33 / 1.8 ms, 96 instances 2.83 (two CTAs each) / - / 2.41.
template <typename T, typename SH>
static int sweep2(const RxPlan &p, SH sh, cudaStream_t st, const SweepField<T> *f, int nf, int t0, int t1)
{
    const RxShape &s = p.sh;
    const RxTables &tb = p.tb[prec_of<T>()];
    const int npair = s.Q2 * s.HP, items = std::max(npair * s.Q1, s.Q2 * s.n1h);
    if (2 * nf <= RX_SMS && rx2_pair_smem<T>(s.n1, s.n2, npair, true) <= SMEM_MOST) {
        auto *k = k2x_pair<T, SH, RX_NT, 1, true>;
        RX_LAUNCH(k, 2 * nf, rx_threads(std::max({items, npair * s.P1, s.P2 * s.n1h})),
                  rx2_pair_smem<T>(s.n1, s.n2, npair, true), st, f, sh, tb, t0, t1);
    } else if (nf <= RX_SMS && rx2_smem<T>(s.n1, s.n2, true) <= SMEM_MOST) {
        auto *k = k2x_sweep<T, SH, 544, 1, true>;
        RX_LAUNCH(k, nf, rx_threads(std::max(items, 2 * s.P2 * s.n1h), 544), rx2_smem<T>(s.n1, s.n2, true), st, f, sh, tb, t0, t1);
    } else if (rx2_smem<T>(s.n1, s.n2, false) <= SMEM_MOST) {
        auto *k = k2x_sweep<T, SH, RX_NT, 2, false>;
        RX_LAUNCH(k, nf, rx_threads(items), rx2_smem<T>(s.n1, s.n2, false), st, f, sh, tb, t0, t1);
    } else {
        return 0;
    }
    return 1;
}

template <typename T> int rx2_sweep(const RxPlan &p, cudaStream_t st, const SweepField<T> *f, int nf, int t0, int t1)
{
    if (!p.plane) return 0;
    if (p.sh.n1 == 64 && p.sh.n2 == 64) return sweep2<T>(p, RxFixed<64, 64, 8, 8>(), st, f, nf, t0, t1);
    return small10(p.sh) ? sweep2<T>(p, RxShape10{p.sh}, st, f, nf, t0, t1) : sweep2<T>(p, p.sh, st, f, nf, t0, t1);
}

template <typename T, typename SH, int NT>
static int stress2(const RxPlan &p, SH sh, int threads, cudaStream_t st, const StressJob<T> *jobs, int njobs, int maxs)
{
    auto *k = k2x_stress<T, SH, NT>;
    RX_LAUNCH(k, dim3(maxs, njobs), threads, rx_smem<T>(p.sh.n1, p.sh.n2, 2 * p.sh.Q2 * p.sh.HP), st, jobs, sh,
              p.tb[prec_of<T>()]);
    return 1;
}

template <typename T> int rx2_stress(const RxPlan &p, cudaStream_t st, const StressJob<T> *jobs, int njobs, int maxs)
{
    const RxShape &s = p.sh;
    if (!p.plane || rx_smem<T>(s.n1, s.n2, 2 * s.Q2 * s.HP) > SMEM_MOST - 1024) return 0;
    if (s.n1 == 64 && s.n2 == 64) return stress2<T, RxFixed<64, 64, 8, 8>, 288>(p, {}, 288, st, jobs, njobs, maxs);
    return stress2<T, RxShape, RX_NT>(p, s, rx_threads(std::max(s.Q2 * s.n1h, s.P2 * s.n1h)), st, jobs, njobs, maxs);
}

// ---------------------------------------------------------------------
// dim 3
// ---------------------------------------------------------------------
template <typename T> static size_t fp_bytes(const RxShape &s, int ppc) { return rx_smem<T>(s.n1, s.n2, ppc * s.n2); }
template <typename T> static size_t rp_bytes(const RxShape &s, int ppc) { return rx_smem<T>(s.n1, s.n2, ppc * s.Q2 * s.HP); }

template <typename T> bool rx3_fits(const RxPlan &p)
{
    return p.plane && p.line && fp_bytes<T>(p.sh, 1) <= SMEM_MOST;
}

// f(shape, RxInt<threads of FP kernels>, RxInt<their CTAs per SM>, RxInt<threads of k3v_mid>, RxInt<CTAs per SM>)
// for launches of `ctas` CTAs: with at most one per SM each gets twice the
// threads.  FP32 values take half the registers: more CTAs per SM.
template <typename T, typename F> static int with_plane(const RxPlan &p, int ctas, F f)
{
    constexpr bool F32 = sizeof(T) == 4;
    const int a = p.sh.n1, b = p.sh.n2;
    if (a == 64 && b == 128)
        return f(RxFixed<64, 128, 8, 8>(), RxInt<F32 ? 288 : 544>(), RxInt<F32 ? 3 : 1>(), RxInt<288>(), RxInt<F32 ? 4 : 2>());
    if (a == 32 && b == 32) return f(RxFixed<32, 32, 4, 4>(), RxInt<288>(), RxInt<3>(), RxInt<288>(), RxInt<3>());
    if (a == 64 && b == 64) {
        using S = RxFixed<64, 64, 8, 8>;
        if (ctas <= RX_SMS) return f(S(), RxInt<544>(), RxInt<1>(), RxInt<288>(), RxInt<2>());
        return f(S(), RxInt<288>(), RxInt<F32 ? 3 : 2>(), RxInt<288>(), RxInt<F32 ? 4 : 2>());
    }
    auto go = [&](auto sh) {
        if (ctas <= RX_SMS) return f(sh, RxInt<544>(), RxInt<1>(), RxInt<RX_NT>(), RxInt<2>());
        return f(sh, RxInt<RX_NT>(), RxInt<2>(), RxInt<RX_NT>(), RxInt<2>());
    };
    return small10(p.sh) ? go(RxShape10{p.sh}) : go(p.sh);
}
// f(shape, RxInt<columns of a tile>, RxInt<threads>, RxInt<CTAs per SM of the
// filter pass>), for nf spectra: half as wide where the wide tiles would
// leave SMs idle.  Threads / columns is at least P and Q.
template <typename T, typename F> static int with_line(const RxPlan &p, int nf, F f)
{
    constexpr bool F32 = sizeof(T) == 4;
    const bool narrow = (long)p.sh.n1h * p.sh.n2 * nf < 32L * 2 * RX_SMS;
    switch (p.z.n3) {
    case 32:
        if (narrow) return f(RzFixed<32, 8>(), RxInt<8>(), RxInt<64>(), RxInt<8>());
        return f(RzFixed<32, 8>(), RxInt<32>(), RxInt<256>(), RxInt<4>());
    case 64:
        if (narrow) return f(RzFixed<64, 8>(), RxInt<16>(), RxInt<128>(), RxInt<4>());
        return f(RzFixed<64, 8>(), RxInt<32>(), RxInt<256>(), RxInt<F32 ? 4 : 2>());
    case 224: return f(RzFixed<224, 16>(), RxInt<16>(), RxInt<256>(), RxInt<F32 ? 3 : 2>());
    default: break;
    }
    const int q = std::max(p.z.P, p.z.Q);
    if (q <= 8 && narrow) return f(RzShape10{p.z}, RxInt<16>(), RxInt<128>(), RxInt<4>());
    if (q <= 8) return f(RzShape10{p.z}, RxInt<32>(), RxInt<256>(), RxInt<3>());
    if (q <= 10) return f(RzShape10{p.z}, RxInt<16>(), RxInt<160>(), RxInt<4>());
    return f(p.z, RxInt<16>(), RxInt<256>(), RxInt<2>());
}

// The same for the stress pass, which holds two tiles: 8 columns where tiles of
// 16 would leave one CTA to an SM (a 64 x 128 x 224 FP64 solve's z pass: 8.2 ms
// with 16, 6.0 with 8).
template <typename T, typename F> static int with_stress_line(const RxPlan &p, F f)
{
    if (2 * rz_smem<T>(p.n3, 16, 2) > SMEM_MOST) {
        if (p.z.n3 == 224) return f(RzFixed<224, 16>(), RxInt<8>(), RxInt<128>(), RxInt<3>());
        return f(p.z, RxInt<8>(), RxInt<128>(), RxInt<3>());
    }
    return with_line<T>(p, 1 << 20, f);
}

template <typename T> static int fp_threads(const RxShape &s, int ppc, int most)
{
    return rx_threads(std::max({ppc * s.n2 * s.Q1, ppc * s.Q2 * s.n1h, ppc * 2 * s.P2 * s.n1h}), most);
}

template <typename T> int rx3_planes(const RxPlan &p, int nf)
{
    return rx_ppc(p.sh.n2 * p.sh.Q1, p.n3, nf, fp_bytes<T>(p.sh, 1));
}

template <typename T> static int rx3_ctas(const RxPlan &p, int nf)
{
    const int ppc = rx3_planes<T>(p, nf);
    return (p.n3 + ppc - 1) / ppc * nf;
}

template <typename T> int rx3_first(const RxPlan &p, cudaStream_t st, const SweepField<T> *f, int nf, int t)
{
    if (!rx3_fits<T>(p)) return 0;
    return with_plane<T>(p, rx3_ctas<T>(p, nf), [&](auto sh, auto nt, auto mb, auto, auto) {
        const int ppc = rx3_planes<T>(p, nf);
        auto *k = k3v_fwd<T, decltype(sh), decltype(nt)::value, decltype(mb)::value>;
        RX_LAUNCH(k, dim3((p.n3 + ppc - 1) / ppc, nf), fp_threads<T>(p.sh, ppc, decltype(nt)::value), fp_bytes<T>(p.sh, ppc),
                  st, f, sh, p.tb[prec_of<T>()], p.n3, ppc, t);
        return 1;
    });
}

template <typename T> static int zconv(const RxPlan &p, cudaStream_t st, const SweepField<T> *f, int nf, int t, int which)
{
    return with_line<T>(p, nf * (which == 3 ? 2 : 1), [&](auto z, auto tc, auto nt, auto mb) {
        constexpr int TC = decltype(tc)::value, NT = decltype(nt)::value;
        auto *k = k3v_zconv<T, decltype(z), TC, NT, decltype(mb)::value>;
        RX_LAUNCH(k, dim3((p.sh.n1h * p.sh.n2 + TC - 1) / TC, nf, which == 3 ? 2 : 1), NT, rz_smem<T>(p.n3, TC, 1), st, f, z,
                  p.zc[prec_of<T>()], t, which);
        return 1;
    });
}

template <typename T> int rx3_half(const RxPlan &p, cudaStream_t st, const SweepField<T> *f, int nf)
{
    if (!rx3_fits<T>(p)) return 0;
    if (zconv<T>(p, st, f, nf, 0, 3) < 0) return -1;
    const int rc = with_plane<T>(p, rx3_ctas<T>(p, nf), [&](auto sh, auto nt, auto mb, auto, auto) {
        const int ppc = rx3_planes<T>(p, nf);
        auto *k = k3v_half<T, decltype(sh), decltype(nt)::value, decltype(mb)::value>;
        RX_LAUNCH(k, dim3((p.n3 + ppc - 1) / ppc, nf), fp_threads<T>(p.sh, ppc, decltype(nt)::value), fp_bytes<T>(p.sh, ppc),
                  st, f, sh, p.tb[prec_of<T>()], p.n3, ppc);
        return 1;
    });
    return rc < 0 ? -1 : 2;
}

template <typename T> int rx3_step(const RxPlan &p, cudaStream_t st, const SweepField<T> *f, int nf, int t)
{
    if (!rx3_fits<T>(p)) return 0;
    if (zconv<T>(p, st, f, nf, t, 3) < 0) return -1;
    int rc = with_plane<T>(p, 1 << 30, [&](auto sh, auto, auto, auto nt, auto mb) {
        const RxShape &s = p.sh;
        const int npair = s.Q2 * s.HP;
        const int ppc = rx_ppc(npair * s.Q1, p.n3, nf, rp_bytes<T>(s, 1));
        const int thr = rx_threads(std::max({ppc * npair * s.Q1, ppc * s.Q2 * s.n1h, ppc * s.P2 * s.n1h}), decltype(nt)::value);
        auto *k = k3v_mid<T, decltype(sh), decltype(nt)::value, decltype(mb)::value>;
        RX_LAUNCH(k, dim3((p.n3 + ppc - 1) / ppc, nf), thr, rp_bytes<T>(s, ppc), st, f, sh, p.tb[prec_of<T>()], p.n3, ppc, t);
        return 1;
    });
    if (rc < 0 || zconv<T>(p, st, f, nf, t, 2) < 0) return -1;
    rc = with_plane<T>(p, rx3_ctas<T>(p, nf), [&](auto sh, auto nt, auto mb, auto, auto) {
        const int ppc = rx3_planes<T>(p, nf);
        auto *k = k3v_final<T, decltype(sh), decltype(nt)::value, decltype(mb)::value>;
        RX_LAUNCH(k, dim3((p.n3 + ppc - 1) / ppc, nf), fp_threads<T>(p.sh, ppc, decltype(nt)::value), fp_bytes<T>(p.sh, ppc),
                  st, f, sh, p.tb[prec_of<T>()], p.n3, ppc, t);
        return 1;
    });
    return rc < 0 ? -1 : 4;
}

// (two tiles of a line have to fit)
template <typename T> int rx3_stress_tiles(const RxPlan &p)
{
    if (!rx3_fits<T>(p)) return 0;
    return with_stress_line<T>(p, [&](auto, auto tc, auto, auto) {
        constexpr int TC = decltype(tc)::value;
        return rz_smem<T>(p.n3, TC, 2) <= SMEM_MOST - 1024 ? (p.sh.n1h * p.sh.n2 + TC - 1) / TC : 0;
    });
}

template <typename T>
int rx3_stress(const RxPlan &p, cudaStream_t st, const StressJob<T> *jobs, int njobs, int s0, int cnt, int cs, cx<T> *spec,
               double *part)
{
    if (rx3_stress_tiles<T>(p) == 0) return 0;
    const int rc = with_plane<T>(p, 1 << 30, [&](auto sh, auto, auto, auto nt, auto mb) {
        const RxShape &s = p.sh;
        const int npair = s.Q2 * s.HP;
        const int ppc = rx_ppc(npair * s.Q1, p.n3, 2 * cnt * njobs, rp_bytes<T>(s, 1));
        const int thr = rx_threads(std::max({ppc * npair * s.Q1, ppc * s.Q2 * s.n1h, ppc * s.P2 * s.n1h}), decltype(nt)::value);
        auto *k = k3v_stress_xy<T, decltype(sh), decltype(nt)::value, decltype(mb)::value>;
        RX_LAUNCH(k, dim3((p.n3 + ppc - 1) / ppc, cnt, 2 * njobs), thr, rp_bytes<T>(s, ppc), st, jobs, sh, p.tb[prec_of<T>()],
                  p.n3, ppc, s0, cs, spec);
        return 1;
    });
    if (rc < 0) return -1;
    return with_stress_line<T>(p, [&](auto z, auto tc, auto nt, auto) {
        constexpr int TC = decltype(tc)::value, NT = decltype(nt)::value;
        auto *k = k3v_stress_z<T, decltype(z), TC, NT>;
        RX_LAUNCH(k, dim3((p.sh.n1h * p.sh.n2 + TC - 1) / TC, cnt, njobs), NT, rz_smem<T>(p.n3, TC, 2), st, jobs, z,
                  p.zc[prec_of<T>()], s0, cs, (const cx<T> *)spec, part);
        return 2;
    });
}

#define RX2_INSTANCES(T)                                                                                             \
    template int rx2_sweep<T>(const RxPlan &, cudaStream_t, const SweepField<T> *, int, int, int);                   \
    template int rx2_stress<T>(const RxPlan &, cudaStream_t, const StressJob<T> *, int, int);
#define RX3_INSTANCES(T)                                                                                             \
    template int rx3_planes<T>(const RxPlan &, int);                                                                 \
    template bool rx3_fits<T>(const RxPlan &);                                                                       \
    template int rx3_first<T>(const RxPlan &, cudaStream_t, const SweepField<T> *, int, int);                        \
    template int rx3_step<T>(const RxPlan &, cudaStream_t, const SweepField<T> *, int, int);                         \
    template int rx3_stress_tiles<T>(const RxPlan &);                                                                \
    template int rx3_stress<T>(const RxPlan &, cudaStream_t, const StressJob<T> *, int, int, int, int, cx<T> *, double *);

}  // namespace pscfg
