// plane_rx.cuh -- plane and z-line transforms with the line passes in
// registers and one shared-memory exchange per pass.
//
// A line of length N = P Q is transformed as P-point transforms of the
// samples n = Q i + r (fixed r), a twiddle, an exchange, and Q-point
// transforms (n = Q i + r, k = k1 + P k2); the inverse runs backwards.  Each
// pass holds its P or Q values in registers (radices up to 16, kernels
// dispatch on them at run time, or the whole shape is a template constant),
// reads and writes only its own slots, so one buffer and one barrier per
// exchange suffice, and whatever precedes the first or follows the last pass
// of a plane (pointwise products, k-space filters, global loads and stores)
// happens on the values in registers.
//
// Two real rows share one complex line z = a + i b, so a plane needs no
// half-length trick: the column pass that follows forms
//   2 A(k) = Z(k) + conj Z(n1 - k),   2 B(k) = -i (Z(k) - conj Z(n1 - k))
// from the two slots it reads anyway.  (Spectra are therefore twice the
// transform; the normalisation takes the factor.)  Either
//   FP  a, b = the same row of two fields (two filters of one step), or
//   RP  a, b = two rows of one column residue class, y0 = 2 j Q2 + r and
//       y0 + Q2, of one field.
// A column c of the half spectrum has the slots pos (kx) and wpos (n1 - kx,
// or one of two spare slots for the real columns kx = 0 and n1/2) of every
// line, one for A and one for B.
//
// Columns are numbered by the order in which the row transform leaves them
// (kx = k1 + P1 k2, k2 fastest, kx = n1/2 last), so that consecutive threads
// meet consecutive slots; the spectra in global memory are [z][ky][c].
#pragma once
#include "fft_ct.cuh"
#include "scf_kernels.cuh"

namespace pscfg {

// ---------------------------------------------------------------------
// Codelets: prime-factor (no twiddles) lengths, and 9 = 3 x 3
// ---------------------------------------------------------------------
template <int P, int Q, int S, typename T> struct DftPfa {
    __device__ __forceinline__ static void run(cx<T> *v)
    {
        constexpr int N = P * Q;
        cx<T> y[P][Q];
#pragma unroll
        for (int a = 0; a < P; a++) {
#pragma unroll
            for (int b = 0; b < Q; b++) y[a][b] = v[(Q * a + P * b) % N];
            Dft<Q, S, T>::run(y[a]);
        }
#pragma unroll
        for (int b = 0; b < Q; b++) {
            cx<T> t[P];
#pragma unroll
            for (int a = 0; a < P; a++) t[a] = y[a][b];
            Dft<P, S, T>::run(t);
#pragma unroll
            for (int a = 0; a < P; a++) y[a][b] = t[a];
        }
#pragma unroll
        for (int k = 0; k < N; k++) v[k] = y[k % P][k % Q];
    }
};
template <int S, typename T> struct Dft<6, S, T> : DftPfa<2, 3, S, T> {};
template <int S, typename T> struct Dft<10, S, T> : DftPfa<2, 5, S, T> {};
template <int S, typename T> struct Dft<12, S, T> : DftPfa<4, 3, S, T> {};
template <int S, typename T> struct Dft<15, S, T> : DftPfa<3, 5, S, T> {};
template <int S, typename T> struct Dft<9, S, T> {
    __device__ __forceinline__ static void run(cx<T> *v)
    {
        // cos, sin of 2 pi m / 9, m = 1, 2, 4
        const T c1 = (T)0.766044443118978035202392650555416673, s1 = (T)0.642787609686539326322643409907263433;
        const T c2 = (T)0.173648177666930348851716626769314796, s2 = (T)0.984807753012208059366743024589523014;
        const T c4 = (T)-0.939692620785908384054109277324731470, s4 = (T)0.342020143325668733044099614682259580;
        cx<T> y[3][3];
#pragma unroll
        for (int b = 0; b < 3; b++) {
            cx<T> t[3] = {v[b], v[3 + b], v[6 + b]};
            Dft<3, S, T>::run(t);
            y[0][b] = t[0];
            y[1][b] = t[1];
            y[2][b] = t[2];
        }
        y[1][1] = cmul(y[1][1], mk<T>(c1, (T)S * s1));
        y[1][2] = cmul(y[1][2], mk<T>(c2, (T)S * s2));
        y[2][1] = cmul(y[2][1], mk<T>(c2, (T)S * s2));
        y[2][2] = cmul(y[2][2], mk<T>(c4, (T)S * s4));
#pragma unroll
        for (int a = 0; a < 3; a++) {
            Dft<3, S, T>::run(y[a]);
#pragma unroll
            for (int k = 0; k < 3; k++) v[a + 3 * k] = y[a][k];
        }
    }
};

// x / d by the reciprocal r = 1 / d with one residual correction (Markstein,
// IBM J. Res. Dev. 34, 1990): a plain product with a rounded 1/3 or 1/N is
// off by the same fraction of an ulp in every step of a contour.  Finite x: the
// quotient x / d to the last bit.  Infinite x: NaN, as the transforms that
// follow make of it (a check costs 2% of a 64 x 64 sweep).
template <typename T> __host__ __device__ __forceinline__ T div_by(T x, T d, T r)
{
    const T q = x * r;
    return fma(fma(-d, q, x), r, q);
}

// ---------------------------------------------------------------------
// Shapes
// ---------------------------------------------------------------------
// floor(w / d) by a multiplication with ceil(2^32 / d), w < 2^16
struct RDiv {
    unsigned d, m;
    __host__ __device__ static RDiv of(int d) { return RDiv{(unsigned)d, d > 1 ? 0xffffffffu / (unsigned)d + 1u : 0u}; }
    __device__ __forceinline__ int div(int w) const { return m ? (int)__umulhi((unsigned)w, m) : w; }
    __device__ __forceinline__ int mod(int w) const { return w - (int)d * div(w); }
};
template <int D> struct SDiv {
    __device__ __forceinline__ static int div(int w) { return w / D; }
    __device__ __forceinline__ static int mod(int w) { return w % D; }
};

// A column of the half spectrum: its kx, its slot, the slot of n1 - kx and
// the slot that holds B.
struct RxCol {
    short kx, pos, ppos, wpos;
};

// Rotation of the slots of a k1 group: with 8 values in a group only half
// of them (kx <= n1/2) are columns, so some groups start at the other half
// and together fill the banks: 8 values of 16 bytes (every other group) or
// 16 of 8 (every other two).
template <typename T> __host__ __device__ __forceinline__ constexpr int rx_rot(int Q1, int k1)
{
    return Q1 == 8 ? 4 * ((sizeof(T) == 8 ? k1 : k1 >> 1) & 1) : 0;
}
template <typename T> __host__ __device__ __forceinline__ constexpr int rx_slot(int Q1, int k1, int k2)
{
    return Q1 * k1 + (k2 + rx_rot<T>(Q1, k1)) % Q1;
}
// Line of the row passes' l-th group of Q1 = 8 items.  An 8-byte half warp
// holds two groups, whose lines must lie 8 units apart on the 16 bank pairs:
// lines j and j + 8 at an odd stride (fixed shapes: whole blocks of 16 lines).
template <typename T, typename SH> __device__ __forceinline__ int rx_line(int l)
{
    if constexpr (SH::FIXED && sizeof(T) == 4) return (l & ~15) | ((l & 1) << 3) | ((l >> 1) & 7);
    else return l;
}
// line stride in complex values: n1 slots, two spare ones, odd
__host__ __device__ __forceinline__ constexpr int rx_stride(int n1) { return (n1 + 2) | 1; }

// run-time plane shape; PM, QM: the largest radices a kernel is compiled for
// (a kernel takes the registers of its largest radix; lines up to 64 points
// do with 8 and 10)
struct RxShape {
    static constexpr bool FIXED = false;
    static constexpr int PM = 10, QM = 16;
    int n1, n2, n1h, nc, P1, Q1, P2, Q2, HP, LS;   // nc: columns without kx = n1/2
    RDiv dQ1, dn1h, dnc, dQ2, dP2;
};
struct RxShape10 : RxShape {
    static constexpr int PM = 8, QM = 10;
};
// compile-time plane shape
template <int N1, int N2, int P1_, int P2_> struct RxFixed {
    static constexpr bool FIXED = true;
    static constexpr int n1 = N1, n2 = N2, n1h = N1 / 2 + 1, nc = (N1 + 1) / 2, P1 = P1_, Q1 = N1 / P1_, P2 = P2_, Q2 = N2 / P2_,
                         HP = (P2_ + 1) / 2, LS = rx_stride(N1);
    SDiv<N1 / P1_> dQ1;
    SDiv<N1 / 2 + 1> dn1h;
    SDiv<(N1 + 1) / 2> dnc;
    SDiv<N2 / P2_> dQ2;
    SDiv<P2_> dP2;
};

// Column c of a fixed shape (even Q1: every k1 group holds Q1 / 2 columns, kx
// = n1/2 follows them), as in the run-time shapes' tables.
template <typename T, typename SH> __device__ __forceinline__ RxCol rx_fixed_col(int c)
{
    constexpr int P = SH::P1, Q = SH::Q1, H = Q / 2;
    static_assert(Q % 2 == 0, "columns in whole groups");
    const int k1 = c == SH::nc ? 0 : c / H, k2 = c == SH::nc ? H : c % H;
    const int q1 = k1 ? P - k1 : 0, q2 = k1 ? Q - 1 - k2 : (Q - k2) % Q;
    RxCol r;
    r.kx = (short)(k1 + P * k2);
    r.pos = (short)rx_slot<T>(Q, k1, k2);
    r.ppos = (short)rx_slot<T>(Q, q1, q2);
    r.wpos = c == 0 ? (short)SH::n1 : c == SH::nc ? (short)(SH::n1 + 1) : r.ppos;
    return r;
}

template <int V> struct RxInt {
    static constexpr int value = V;
};
// f(RxInt<radix>) for the first radix of a line (1..10, rows also 12..16
// through rx_q) or the second
template <int PM, typename F> __device__ __forceinline__ void rx_p(int r, F f)
{
    if constexpr (PM > 8) {
        if (r == 9) return f(RxInt<9>());
        if (r == 10) return f(RxInt<10>());
    }
    switch (r) {
    case 1: f(RxInt<1>()); break;
    case 2: f(RxInt<2>()); break;
    case 3: f(RxInt<3>()); break;
    case 4: f(RxInt<4>()); break;
    case 5: f(RxInt<5>()); break;
    case 6: f(RxInt<6>()); break;
    case 7: f(RxInt<7>()); break;
    case 8: f(RxInt<8>()); break;
    default: break;
    }
}
template <int QM, typename F> __device__ __forceinline__ void rx_q(int r, F f)
{
    if constexpr (QM > 10) {
        switch (r) {
        case 12: f(RxInt<12>()); return;
        case 14: f(RxInt<14>()); return;
        case 15: f(RxInt<15>()); return;
        case 16: f(RxInt<16>()); return;
        default: break;
        }
    }
    rx_p<10>(r, f);
}
#define RX_P(SH, r, F)                                             \
    do {                                                           \
        if constexpr (SH::FIXED) F(RxInt<SH::r>()); else rx_p<SH::PM>(sh.r, F); \
    } while (0)
#define RX_Q(SH, r, F)                                             \
    do {                                                           \
        if constexpr (SH::FIXED) F(RxInt<SH::r>()); else rx_q<SH::QM>(sh.r, F); \
    } while (0)

// ---------------------------------------------------------------------
// Passes.  buf: [line][LS]; in shared memory tw1[Q1 k + r] = W_n1^(r k)
// (consecutive threads take consecutive r: W_n1^m itself would meet 4-way
// bank conflicts) and tw2[m] = W_n2^m (one r for a whole warp, mostly).
// None of them synchronises.
// ---------------------------------------------------------------------
template <typename T, typename SH> struct Rx {
    using C = cx<T>;

    // rows, first pass of the forward transform on values in registers:
    // v[i] = z(Q1 i + r) of the line at b; leaves them in the line's slots
    template <int P>
    __device__ __forceinline__ static void row_fwd1(const SH &sh, C *b, int r, C *v, const C *tw1)
    {
        Dft<P, -1, T>::run(v);
        b[r] = v[0];
#pragma unroll
        for (int k = 1; k < P; k++) b[sh.Q1 * k + r] = cmul(v[k], tw1[sh.Q1 * k + r]);
    }
    // rows, last pass of the inverse: v[i] = z(Q1 i + r)
    template <int P>
    __device__ __forceinline__ static void row_inv1(const SH &sh, const C *b, int r, C *v, const C *tw1)
    {
        v[0] = b[r];
#pragma unroll
        for (int k = 1; k < P; k++) v[k] = cmul(b[sh.Q1 * k + r], conjg(tw1[sh.Q1 * k + r]));
        Dft<P, 1, T>::run(v);
    }
    // rows, second forward (S < 0) or first inverse pass of nl lines,
    // consecutive threads on consecutive lines; line(j) is the buffer line
    template <int S, typename L>
    __device__ __forceinline__ static void rows2(const SH &sh, C *buf, int nl, RDiv dnl, L line)
    {
        auto go = [&](auto qc) {
            constexpr int Q = decltype(qc)::value;
            for (int w = threadIdx.x; w < nl * sh.P1; w += blockDim.x) {
                const int k1 = dnl.div(w), l = w - nl * k1;
                C *b = buf + line(l) * sh.LS + Q * k1;
                const int rot = rx_rot<T>(Q, k1);   // Q = 8: slot of k2 is k2 ^ rot
                C v[Q];
                if (S < 0) {
#pragma unroll
                    for (int j = 0; j < Q; j++) v[j] = b[j];
                    Dft<Q, S, T>::run(v);
#pragma unroll
                    for (int k = 0; k < Q; k++) b[Q == 8 ? (k < 4 ? k + rot : k - rot) : k] = v[k];
                } else {
#pragma unroll
                    for (int k = 0; k < Q; k++) v[k] = b[Q == 8 ? (k < 4 ? k + rot : k - rot) : k];
                    Dft<Q, S, T>::run(v);
#pragma unroll
                    for (int j = 0; j < Q; j++) b[j] = v[j];
                }
            }
        };
        RX_Q(SH, Q1, go);
    }

    // Item w of a column pass over nt groups -> (group t, column c): the nc
    // columns of every group first (for powers of two whole warps on one
    // group, aligned to the banks), then the column kx = n1/2 of each.
    __device__ __forceinline__ static void col_item(const SH &sh, int w, int nt, int &t, int &c)
    {
        if (w < nt * sh.nc) {
            t = sh.dnc.div(w);
            c = w - sh.nc * t;
        } else {
            t = w - nt * sh.nc;
            c = sh.nc;
        }
    }

    __device__ __forceinline__ static RxCol column(const RxCol *ct, int c)
    {
        if constexpr (SH::FIXED) return rx_fixed_col<T, SH>(c);
        else return ct[c];
    }

    __device__ __forceinline__ static C sumc(C z, C zp) { return mk<T>(z.x + zp.x, z.y - zp.y); }    // z + conj zp
    __device__ __forceinline__ static C difc(C z, C zp) { return mk<T>(z.y + zp.y, zp.x - z.x); }    // -i (z - conj zp)

    // columns, first forward pass of np planes.  FP: lines y of a plane;
    // RP: line(r, j) holds the rows r + 2 j Q2 and r + (2 j + 1) Q2, at
    // r + j Q2 LSTEP, ld lines per plane.
    template <bool FP, int LSTEP>
    __device__ __forceinline__ static void cols_fwd1(const SH &sh, C *buf, int np, int ld, const RxCol *ct, const C *tw2)
    {
        auto go = [&](auto pc) {
            constexpr int P = decltype(pc)::value;
            for (int w = threadIdx.x; w < np * sh.Q2 * sh.n1h; w += blockDim.x) {
                int t, c;
                col_item(sh, w, np * sh.Q2, t, c);
                const int pl = sh.dQ2.div(t), r = t - sh.Q2 * pl;
                const RxCol col = column(ct, c);
                C *b = buf + (pl * ld + r) * sh.LS;
                if constexpr (FP) {
                    C a[P], d[P];
#pragma unroll
                    for (int i = 0; i < P; i++) {
                        const C z = b[sh.Q2 * i * sh.LS + col.pos], zp = b[sh.Q2 * i * sh.LS + col.ppos];
                        a[i] = sumc(z, zp);
                        d[i] = difc(z, zp);
                    }
                    Dft<P, -1, T>::run(a);
                    b[col.pos] = a[0];
#pragma unroll
                    for (int k = 1; k < P; k++) b[sh.Q2 * k * sh.LS + col.pos] = cmul(a[k], tw2[r * k]);
                    Dft<P, -1, T>::run(d);
                    b[col.wpos] = d[0];
#pragma unroll
                    for (int k = 1; k < P; k++) b[sh.Q2 * k * sh.LS + col.wpos] = cmul(d[k], tw2[r * k]);
                } else {
                    constexpr int H = (P + 1) / 2;
                    C a[2 * H];
#pragma unroll
                    for (int j = 0; j < H; j++) {
                        const C z = b[sh.Q2 * LSTEP * j * sh.LS + col.pos], zp = b[sh.Q2 * LSTEP * j * sh.LS + col.ppos];
                        a[2 * j] = sumc(z, zp);
                        a[2 * j + 1] = difc(z, zp);
                    }
                    Dft<P, -1, T>::run(a);
#pragma unroll
                    for (int k = 0; k < P; k++)
                        b[sh.Q2 * LSTEP * (k / 2) * sh.LS + ((k & 1) ? col.wpos : col.pos)] = k ? cmul(a[k], tw2[r * k]) : a[k];
                }
            }
        };
        RX_P(SH, P2, go);
    }

    // columns, last inverse pass: back to the lines z = a + i b
    template <bool FP, int LSTEP>
    __device__ __forceinline__ static void cols_inv1(const SH &sh, C *buf, int np, int ld, const RxCol *ct, const C *tw2)
    {
        auto go = [&](auto pc) {
            constexpr int P = decltype(pc)::value;
            for (int w = threadIdx.x; w < np * sh.Q2 * sh.n1h; w += blockDim.x) {
                int t, c;
                col_item(sh, w, np * sh.Q2, t, c);
                const int pl = sh.dQ2.div(t), r = t - sh.Q2 * pl;
                const RxCol col = column(ct, c);
                const bool real = col.pos == col.ppos;   // kx = 0 or n1/2: the rows' spectra are real there
                C *b = buf + (pl * ld + r) * sh.LS;
                auto put = [&](C *s, C a, C d) {
                    if (real) {
                        s[col.pos] = mk<T>(a.x, d.x);
                    } else {
                        s[col.pos] = mk<T>(a.x - d.y, a.y + d.x);    // a + i d
                        s[col.ppos] = mk<T>(a.x + d.y, d.x - a.y);   // conj a + i conj d
                    }
                };
                if constexpr (FP) {
                    C a[P], d[P];
#pragma unroll
                    for (int k = 0; k < P; k++) {
                        const C u = b[sh.Q2 * k * sh.LS + col.pos], v = b[sh.Q2 * k * sh.LS + col.wpos];
                        if (k) {
                            const C w1 = conjg(tw2[r * k]);
                            a[k] = cmul(u, w1);
                            d[k] = cmul(v, w1);
                        } else {
                            a[k] = u;
                            d[k] = v;
                        }
                    }
                    Dft<P, 1, T>::run(a);
                    Dft<P, 1, T>::run(d);
#pragma unroll
                    for (int i = 0; i < P; i++) put(b + sh.Q2 * i * sh.LS, a[i], d[i]);
                } else {
                    constexpr int H = (P + 1) / 2;
                    C a[2 * H];
                    if (P & 1) a[2 * H - 1] = mk<T>((T)0, (T)0);
#pragma unroll
                    for (int k = 0; k < P; k++) {
                        const C u = b[sh.Q2 * LSTEP * (k / 2) * sh.LS + ((k & 1) ? col.wpos : col.pos)];
                        a[k] = k ? cmul(u, conjg(tw2[r * k])) : u;
                    }
                    Dft<P, 1, T>::run(a);
#pragma unroll
                    for (int j = 0; j < H; j++) put(b + sh.Q2 * LSTEP * j * sh.LS, a[2 * j], a[2 * j + 1]);
                }
            }
        };
        RX_P(SH, P2, go);
    }

    // columns, the Q2-point pass: f(column, ab, plane, k1, slots, v) with
    // v[k2] <-> ky = k1 + P2 k2.  The callers read or write v and the slots
    // s[n * Q] (n < Q2) as their direction needs.
    template <bool FP, int LSTEP, typename F>
    __device__ __forceinline__ static void cols2(const SH &sh, C *buf, int np, int ld, const RxCol *ct, F f)
    {
        auto go = [&](auto qc) {
            constexpr int Q = decltype(qc)::value;
            const int ng = (FP ? 2 : 1) * np * sh.P2;
            for (int w = threadIdx.x; w < ng * sh.n1h; w += blockDim.x) {
                int t, c;
                col_item(sh, w, ng, t, c);
                const int u = sh.dP2.div(t), k1 = t - sh.P2 * u;
                const int ab = FP ? (u & 1) : 0, pl = FP ? (u >> 1) : u;
                const RxCol col = column(ct, c);
                // FP: lines Q2 k1 + n; RP: lines (k1 / 2) Q2 LSTEP + n
                C *s = buf + (pl * ld + (FP ? Q * k1 : Q * LSTEP * (k1 / 2))) * sh.LS +
                       ((FP ? ab : (k1 & 1)) ? col.wpos : col.pos);
                C v[Q];
                f(RxInt<Q>(), c, (int)col.kx, ab, pl, k1, s, v);
            }
        };
        RX_Q(SH, Q2, go);
    }
};

// ---------------------------------------------------------------------
// Shared memory of a plane kernel: buffer, twiddles, column table
// ---------------------------------------------------------------------
struct RxTables {
    const void *tw1, *tw2;   // cx<T>[n1], cx<T>[n2]
    const RxCol *cols;       // [n1h]
};

template <typename T> __host__ __device__ constexpr size_t rx_smem(int n1, int n2, int lines)
{
    return sizeof(cx<T>) * ((size_t)lines * rx_stride(n1) + n1 + n2) + sizeof(RxCol) * (n1 / 2 + 1);
}

template <typename T, typename SH> struct RxMem {
    cx<T> *buf, *tw1, *tw2;
    RxCol *ct;
    // copies the tables in; the first barrier of the transform covers them
    // for all passes but the first, whose callers synchronise
    __device__ __forceinline__ RxMem(const SH &sh, const RxTables &tb, int lines)
    {
        extern __shared__ __align__(16) unsigned char smem_raw[];
        buf = (cx<T> *)smem_raw;
        tw1 = buf + lines * sh.LS;
        tw2 = tw1 + sh.n1;
        ct = (RxCol *)(tw2 + sh.n2);
        for (int i = threadIdx.x; i < sh.n1; i += blockDim.x) {
            const int k = sh.dQ1.div(i);
            tw1[i] = ((const cx<T> *)tb.tw1)[k * (i - sh.Q1 * k)];
        }
        for (int i = threadIdx.x; i < sh.n2; i += blockDim.x) tw2[i] = ((const cx<T> *)tb.tw2)[i];
        for (int i = threadIdx.x; i < sh.n1h; i += blockDim.x) ct[i] = tb.cols[i];
    }
    __device__ __forceinline__ void *end(const SH &sh) const { return ct + sh.n1h; }
};

// Row stride of a real plane in shared memory: 8 (mod 16) values, so that the
// two rows of a half warp lie on different banks.
__host__ __device__ __forceinline__ constexpr int rx2_stride(int n1) { return n1 + (24 - n1 % 16) % 16; }
// ---------------------------------------------------------------------
// dim 2: a field's whole sweep in one CTA.  Per step one FP transform pair
// (a = exp(-w ds/4) q with the filter ek2, b = exp(-w ds/2) q with ek1) and
// one RP pair (the second half step), the filter applied between the two
// column passes in registers: 12 barriers.  q and q1 share one real plane
// (a slot's thread reads q there before it writes q1, and q1 before q).
// Bound: the chain of barriers and shared-memory exchanges (6 reads and
// writes of the plane per transform pair); FP64 issue where two fields share
// an SM.
// grid = nfields.
// ---------------------------------------------------------------------
// TAB: the current block's tables (exp(-w ds/4), and both filters in column
// order) sit in shared memory too: for launches of at most one CTA per SM.
template <typename T> __host__ __device__ constexpr size_t rx2_smem(int n1, int n2, bool tab)
{
    return (rx_smem<T>(n1, n2, n2) + 15) / 16 * 16 +
           sizeof(T) * ((size_t)rx2_stride(n1) * n2 * (tab ? 2 : 1) + (tab ? 2 * (n1 / 2 + 1) * n2 : 0));
}

template <typename T, typename SH, int NT, int MB, bool TAB>
__global__ void __launch_bounds__(NT, MB)
    k2x_sweep(const SweepField<T> *fields, SH sh, RxTables tb, int t0, int t1)
{
    using X = Rx<T, SH>;
    using C = cx<T>;
    const SweepField<T> &f = fields[blockIdx.x];
    const RxMem<T, SH> m(sh, tb, sh.n2);
    T *q = (T *)(((size_t)m.end(sh) + 15) / 16 * 16);   // (shared addresses are 16-byte aligned at the buffer)
    const int nr = sh.n1 * sh.n2, nkc = sh.n1h * sh.n2;
    const int QS = rx2_stride(sh.n1);
    T *te2 = q + QS * sh.n2, *tek = te2 + QS * sh.n2;   // (TAB)
    const T rn = (T)(2.0 * nr), rr = (T)(1.0 / (2.0 * nr)), rt = (T)(1.0 / 3.0);
    const int npair = sh.Q2 * sh.HP;
    const RDiv dpair = RDiv::of(npair), dn2 = RDiv::of(sh.n2);
    auto pair_line = [&](int l) { const int j = sh.dQ2.div(l); return l - sh.Q2 * j + 2 * sh.Q2 * j; };   // row y0 of a pair
    auto row_line = [&](int l) { return l; };
    int blk, src, dst;
    if (!step_slices(f, t0, blk, src, dst)) return;
    const RDiv dn1 = RDiv::of(sh.n1);
    auto padded = [&](int i) { const int y = dn1.div(i); return i + (QS - sh.n1) * y; };
    {
        const T *qs = src_slice(f, src, nr);
        for (int i = threadIdx.x; i < nr; i += blockDim.x) q[padded(i)] = qs[i];
    }
    __syncthreads();
    // The plane work of one (pair of rows, residue r) item at the row
    // passes' real-space end.  FIRST: q -> FP lines.  MID: FP lines -> q1,
    // h -> RP line.  LAST: RP line -> q_out, then FP lines of the next step.
    // e2 (with TAB, and e2n if in_table) lies in the padded table.
    enum { FIRST, MID, LAST };
    auto rows1 = [&](auto phase, const T *e2, const T *e2n, bool in_table, T *out) {
        constexpr int PH = decltype(phase)::value;
        auto go = [&](auto pc) {
            constexpr int P = decltype(pc)::value;
            for (int w = threadIdx.x; w < npair * sh.Q1; w += blockDim.x) {
                const int l = sh.dQ1.div(w), r = w - sh.Q1 * l;
                const int y0 = pair_line(l), y1 = y0 + sh.Q2;
                const bool two = y1 < sh.n2;   // an odd P2 leaves the last row of a residue alone
                C *b0 = m.buf + y0 * sh.LS, *b1 = m.buf + y1 * sh.LS;
                const int i0 = y0 * sh.n1 + r, i1 = y1 * sh.n1 + r;   // in global planes
                const int p0 = y0 * QS + r, p1 = y1 * QS + r;         // in the padded ones
                const int t0 = TAB ? p0 : i0, t1 = TAB ? p1 : i1;
                C v[P];
                T u0[P], u1[P], e[P];
                // (a row's table values ahead of its stores, which the
                // compiler must assume to alias the tables)
                auto load_e = [&](const T *src) {
#pragma unroll
                    for (int i = 0; i < P; i++) e[i] = src[sh.Q1 * i];
                };
                if (PH == FIRST) {
#pragma unroll
                    for (int i = 0; i < P; i++) {
                        u0[i] = q[p0 + sh.Q1 * i];
                        u1[i] = two ? q[p1 + sh.Q1 * i] : (T)0;
                    }
                } else if (PH == MID) {
                    // a: first half step, b: full step
                    load_e(e2 + t0);
                    X::template row_inv1<P>(sh, b0, r, v, m.tw1);
#pragma unroll
                    for (int i = 0; i < P; i++) {
                        const T ee = e[i] * e[i], q1 = div_by(ee * v[i].y, rn, rr);
                        q[p0 + sh.Q1 * i] = q1;
                        u0[i] = div_by(ee * v[i].x, rn, rr);
                        if (f.q1) f.q1[i0 + sh.Q1 * i] = q1;
                        if (f.h_out) f.h_out[i0 + sh.Q1 * i] = u0[i];
                    }
                    if (two) {
                        load_e(e2 + t1);
                        X::template row_inv1<P>(sh, b1, r, v, m.tw1);
#pragma unroll
                        for (int i = 0; i < P; i++) {
                            const T ee = e[i] * e[i], q1 = div_by(ee * v[i].y, rn, rr);
                            q[p1 + sh.Q1 * i] = q1;
                            u1[i] = div_by(ee * v[i].x, rn, rr);
                            if (f.q1) f.q1[i1 + sh.Q1 * i] = q1;
                            if (f.h_out) f.h_out[i1 + sh.Q1 * i] = u1[i];
                        }
                    }
#pragma unroll
                    for (int i = 0; i < P; i++) v[i] = mk<T>(u0[i], two ? u1[i] : (T)0);
                    X::template row_fwd1<P>(sh, b0, r, v, m.tw1);
                    continue;
                } else {
                    load_e(e2 + t0);
                    X::template row_inv1<P>(sh, b0, r, v, m.tw1);
                    auto row = [&](T *u, int pr, int ir, bool second) {
#pragma unroll
                        for (int i = 0; i < P; i++) {
                            const T q2 = div_by(e[i] * (second ? v[i].y : v[i].x), rn, rr);
                            u[i] = div_by((T)4 * q2 - q[pr + sh.Q1 * i], (T)3, rt);
                            q[pr + sh.Q1 * i] = u[i];
                            out[ir + sh.Q1 * i] = u[i];
                            if (f.q2_out) f.q2_out[ir + sh.Q1 * i] = q2;
                        }
                    };
                    row(u0, p0, i0, false);
                    if (two) {
                        load_e(e2 + t1);
                        row(u1, p1, i1, true);
                    }
                    if (!e2n) continue;
                }
                const int n0 = in_table ? p0 : i0, n1 = in_table ? p1 : i1;
#pragma unroll
                for (int i = 0; i < P; i++) {
                    const T e = e2n[n0 + sh.Q1 * i], a = e * u0[i];
                    v[i] = mk<T>(a, e * a);
                }
                X::template row_fwd1<P>(sh, b0, r, v, m.tw1);
                if (two) {
#pragma unroll
                    for (int i = 0; i < P; i++) {
                        const T e = e2n[n1 + sh.Q1 * i], a = e * u1[i];
                        v[i] = mk<T>(a, e * a);
                    }
                    X::template row_fwd1<P>(sh, b1, r, v, m.tw1);
                }
            }
        };
        RX_P(SH, P1, go);
    };
    // transform, filter, transform back, up to the real-space row passes
    auto conv = [&](auto fp, const T *eka, const T *ekb) {
        constexpr bool FP = decltype(fp)::value != 0;
        __syncthreads();
        if constexpr (FP) X::template rows2<-1>(sh, m.buf, sh.n2, dn2, row_line);
        else X::template rows2<-1>(sh, m.buf, npair, dpair, pair_line);
        __syncthreads();
        X::template cols_fwd1<FP, 2>(sh, m.buf, 1, sh.n2, m.ct, m.tw2);
        __syncthreads();
        X::template cols2<FP, 2>(sh, m.buf, 1, sh.n2, m.ct, [&](auto qc, int c, int kx, int ab, int, int k1, C *s, C *v) {
            constexpr int Q = decltype(qc)::value;
            const T *ek = (ab ? ekb : eka) + (TAB ? c : kx) + sh.n1h * k1;
            T e[Q];
#pragma unroll
            for (int k = 0; k < Q; k++) e[k] = TAB ? ek[sh.n1h * sh.P2 * k] : __ldg(ek + sh.n1h * sh.P2 * k);
#pragma unroll
            for (int n = 0; n < Q; n++) v[n] = s[n * sh.LS];
            Dft<Q, -1, T>::run(v);
#pragma unroll
            for (int k = 0; k < Q; k++) v[k] = scale(v[k], e[k]);
            Dft<Q, 1, T>::run(v);
#pragma unroll
            for (int n = 0; n < Q; n++) s[n * sh.LS] = v[n];
        });
        __syncthreads();
        X::template cols_inv1<FP, 2>(sh, m.buf, 1, sh.n2, m.ct, m.tw2);
        __syncthreads();
        if constexpr (FP) X::template rows2<1>(sh, m.buf, sh.n2, dn2, row_line);
        else X::template rows2<1>(sh, m.buf, npair, dpair, pair_line);
        __syncthreads();
    };
    rows1(RxInt<FIRST>(), nullptr, f.eo2[blk], false, nullptr);
    int cur = -1;
    for (int t = t0; t < t1; t++) {
        if (!step_slices(f, t, blk, src, dst)) break;
        if (TAB && blk != cur) {
            cur = blk;
            __syncthreads();
            for (int i = threadIdx.x; i < nr; i += blockDim.x) te2[padded(i)] = f.eo2[blk][i];
            for (int i = threadIdx.x; i < nkc; i += blockDim.x) {
                const int ky = sh.dn1h.div(i), k = m.ct[i - sh.n1h * ky].kx + sh.n1h * ky;
                tek[i] = f.ek2[blk][k];
                tek[nkc + i] = f.ek1[blk][k];
            }
        }
        const T *e2 = TAB ? te2 : f.eo2[blk], *k2 = TAB ? tek : f.ek2[blk], *k1 = TAB ? tek + nkc : f.ek1[blk];
        conv(RxInt<1>(), k2, k1);
        rows1(RxInt<MID>(), e2, nullptr, false, nullptr);
        conv(RxInt<0>(), k2, nullptr);
        int blk2, src2, dst2;
        const bool next = t + 1 < t1 && step_slices(f, t + 1, blk2, src2, dst2);
        rows1(RxInt<LAST>(), e2, !next ? nullptr : blk2 == blk ? e2 : f.eo2[blk2], TAB && next && blk2 == blk, dst_slice(f, dst, nr));
    }
}


// ---------------------------------------------------------------------
// dim 2: a field's whole sweep by a cluster of two CTAs: rank 0 makes the
// full steps q1, rank 1 the two half steps and the combination.  Each works
// on RP lines with the filter applied between the two column passes in
// registers (6 barriers a transform pair).  q1 crosses through the slice that
// the step is about to write, q through that slice once it is written; two
// cluster barriers a step order them, and rank 0 has half of rank 1's work,
// so that neither wait is long.
// Bound: rank 1's chain of 12 barriers and exchanges a step, or shared memory
// wavefronts where several CTAs share an SM.
// TAB: the current block's tables (exp(-w ds/4) and the rank's filter in
// column order) sit in shared memory too: for launches of at most one CTA
// per SM.
// grid = 2 nfields.
// ---------------------------------------------------------------------
template <typename T> __host__ __device__ constexpr size_t rx2_pair_smem(int n1, int n2, int npair, bool tab)
{
    return (rx_smem<T>(n1, n2, npair) + 15) / 16 * 16 +
           (tab ? sizeof(T) * ((size_t)rx2_stride(n1) * n2 + (n1 / 2 + 1) * n2) : 0);
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

template <typename T, typename SH, int NT, int MB, bool TAB>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NT, MB)
    k2x_pair(const SweepField<T> *fields, SH sh, RxTables tb, int t0, int t1)
{
    using X = Rx<T, SH>;
    using C = cx<T>;
    const SweepField<T> &f = fields[blockIdx.x >> 1];
    const int rank = blockIdx.x & 1, npair = sh.Q2 * sh.HP;
    const RxMem<T, SH> m(sh, tb, npair);
    const int nr = sh.n1 * sh.n2, nkc = sh.n1h * sh.n2, QS = rx2_stride(sh.n1);
    T *te2 = (T *)(((size_t)m.end(sh) + 15) / 16 * 16), *tek = te2 + QS * sh.n2;   // (TAB)
    const T rn = (T)(2.0 * nr), rr = (T)(1.0 / (2.0 * nr)), rt = (T)(1.0 / 3.0);
    const RDiv dpair = RDiv::of(npair), dn1 = RDiv::of(sh.n1);
    auto same = [](int l) { return l; };
    int blk, src, dst;
    if (!step_slices(f, t0, blk, src, dst)) return;   // the same for the whole cluster
    __syncthreads();
    // f(P, line, r, y0's offset + r in a global plane, in a padded one, y1 exists)
    auto items = [&](auto f2) {
        auto go = [&](auto pc) {
            for (int w = threadIdx.x; w < npair * sh.Q1; w += blockDim.x) {
                const int l = sh.dQ1.div(w), r = w - sh.Q1 * l, y0 = l + sh.Q2 * sh.dQ2.div(l);   // r2 + 2 j Q2
                f2(pc, m.buf + l * sh.LS, r, y0 * sh.n1 + r, y0 * QS + r, y0 + sh.Q2 < sh.n2);
            }
        };
        RX_P(SH, P1, go);
    };
    // P values of rows y0 and y1 of a global plane (or of the padded table)
    auto load2 = [&](auto pc, const T *p, int row, bool two, T *a, T *b, bool cg) {
        constexpr int P = decltype(pc)::value;
#pragma unroll
        for (int i = 0; i < P; i++) {
            a[i] = cg ? __ldcg(p + sh.Q1 * i) : p[sh.Q1 * i];
            b[i] = !two ? (T)0 : cg ? __ldcg(p + sh.Q2 * row + sh.Q1 * i) : p[sh.Q2 * row + sh.Q1 * i];
        }
    };
    auto load_e = [&](auto pc, const T *e2, bool table, int g, int pd, bool two, T *a, T *b) {
        if (table) load2(pc, te2 + pd, QS, two, a, b, false);
        else load2(pc, e2 + g, sh.n1, two, a, b, false);
    };
    // transform, filter, transform back, up to the real-space row passes
    auto conv = [&](const T *ekt) {
        __syncthreads();
        X::template rows2<-1>(sh, m.buf, npair, dpair, same);
        __syncthreads();
        X::template cols_fwd1<false, 1>(sh, m.buf, 1, npair, m.ct, m.tw2);
        __syncthreads();
        X::template cols2<false, 1>(sh, m.buf, 1, npair, m.ct, [&](auto qc, int c, int kx, int, int, int k1, C *s, C *v) {
            constexpr int Q = decltype(qc)::value;
            const T *ek = ekt + (TAB ? c : kx) + sh.n1h * k1;
            T e[Q];
#pragma unroll
            for (int k = 0; k < Q; k++) e[k] = TAB ? ek[sh.n1h * sh.P2 * k] : __ldg(ek + sh.n1h * sh.P2 * k);
#pragma unroll
            for (int n = 0; n < Q; n++) v[n] = s[n * sh.LS];
            Dft<Q, -1, T>::run(v);
#pragma unroll
            for (int k = 0; k < Q; k++) v[k] = scale(v[k], e[k]);
            Dft<Q, 1, T>::run(v);
#pragma unroll
            for (int n = 0; n < Q; n++) s[n * sh.LS] = v[n];
        });
        __syncthreads();
        X::template cols_inv1<false, 1>(sh, m.buf, 1, npair, m.ct, m.tw2);
        __syncthreads();
        X::template rows2<1>(sh, m.buf, npair, dpair, same);
        __syncthreads();
    };
    int cur = -1;
    for (int t = t0; t < t1; t++) {
        if (!step_slices(f, t, blk, src, dst)) break;
        const T *e2 = f.eo2[blk], *ekt = rank ? f.ek2[blk] : f.ek1[blk];
        if (TAB) {
            if (blk != cur) {
                cur = blk;
                __syncthreads();
                for (int i = threadIdx.x; i < nr; i += blockDim.x) te2[i + (QS - sh.n1) * dn1.div(i)] = e2[i];
                for (int i = threadIdx.x; i < nkc; i += blockDim.x) {
                    const int ky = sh.dn1h.div(i);
                    tek[i] = ekt[m.ct[i - sh.n1h * ky].kx + sh.n1h * ky];
                }
                __syncthreads();
            }
            ekt = tek;
        }
        T *out = dst_slice(f, dst, nr);
        if (rank == 0) {
            const T *q = src_slice(f, src, nr);
            items([&](auto pc, C *b, int r, int g, int pd, bool two) {
                constexpr int P = decltype(pc)::value;
                T q0[P], q1[P], ea[P], eb[P];
                load2(pc, q + g, sh.n1, two, q0, q1, true);
                load_e(pc, e2, TAB, g, pd, two, ea, eb);
                C v[P];
#pragma unroll
                for (int i = 0; i < P; i++) v[i] = mk<T>(ea[i] * (ea[i] * q0[i]), eb[i] * (eb[i] * q1[i]));
                X::template row_fwd1<P>(sh, b, r, v, m.tw1);
            });
            conv(ekt);
            items([&](auto pc, C *b, int r, int g, int pd, bool two) {
                constexpr int P = decltype(pc)::value;
                T ea[P], eb[P];
                load_e(pc, e2, TAB, g, pd, two, ea, eb);
                C v[P];
                X::template row_inv1<P>(sh, b, r, v, m.tw1);
                auto put = [&](T *p) {
#pragma unroll
                    for (int i = 0; i < P; i++) {
                        p[g + sh.Q1 * i] = div_by(ea[i] * ea[i] * v[i].x, rn, rr);
                        if (two) p[g + sh.Q2 * sh.n1 + sh.Q1 * i] = div_by(eb[i] * eb[i] * v[i].y, rn, rr);
                    }
                };
                put(out);
                if (f.q1) put(f.q1);
            });
            cluster_arrive();   // q1 is in the destination slice
            cluster_wait();
            cluster_arrive();
            cluster_wait();     // ... and now q
        } else {
            if (t == t0) {
                const T *q = src_slice(f, src, nr);
                items([&](auto pc, C *b, int r, int g, int pd, bool two) {
                    constexpr int P = decltype(pc)::value;
                    T q0[P], q1[P], ea[P], eb[P];
                    load2(pc, q + g, sh.n1, two, q0, q1, false);
                    load_e(pc, e2, TAB, g, pd, two, ea, eb);
                    C v[P];
#pragma unroll
                    for (int i = 0; i < P; i++) v[i] = mk<T>(ea[i] * q0[i], eb[i] * q1[i]);
                    X::template row_fwd1<P>(sh, b, r, v, m.tw1);
                });
            }
            cluster_arrive();
            conv(ekt);
            items([&](auto pc, C *b, int r, int g, int pd, bool two) {
                constexpr int P = decltype(pc)::value;
                T ea[P], eb[P];
                load_e(pc, e2, TAB, g, pd, two, ea, eb);
                C v[P];
                X::template row_inv1<P>(sh, b, r, v, m.tw1);
#pragma unroll
                for (int i = 0; i < P; i++) {
                    v[i] = mk<T>(div_by(ea[i] * ea[i] * v[i].x, rn, rr), two ? div_by(eb[i] * eb[i] * v[i].y, rn, rr) : (T)0);
                    if (f.h_out) {
                        f.h_out[g + sh.Q1 * i] = v[i].x;
                        if (two) f.h_out[g + sh.Q2 * sh.n1 + sh.Q1 * i] = v[i].y;
                    }
                }
                X::template row_fwd1<P>(sh, b, r, v, m.tw1);
            });
            conv(ekt);
            int blk2, src2, dst2;
            const bool next = t + 1 < t1 && step_slices(f, t + 1, blk2, src2, dst2);
            const bool table = TAB && next && blk2 == blk;
            const T *n2 = next ? f.eo2[blk2] : nullptr;
            cluster_wait();     // q1 is in the destination slice
            items([&](auto pc, C *b, int r, int g, int pd, bool two) {
                constexpr int P = decltype(pc)::value;
                // (all loads ahead of the stores, which the compiler must
                // assume to alias them)
                T q0[P], q1[P], ea[P], eb[P];
                load2(pc, out + g, sh.n1, two, q0, q1, true);
                load_e(pc, e2, TAB, g, pd, two, ea, eb);
                C v[P];
                X::template row_inv1<P>(sh, b, r, v, m.tw1);
#pragma unroll
                for (int i = 0; i < P; i++) {
                    const T qa = div_by(ea[i] * v[i].x, rn, rr), qb = div_by(eb[i] * v[i].y, rn, rr);
                    if (f.q2_out) {
                        f.q2_out[g + sh.Q1 * i] = qa;
                        if (two) f.q2_out[g + sh.Q2 * sh.n1 + sh.Q1 * i] = qb;
                    }
                    q0[i] = div_by((T)4 * qa - q0[i], (T)3, rt);
                    q1[i] = div_by((T)4 * qb - q1[i], (T)3, rt);
                }
                if (next && n2 != e2) load_e(pc, n2, table, g, pd, two, ea, eb);
#pragma unroll
                for (int i = 0; i < P; i++) {
                    out[g + sh.Q1 * i] = q0[i];
                    if (two) out[g + sh.Q2 * sh.n1 + sh.Q1 * i] = q1[i];
                    v[i] = mk<T>(ea[i] * q0[i], two ? eb[i] * q1[i] : (T)0);
                }
                if (next) X::template row_fwd1<P>(sh, b, r, v, m.tw1);
            });
            cluster_arrive();
            cluster_wait();
        }
    }
}

// First forward row passes of the RP lines of one real plane: pairs of rows
// of src into the lines from `line0` on.
template <int P, typename T, typename SH>
__device__ __forceinline__ void rp_load(const SH &sh, const RxMem<T, SH> &m, int w, int line0, const T *src)
{
    const int lw = sh.dQ1.div(w), r = w - sh.Q1 * lw, l = rx_line<T, SH>(lw), y0 = l + sh.Q2 * sh.dQ2.div(l);   // r2 + 2 j Q2
    const bool two = y0 + sh.Q2 < sh.n2;
    const T *a = src + y0 * sh.n1 + r, *b = a + sh.Q2 * sh.n1;
    cx<T> v[P];
#pragma unroll
    for (int i = 0; i < P; i++) v[i] = mk<T>(a[sh.Q1 * i], two ? b[sh.Q1 * i] : (T)0);
    Rx<T, SH>::template row_fwd1<P>(sh, m.buf + (line0 + l) * sh.LS, r, v, m.tw1);
}

// Stress slice sums for dim 2 (contract of k2_stress_slices): one CTA per
// (slice, job), qf and qr as RP planes, the products formed in registers
// after the last column pass.  (Not as one FP pair: at the chain's ends qf
// and qr differ by many orders of magnitude, and the smaller one would carry
// the larger one's rounding.)
template <typename T, typename SH, int NT>
__global__ void __launch_bounds__(NT) k2x_stress(const StressJob<T> *jobs, SH sh, RxTables tb)
{
    using X = Rx<T, SH>;
    using C = cx<T>;
    const StressJob<T> &J = jobs[blockIdx.y];
    const int s = blockIdx.x;
    if (s >= J.nslices) return;
    const int npair = sh.Q2 * sh.HP;
    const RxMem<T, SH> m(sh, tb, 2 * npair);
    __shared__ double red[32];
    const int nr = sh.n1 * sh.n2;
    const long nk = (long)sh.n1h * sh.n2;
    const T *qf = J.qf + (long)s * nr, *qr = J.qr + (long)s * nr;
    __syncthreads();
    auto go = [&](auto pc) {
        constexpr int P = decltype(pc)::value;
        const int ni = npair * sh.Q1;
        for (int w = threadIdx.x; w < 2 * ni; w += blockDim.x)
            rp_load<P, T, SH>(sh, m, w < ni ? w : w - ni, w < ni ? 0 : npair, w < ni ? qf : qr);
    };
    RX_P(SH, P1, go);
    __syncthreads();
    X::template rows2<-1>(sh, m.buf, 2 * npair, RDiv::of(2 * npair), [](int l) { return l; });
    __syncthreads();
    X::template cols_fwd1<false, 1>(sh, m.buf, 2, npair, m.ct, m.tw2);
    __syncthreads();
    double acc[PSCFG_MAXCP] = {0, 0, 0, 0, 0, 0};
    auto dots = [&](auto qc) {
        constexpr int Q = decltype(qc)::value;
        for (int w = threadIdx.x; w < sh.P2 * sh.n1h; w += blockDim.x) {
            int k1, c;
            X::col_item(sh, w, sh.P2, k1, c);
            const RxCol col = X::column(m.ct, c);
            const C *b0 = m.buf + Q * (k1 / 2) * sh.LS + ((k1 & 1) ? col.wpos : col.pos), *b1 = b0 + npair * sh.LS;
            C a[Q], b[Q];
#pragma unroll
            for (int n = 0; n < Q; n++) {
                a[n] = b0[n * sh.LS];
                b[n] = b1[n * sh.LS];
            }
            Dft<Q, -1, T>::run(a);
            Dft<Q, -1, T>::run(b);
#pragma unroll
            for (int k = 0; k < Q; k++) {
                const double pr = (double)a[k].x * (double)b[k].x + (double)a[k].y * (double)b[k].y;
                const double *wd = J.wdgsq + col.kx + (long)sh.n1h * (k1 + sh.P2 * k);
#pragma unroll
                for (int p = 0; p < PSCFG_MAXCP; p++)
                    if (p < J.ncp) acc[p] += __ldg(wd + p * nk) * pr;
            }
        }
    };
    RX_Q(SH, Q2, dots);
#pragma unroll
    for (int p = 0; p < PSCFG_MAXCP; p++) {
        if (p >= J.ncp) break;   // uniform across the CTA
        const double tot = block_sum(acc[p], red);
        if (threadIdx.x == 0) J.inc[(long)s * PSCFG_MAXCP + p] = 0.25 * tot;
        __syncthreads();
    }
}

// ---------------------------------------------------------------------
// dim 3: the x-y passes of a step.  A CTA holds `ppc` z-planes.
//   k3v_fwd    S2, S1 <- Fxy of exp(-w ds/4) q, exp(-w ds/2) q     (first step)
//   k3v_zconv  S <- Fz^-1[ek Fz S], S1 with ek1 and S2 with ek2
//   k3v_mid    S2 <- Fxy[eo1 Fxy^-1[S2] / N]
//   k3v_zconv  S2 with ek2
//   k3v_final  q_out = (4 eo2 Fxy^-1[S2] - eo1 Fxy^-1[S1]) / 3 N, then the
//              next step's S2, S1
// S1 and S2 are the two halves of FP pairs, so the full step's q1 never
// leaves the chip.  With f.h_out set (the adjoint's single steps) the
// intermediates q1, h and q2 are written too.
// ---------------------------------------------------------------------
template <typename T, typename SH> struct Rx3 {
    using X = Rx<T, SH>;
    using C = cx<T>;

    // rows and columns of np FP planes (lines already through row_fwd1) into
    // sa, sb (spectra of the first plane)
    __device__ __forceinline__ static void fwd_fp(const SH &sh, const RxMem<T, SH> &m, int np, C *sa, C *sb)
    {
        __syncthreads();
        X::template rows2<-1>(sh, m.buf, np * sh.n2, RDiv::of(np * sh.n2), [](int l) { return l; });
        __syncthreads();
        X::template cols_fwd1<true, 1>(sh, m.buf, np, sh.n2, m.ct, m.tw2);
        __syncthreads();
        X::template cols2<true, 1>(sh, m.buf, np, sh.n2, m.ct, [&](auto qc, int c, int, int ab, int pl, int k1, C *s, C *v) {
            constexpr int Q = decltype(qc)::value;
            C *d = (ab ? sb : sa) + (long)(pl * sh.n2 + k1) * sh.n1h + c;
#pragma unroll
            for (int n = 0; n < Q; n++) v[n] = s[n * sh.LS];
            Dft<Q, -1, T>::run(v);
#pragma unroll
            for (int k = 0; k < Q; k++) d[(long)sh.n1h * sh.P2 * k] = v[k];
        });
    }
};

template <typename T, typename SH, int NT, int MB>
__global__ void __launch_bounds__(NT, MB)
    k3v_fwd(const SweepField<T> *fields, SH sh, RxTables tb, int n3, int ppc, int t)
{
    using X = Rx<T, SH>;
    const SweepField<T> &f = fields[blockIdx.y];
    int blk, src, dst;
    if (!step_slices(f, t, blk, src, dst)) return;
    const int z0 = blockIdx.x * ppc, np = min(ppc, n3 - z0), npl = sh.n1 * sh.n2;
    const RxMem<T, SH> m(sh, tb, ppc * sh.n2);
    const T *q = src_slice(f, src, (long)npl * n3) + (long)z0 * npl, *e2 = f.eo2[blk] + (long)z0 * npl;
    __syncthreads();
    auto go = [&](auto pc) {
        constexpr int P = decltype(pc)::value;
        for (int w = threadIdx.x; w < np * sh.n2 * sh.Q1; w += blockDim.x) {
            const int lw = sh.dQ1.div(w), r = w - sh.Q1 * lw, l = rx_line<T, SH>(lw);
            cx<T> v[P];
#pragma unroll
            for (int i = 0; i < P; i++) {
                const int x = l * sh.n1 + sh.Q1 * i + r;
                const T e = e2[x], a = e * q[x];
                v[i] = mk<T>(a, e * a);
            }
            X::template row_fwd1<P>(sh, m.buf + l * sh.LS, r, v, m.tw1);
        }
    };
    RX_P(SH, P1, go);
    const long so = (long)z0 * sh.n2 * sh.n1h;
    Rx3<T, SH>::fwd_fp(sh, m, np, f.S2 + so, f.S1 + so);
}

template <typename T, typename SH, int NT, int MB>
__global__ void __launch_bounds__(NT, MB)
    k3v_mid(const SweepField<T> *fields, SH sh, RxTables tb, int n3, int ppc, int t)
{
    using X = Rx<T, SH>;
    using C = cx<T>;
    const SweepField<T> &f = fields[blockIdx.y];
    const int z0 = blockIdx.x * ppc, np = min(ppc, n3 - z0), npl = sh.n1 * sh.n2, npair = sh.Q2 * sh.HP;
    C *S = f.S2 + (long)z0 * sh.n2 * sh.n1h;
    const RxMem<T, SH> m(sh, tb, ppc * npair);
    const T rn = (T)(2.0 * npl * n3), rr = (T)(1.0 / (2.0 * npl * n3));
    const RDiv dl = RDiv::of(np * npair), dpair = RDiv::of(npair);
    auto same = [](int l) { return l; };
    // (the spectrum's loads go out before the step's descriptor is read; a
    // field past its last step stops after them)
    if (!SH::FIXED) __syncthreads();
    X::template cols2<false, 1>(sh, m.buf, np, npair, m.ct, [&](auto qc, int c, int, int, int pl, int k1, C *s, C *v) {
        constexpr int Q = decltype(qc)::value;
        const C *d = S + (long)(pl * sh.n2 + k1) * sh.n1h + c;
#pragma unroll
        for (int k = 0; k < Q; k++) v[k] = d[(long)sh.n1h * sh.P2 * k];
        Dft<Q, 1, T>::run(v);
#pragma unroll
        for (int n = 0; n < Q; n++) s[n * sh.LS] = v[n];
    });
    int blk, src, dst;
    if (!step_slices(f, t, blk, src, dst)) return;
    const T *e2 = f.eo2[blk] + (long)z0 * npl;
    T *ho = f.h_out ? f.h_out + (long)z0 * npl : nullptr;
    __syncthreads();
    X::template cols_inv1<false, 1>(sh, m.buf, np, npair, m.ct, m.tw2);
    __syncthreads();
    X::template rows2<1>(sh, m.buf, np * npair, dl, same);
    __syncthreads();
    auto go = [&](auto pc) {
        constexpr int P = decltype(pc)::value;
        for (int w = threadIdx.x; w < np * npair * sh.Q1; w += blockDim.x) {
            const int lw = sh.dQ1.div(w), r = w - sh.Q1 * lw, l = rx_line<T, SH>(lw);
            const int pl = dpair.div(l), lp = l - npair * pl, j = sh.dQ2.div(lp);
            const int y0 = lp + sh.Q2 * j;   // r2 + 2 j Q2
            const bool two = y0 + sh.Q2 < sh.n2;
            const int i0 = (pl * sh.n2 + y0) * sh.n1 + r, i1 = i0 + sh.Q2 * sh.n1;
            C v[P];
            T e0[P], e1[P];
#pragma unroll
            for (int i = 0; i < P; i++) {
                e0[i] = e2[i0 + sh.Q1 * i];
                e1[i] = two ? e2[i1 + sh.Q1 * i] : (T)0;
            }
            X::template row_inv1<P>(sh, m.buf + l * sh.LS, r, v, m.tw1);
#pragma unroll
            for (int i = 0; i < P; i++) {
                v[i] = mk<T>(div_by(e0[i] * e0[i] * v[i].x, rn, rr), two ? div_by(e1[i] * e1[i] * v[i].y, rn, rr) : (T)0);
                if (ho) {
                    ho[i0 + sh.Q1 * i] = v[i].x;
                    if (two) ho[i1 + sh.Q1 * i] = v[i].y;
                }
            }
            X::template row_fwd1<P>(sh, m.buf + l * sh.LS, r, v, m.tw1);
        }
    };
    RX_P(SH, P1, go);
    __syncthreads();
    X::template rows2<-1>(sh, m.buf, np * npair, dl, same);
    __syncthreads();
    X::template cols_fwd1<false, 1>(sh, m.buf, np, npair, m.ct, m.tw2);
    __syncthreads();
    X::template cols2<false, 1>(sh, m.buf, np, npair, m.ct, [&](auto qc, int c, int, int, int pl, int k1, C *s, C *v) {
        constexpr int Q = decltype(qc)::value;
        C *d = S + (long)(pl * sh.n2 + k1) * sh.n1h + c;
#pragma unroll
        for (int n = 0; n < Q; n++) v[n] = s[n * sh.LS];
        Dft<Q, -1, T>::run(v);
#pragma unroll
        for (int k = 0; k < Q; k++) d[(long)sh.n1h * sh.P2 * k] = v[k];
    });
}

template <typename T, typename SH, int NT, int MB>
__global__ void __launch_bounds__(NT, MB)
    k3v_final(const SweepField<T> *fields, SH sh, RxTables tb, int n3, int ppc, int t)
{
    using X = Rx<T, SH>;
    using C = cx<T>;
    const SweepField<T> &f = fields[blockIdx.y];
    const int z0 = blockIdx.x * ppc, np = min(ppc, n3 - z0), npl = sh.n1 * sh.n2;
    const long po = (long)z0 * npl, so = (long)z0 * sh.n2 * sh.n1h;
    const C *sa = f.S2 + so, *sb = f.S1 + so;
    const RxMem<T, SH> m(sh, tb, ppc * sh.n2);
    const T rn = (T)(6.0 * npl * n3), rr = (T)(1.0 / (6.0 * npl * n3));
    if (!SH::FIXED) __syncthreads();
    X::template cols2<true, 1>(sh, m.buf, np, sh.n2, m.ct, [&](auto qc, int c, int, int ab, int pl, int k1, C *s, C *v) {
        constexpr int Q = decltype(qc)::value;
        const C *d = (ab ? sb : sa) + (long)(pl * sh.n2 + k1) * sh.n1h + c;
#pragma unroll
        for (int k = 0; k < Q; k++) v[k] = d[(long)sh.n1h * sh.P2 * k];
        Dft<Q, 1, T>::run(v);
#pragma unroll
        for (int n = 0; n < Q; n++) s[n * sh.LS] = v[n];
    });
    int blk, src, dst, blk2, src2, dst2;
    if (!step_slices(f, t, blk, src, dst)) return;   // (as in k3v_mid)
    const T *e2 = f.eo2[blk] + po;
    T *out = dst_slice(f, dst, (long)npl * n3) + po;
    T *q1o = f.h_out ? f.q1 + po : nullptr, *q2o = f.h_out && f.q2_out ? f.q2_out + po : nullptr;
    const bool next = step_slices(f, t + 1, blk2, src2, dst2);   // the same for the whole CTA
    const T *n2 = f.eo2[next ? blk2 : blk] + po;
    __syncthreads();
    X::template cols_inv1<true, 1>(sh, m.buf, np, sh.n2, m.ct, m.tw2);
    __syncthreads();
    X::template rows2<1>(sh, m.buf, np * sh.n2, RDiv::of(np * sh.n2), [](int l) { return l; });
    __syncthreads();
    auto go = [&](auto pc) {
        constexpr int P = decltype(pc)::value;
        for (int w = threadIdx.x; w < np * sh.n2 * sh.Q1; w += blockDim.x) {
            const int lw = sh.dQ1.div(w), r = w - sh.Q1 * lw, l = rx_line<T, SH>(lw), x0 = l * sh.n1 + r;
            C v[P];
            T e[P], en[P];
            // (ahead of the stores to out, which the compiler must assume to
            // alias the tables)
#pragma unroll
            for (int i = 0; i < P; i++) e[i] = e2[x0 + sh.Q1 * i];
#pragma unroll
            for (int i = 0; i < P; i++) en[i] = n2 == e2 ? e[i] : n2[x0 + sh.Q1 * i];
            X::template row_inv1<P>(sh, m.buf + l * sh.LS, r, v, m.tw1);
#pragma unroll
            for (int i = 0; i < P; i++) {
                const int x = x0 + sh.Q1 * i;
                const T o = div_by(e[i] * ((T)4 * v[i].x - e[i] * v[i].y), rn, rr);
                out[x] = o;
                if (q1o) q1o[x] = div_by((T)3 * (e[i] * e[i] * v[i].y), rn, rr);
                if (q2o) q2o[x] = div_by((T)3 * (e[i] * v[i].x), rn, rr);
                const T a = en[i] * o;
                v[i] = mk<T>(a, en[i] * a);
            }
            if (next) X::template row_fwd1<P>(sh, m.buf + l * sh.LS, r, v, m.tw1);
        }
    };
    RX_P(SH, P1, go);
    if (!next) return;
    Rx3<T, SH>::fwd_fp(sh, m, np, f.S2 + so, f.S1 + so);
}

// After k3v_fwd and k3v_zconv on S1 and S2: q1 = eo1 Fxy^-1[S1] / N and
// h = eo1 Fxy^-1[S2] / N alone (the adjoint's steps of stored slices, whose
// second half step follows from the next slice).  ns = 1 fields, t = 0.
template <typename T, typename SH, int NT, int MB>
__global__ void __launch_bounds__(NT, MB) k3v_half(const SweepField<T> *fields, SH sh, RxTables tb, int n3, int ppc)
{
    using X = Rx<T, SH>;
    using C = cx<T>;
    const SweepField<T> &f = fields[blockIdx.y];
    const int z0 = blockIdx.x * ppc, np = min(ppc, n3 - z0), npl = sh.n1 * sh.n2;
    const long po = (long)z0 * npl, so = (long)z0 * sh.n2 * sh.n1h;
    const C *sa = f.S2 + so, *sb = f.S1 + so;
    const RxMem<T, SH> m(sh, tb, ppc * sh.n2);
    const T rn = (T)(2.0 * npl * n3), rr = (T)(1.0 / (2.0 * npl * n3));
    const T *e2 = f.eo2[0] + po;
    T *q1 = f.q1 + po, *h = f.h_out + po;
    if (!SH::FIXED) __syncthreads();
    X::template cols2<true, 1>(sh, m.buf, np, sh.n2, m.ct, [&](auto qc, int c, int, int ab, int pl, int k1, C *s, C *v) {
        constexpr int Q = decltype(qc)::value;
        const C *d = (ab ? sb : sa) + (long)(pl * sh.n2 + k1) * sh.n1h + c;
#pragma unroll
        for (int k = 0; k < Q; k++) v[k] = d[(long)sh.n1h * sh.P2 * k];
        Dft<Q, 1, T>::run(v);
#pragma unroll
        for (int n = 0; n < Q; n++) s[n * sh.LS] = v[n];
    });
    __syncthreads();
    X::template cols_inv1<true, 1>(sh, m.buf, np, sh.n2, m.ct, m.tw2);
    __syncthreads();
    X::template rows2<1>(sh, m.buf, np * sh.n2, RDiv::of(np * sh.n2), [](int l) { return l; });
    __syncthreads();
    auto go = [&](auto pc) {
        constexpr int P = decltype(pc)::value;
        for (int w = threadIdx.x; w < np * sh.n2 * sh.Q1; w += blockDim.x) {
            const int lw = sh.dQ1.div(w), r = w - sh.Q1 * lw, l = rx_line<T, SH>(lw), x0 = l * sh.n1 + r;
            C v[P];
            T e[P];
#pragma unroll
            for (int i = 0; i < P; i++) e[i] = e2[x0 + sh.Q1 * i];
            X::template row_inv1<P>(sh, m.buf + l * sh.LS, r, v, m.tw1);
#pragma unroll
            for (int i = 0; i < P; i++) {
                h[x0 + sh.Q1 * i] = div_by(e[i] * e[i] * v[i].x, rn, rr);
                q1[x0 + sh.Q1 * i] = div_by(e[i] * e[i] * v[i].y, rn, rr);
            }
        }
    };
    RX_P(SH, P1, go);
}

// x-y transform of slices s0 .. s0 + cs of qf and qr of every job (RP
// planes, see k2x_stress); spectra at ((job cs + slice) 2 + which) nk.
// grid = (planes / ppc, cs, 2 njobs).
template <typename T, typename SH, int NT, int MB>
__global__ void __launch_bounds__(NT, MB)
    k3v_stress_xy(const StressJob<T> *jobs, SH sh, RxTables tb, int n3, int ppc, int s0, int cs, cx<T> *spec)
{
    using X = Rx<T, SH>;
    using C = cx<T>;
    const int job = blockIdx.z >> 1, which = blockIdx.z & 1;
    const StressJob<T> &J = jobs[job];
    const int s = s0 + blockIdx.y;
    if (s >= J.nslices) return;
    const int z0 = blockIdx.x * ppc, np = min(ppc, n3 - z0), npl = sh.n1 * sh.n2, npair = sh.Q2 * sh.HP;
    const RxMem<T, SH> m(sh, tb, ppc * npair);
    const T *q = (which ? J.qr : J.qf) + (long)s * npl * n3 + (long)z0 * npl;
    const RDiv dni = RDiv::of(npair * sh.Q1);
    __syncthreads();
    auto go = [&](auto pc) {
        constexpr int P = decltype(pc)::value;
        const int ni = npair * sh.Q1;
        for (int w = threadIdx.x; w < np * ni; w += blockDim.x) {
            const int pl = dni.div(w);
            rp_load<P, T, SH>(sh, m, w - ni * pl, pl * npair, q + pl * npl);
        }
    };
    RX_P(SH, P1, go);
    __syncthreads();
    X::template rows2<-1>(sh, m.buf, np * npair, RDiv::of(np * npair), [](int l) { return l; });
    __syncthreads();
    X::template cols_fwd1<false, 1>(sh, m.buf, np, npair, m.ct, m.tw2);
    __syncthreads();
    const long nk = (long)sh.n1h * sh.n2 * n3;
    C *S = spec + (((long)job * cs + blockIdx.y) * 2 + which) * nk + (long)z0 * sh.n2 * sh.n1h;
    X::template cols2<false, 1>(sh, m.buf, np, npair, m.ct, [&](auto qc, int c, int, int, int pl, int k1, C *s, C *v) {
        constexpr int Q = decltype(qc)::value;
        C *d = S + (long)(pl * sh.n2 + k1) * sh.n1h + c;
#pragma unroll
        for (int n = 0; n < Q; n++) v[n] = s[n * sh.LS];
        Dft<Q, -1, T>::run(v);
#pragma unroll
        for (int k = 0; k < Q; k++) d[(long)sh.n1h * sh.P2 * k] = v[k];
    });
}

// ---------------------------------------------------------------------
// z lines of TC columns, N3 = P Q: two exchanges around the filter.
// ---------------------------------------------------------------------
struct RzShape {
    static constexpr bool FIXED = false;
    static constexpr int QM = 16;
    int n3, P, Q;
};
struct RzShape10 : RzShape {
    static constexpr int QM = 10;
};
template <int N3, int P_> struct RzFixed {
    static constexpr bool FIXED = true;
    static constexpr int n3 = N3, P = P_, Q = N3 / P_;
};
template <typename T> __host__ __device__ constexpr size_t rz_smem(int n3, int tc, int bufs) { return sizeof(cx<T>) * ((size_t)n3 * tc * bufs + n3); }

// geometry of the columns: c -> (kx, ky)
struct RzCols {
    int n1h, n2;
    RDiv dn1h;
    const RxCol *cols;
    const void *twz;
};

// A filter value as the product of its 1-D factors.  In FP64 they are rounded
// values, whose product (2.5 ulp) is no worse than a table's exp with its
// rounded argument.  In FP32 each is a pair, the value and its remainder (side
// by side in memory), so that the product is rounded once, like a table's
// value: an FP32 density of 64 x 128 x 224 is off by 1.5e-5, and by 2.3e-5
// with rounded factors, at the same time but for 0.5%.
template <typename T> struct EkFactor {
    T v, rest;
};
template <typename T> __device__ __forceinline__ EkFactor<T> ek_factor(const T *f, int i)
{
    if constexpr (sizeof(T) == 8) {
        return EkFactor<T>{__ldg(f + i), (T)0};
    } else {
        const float2 p = __ldg((const float2 *)f + i);
        return EkFactor<T>{p.x, p.y};
    }
}
// fx fy (once per column), and (fx fy) fz
template <typename T> __host__ __device__ __forceinline__ EkFactor<T> ek_xy(EkFactor<T> x, EkFactor<T> y)
{
    if (sizeof(T) == 8) return EkFactor<T>{x.v * y.v, (T)0};
    const double d = ((double)x.v + (double)x.rest) * ((double)y.v + (double)y.rest);
    return EkFactor<T>{(T)d, (T)(d - (double)(T)d)};
}
template <typename T> __host__ __device__ __forceinline__ T ek_value(EkFactor<T> xy, EkFactor<T> z)
{
    return sizeof(T) == 8 ? xy.v * z.v : fma(xy.v, z.v, fma(xy.v, z.rest, xy.rest * z.v));
}

// grid = (ceil(n1h n2 / TC), nfields, 1 or 2); which: 1 = S1/ek1, 2 =
// S2/ek2, 3 = both (grid.z selects).  ekf: the filter as products of 1-D
// factors over kx, ky, kz (orthogonal cells), which saves the read of ek.
template <typename T, typename ZS, int TC, int NT, int MB>
__global__ void __launch_bounds__(NT, MB) k3v_zconv(const SweepField<T> *fields, ZS sh, RzCols g, int t, int which)
{
    using C = cx<T>;
    const SweepField<T> &f = fields[blockIdx.y];
    const int sel = which == 3 ? (int)blockIdx.z + 1 : which;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *buf = (C *)smem_raw, *tw = buf + sh.n3 * TC;
    const int ncol = g.n1h * g.n2, c = threadIdx.x % TC, col = blockIdx.x * TC + c, r0 = threadIdx.x / TC;
    constexpr int NR = NT / TC;   // at least P and Q: one item a thread and pass
    const bool ok = col < ncol;
    C *S = ((sel == 1) ? f.S1 : f.S2) + (ok ? col : 0);
    int blk, src, dst;
    bool live = true;
    auto first = [&](auto pc) {
        constexpr int P = decltype(pc)::value;
        const int r = r0;
        C v[P];
        // (the loads go out before the tables and the step's descriptor are read)
        if (r < sh.Q) {
#pragma unroll
            for (int i = 0; i < P; i++) v[i] = ok ? S[(long)(sh.Q * i + r) * ncol] : mk<T>((T)0, (T)0);
        }
        for (int i = threadIdx.x; i < sh.n3; i += NT) tw[i] = ((const C *)g.twz)[i];
        live = step_slices(f, t, blk, src, dst);
        __syncthreads();
        if (r < sh.Q && live) {
            Dft<P, -1, T>::run(v);
            C *b = buf + r * TC + c;
            b[0] = v[0];
#pragma unroll
            for (int k = 1; k < P; k++) b[sh.Q * k * TC] = cmul(v[k], tw[r * k]);
        }
    };
    RX_Q(ZS, P, first);
    if (!live) return;   // a field past its last step, the same for the whole CTA
    const int ky = g.dn1h.div(ok ? col : 0), kx = g.cols[(ok ? col : 0) - ky * g.n1h].kx;
    __syncthreads();
    const T *ekf = f.ekf[blk];
    const T *ek = ((sel == 1) ? f.ek1[blk] : f.ek2[blk]) + kx + (long)g.n1h * ky;
    const T *fz = nullptr;
    EkFactor<T> exy = {};
    if (ekf) {
        constexpr int W = sizeof(T) == 4 ? 2 : 1;   // values of a factor
        const T *fx = ekf + (sel == 1 ? 0 : W * (g.n1h + g.n2 + sh.n3)), *fy = fx + W * g.n1h;
        exy = ek_xy<T>(ek_factor(fx, kx), ek_factor(fy, ky));
        fz = fy + W * g.n2;
    }
    auto second = [&](auto qc) {
        constexpr int Q = decltype(qc)::value;
        for (int k1 = r0; k1 < sh.P; k1 += NR) {
            C v[Q], *b = buf + Q * k1 * TC + c;
#pragma unroll
            for (int j = 0; j < Q; j++) v[j] = b[j * TC];
            Dft<Q, -1, T>::run(v);
            if (ekf) {
#pragma unroll
                for (int k = 0; k < Q; k++) v[k] = scale(v[k], ek_value<T>(exy, ek_factor(fz, k1 + sh.P * k)));
            } else {
#pragma unroll
                for (int k = 0; k < Q; k++) v[k] = scale(v[k], __ldg(ek + (long)(k1 + sh.P * k) * ncol));
            }
            Dft<Q, 1, T>::run(v);
#pragma unroll
            for (int j = 0; j < Q; j++) b[j * TC] = v[j];
        }
    };
    RX_Q(ZS, Q, second);
    __syncthreads();
    auto third = [&](auto pc) {
        constexpr int P = decltype(pc)::value;
        for (int r = r0; r < sh.Q; r += NR) {
            C v[P];
            const C *b = buf + r * TC + c;
            v[0] = b[0];
#pragma unroll
            for (int k = 1; k < P; k++) v[k] = cmul(b[sh.Q * k * TC], conjg(tw[r * k]));
            Dft<P, 1, T>::run(v);
            if (ok) {
#pragma unroll
                for (int i = 0; i < P; i++) S[(long)(sh.Q * i + r) * ncol] = v[i];
            }
        }
    };
    RX_Q(ZS, P, third);
}

// z transforms of both spectra of a slice and the partial sums
// sum_k wdgsq_b(k) Re(F_qf conj F_qr) into part[((job cs + slice) ntiles +
// tile) MAXCP + b].  grid = (ceil(n1h n2 / TC), cs, njobs).
template <typename T, typename ZS, int TC, int NT>
__global__ void __launch_bounds__(NT)
    k3v_stress_z(const StressJob<T> *jobs, ZS sh, RzCols g, int s0, int cs, const cx<T> *spec, double *part)
{
    using C = cx<T>;
    const StressJob<T> &J = jobs[blockIdx.z];
    if (s0 + (int)blockIdx.y >= J.nslices) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double red[32];
    const int nb = sh.n3 * TC;
    C *buf = (C *)smem_raw, *tw = buf + 2 * nb;
    const int ncol = g.n1h * g.n2, c = threadIdx.x % TC, col = blockIdx.x * TC + c, r0 = threadIdx.x / TC;
    constexpr int NR = NT / TC;
    const bool ok = col < ncol;
    const long nk = (long)ncol * sh.n3;
    const C *S = spec + ((long)blockIdx.z * cs + blockIdx.y) * 2 * nk + (ok ? col : 0);
    for (int i = threadIdx.x; i < sh.n3; i += NT) tw[i] = ((const C *)g.twz)[i];
    const int ky = g.dn1h.div(ok ? col : 0), kx = g.cols[(ok ? col : 0) - ky * g.n1h].kx;
    __syncthreads();
    auto first = [&](auto pc) {
        constexpr int P = decltype(pc)::value;
        for (int r2 = r0; r2 < 2 * sh.Q; r2 += NR) {
            const int h = r2 >= sh.Q, r = r2 - h * sh.Q;
            C v[P];
#pragma unroll
            for (int i = 0; i < P; i++) v[i] = ok ? S[h * nk + (long)(sh.Q * i + r) * ncol] : mk<T>((T)0, (T)0);
            Dft<P, -1, T>::run(v);
            C *b = buf + h * nb + r * TC + c;
            b[0] = v[0];
#pragma unroll
            for (int k = 1; k < P; k++) b[sh.Q * k * TC] = cmul(v[k], tw[r * k]);
        }
    };
    RX_Q(ZS, P, first);
    __syncthreads();
    double acc[PSCFG_MAXCP] = {0, 0, 0, 0, 0, 0};
    const double *wd = J.wdgsq + kx + (long)g.n1h * ky;
    auto second = [&](auto qc) {
        constexpr int Q = decltype(qc)::value;
        for (int k1 = r0; k1 < sh.P; k1 += NR) {
            C a[Q], d[Q];
            const C *b = buf + Q * k1 * TC + c;
#pragma unroll
            for (int j = 0; j < Q; j++) {
                a[j] = b[j * TC];
                d[j] = b[nb + j * TC];
            }
            Dft<Q, -1, T>::run(a);
            Dft<Q, -1, T>::run(d);
            if (ok) {
#pragma unroll
                for (int k = 0; k < Q; k++) {
                    const double pr = (double)a[k].x * (double)d[k].x + (double)a[k].y * (double)d[k].y;
#pragma unroll
                    for (int p = 0; p < PSCFG_MAXCP; p++)
                        if (p < J.ncp) acc[p] += __ldg(wd + p * nk + (long)(k1 + sh.P * k) * ncol) * pr;
                }
            }
        }
    };
    RX_Q(ZS, Q, second);
#pragma unroll
    for (int p = 0; p < PSCFG_MAXCP; p++) {
        if (p >= J.ncp) break;   // uniform across the CTA
        const double tot = block_sum(acc[p], red);
        if (threadIdx.x == 0)
            part[(((long)blockIdx.z * cs + blockIdx.y) * gridDim.x + blockIdx.x) * PSCFG_MAXCP + p] = 0.25 * tot;
        __syncthreads();
    }
}

}  // namespace pscfg
