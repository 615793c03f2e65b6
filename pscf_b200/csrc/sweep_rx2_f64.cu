// plane_rx.cuh kernels for dim 2 in FP64, and the shapes all of them take.
#include "sweep_rx.inl"

namespace pscfg {

static bool has_radix(int r, bool first) { return (r >= 1 && r <= 10) || (!first && (r == 12 || r == 14 || r == 15 || r == 16)); }

// N = P Q with the least P + Q; rows and z lines want the wider second
// factor (consecutive threads load Q consecutive points), columns an even P
// (rows go in pairs of one residue class); first factors above 8 only where
// there is no other.
static bool split(int n, bool first_small, bool even, int &P, int &Q)
{
    int best = 1 << 30;
    for (int p = 1; p <= 16; p++) {
        if (n % p || !has_radix(p, first_small) || !has_radix(n / p, false)) continue;
        const int q = n / p;
        const int cost = 4 * (p + q) + (even && (p & 1) && p > 1 ? 8 : 0) + (!even && q < p ? 1 : 0) + (first_small && p > 8 ? 100 : 0);
        if (cost < best) {
            best = cost;
            P = p;
            Q = q;
        }
    }
    return best < (1 << 30);
}

bool rx_shape(int dim, const int n[3], RxPlan &p, RxCol *cols, bool f32)
{
    RxShape &s = p.sh;
    s.n1 = n[0];
    s.n2 = n[1];
    p.n3 = n[2];
    s.n1h = s.n1 / 2 + 1;
    s.nc = (s.n1 + 1) / 2;
    p.plane = dim >= 2 && split(s.n1, true, false, s.P1, s.Q1) && split(s.n2, true, true, s.P2, s.Q2) &&
              s.n1 * s.n2 < 65536 / 2;
    if (!p.plane) return false;
    s.HP = (s.P2 + 1) / 2;
    s.LS = rx_stride(s.n1);
    s.dQ1 = RDiv::of(s.Q1);
    s.dn1h = RDiv::of(s.n1h);
    s.dnc = RDiv::of(s.nc);
    s.dQ2 = RDiv::of(s.Q2);
    s.dP2 = RDiv::of(s.P2);
    int c = 0;
    auto slot = [&](int kx) {
        return f32 ? rx_slot<float>(s.Q1, kx % s.P1, kx / s.P1) : rx_slot<double>(s.Q1, kx % s.P1, kx / s.P1);
    };
    auto add = [&](int kx) {
        RxCol &k = cols[c++];
        k.kx = (short)kx;
        k.pos = (short)slot(kx);
        k.ppos = (short)slot((s.n1 - kx) % s.n1);
        k.wpos = kx == 0 ? (short)s.n1 : 2 * kx == s.n1 ? (short)(s.n1 + 1) : k.ppos;
    };
    for (int k1 = 0; k1 < s.P1; k1++)
        for (int kx = k1; 2 * kx < s.n1; kx += s.P1) add(kx);
    if (s.n1 % 2 == 0) add(s.n1 / 2);
    p.z.n3 = p.n3;
    p.line = dim == 3 && split(p.n3, false, false, p.z.Q, p.z.P);   // (the first pass loads P points a thread: the wider one)
    for (RzCols &g : p.zc) {
        g.n1h = s.n1h;
        g.n2 = s.n2;
        g.dn1h = s.dn1h;
    }
    return true;
}

RX2_INSTANCES(double)

}  // namespace pscfg
