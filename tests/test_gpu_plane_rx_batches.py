"""The plane and z-line kernels on batches: several planes to a CTA with a
last CTA that holds fewer, fields in more than one group, wide z tiles and
sweeps launched without a graph.  Every instance has fields of its own, so
that a wrong plane, field or group offset shows."""
import numpy as np
import pytest

from oracle import oracle as O
from pscf_b200.engine import Engine, FP32, FP64
from tests.cases import diblock, omega_guess, rel_err

pytestmark = pytest.mark.gpu


def batch(n, count, ds):
    s = diblock(3, n, "orthorhombic", [1.6, 2.1, 1.9], fA=0.5, ds=ds, b=(1.0, 1.3))
    w = np.stack([omega_guess(s, 5, 2.0) * (1.0 + 0.3 * i / count) for i in range(count)])
    return s, w


# 9 x 10 x 7 x 150: 6 planes to a CTA, 1 in the last; 20 x 12 x 21 x 60: 4 and
# 1; 12 x 10 x 15 x 100: 7 and 1 (the launches hold half the
# fields).  32^3 x 40 and 64^3 x 5: two groups of fields, 32 columns to a z
# tile, no graph.  FP64: rounding of a few steps of six transforms: 1e-12.
# FP32: 2e-5.
@pytest.mark.parametrize("precision,tol", [(FP64, 1e-12), (FP32, 2e-5)])
@pytest.mark.parametrize("n,count,ds", [([9, 10, 7], 150, 0.125), ([20, 12, 21], 60, 0.125), ([12, 10, 15], 100, 0.125),
                                        ([32, 32, 32], 40, 0.25), ([64, 64, 64], 5, 0.25)])
def test_batches_match_oracle(n, count, ds, precision, tol):
    s, w = batch(n, count, ds)
    e = Engine([s] * count, precision)
    rho, q = e.density(w)
    st = e.scf_stress()
    e.close()
    for i in (0, 1, count // 2 - 1, count // 2, count - 1):
        o = O.Oracle(s)
        rho_ref, q_ref = o.density(w[i])
        st_ref = np.asarray(o.stress())
        assert rel_err(q[i, :1], q_ref) < tol
        assert rel_err(rho[i], rho_ref) < tol
        assert np.max(np.abs(st[i, : len(st_ref)] - st_ref)) < 100 * tol * max(1.0, np.max(np.abs(st_ref)))


# (the adjoint of one instance alone takes one plane to a CTA; 1e-12 of
# rounding through twice the steps)
@pytest.mark.parametrize("n,count", [([9, 10, 7], 160), ([20, 12, 21], 60)])
def test_adjoints_of_batches_match_single_ones(n, count):
    s, w = batch(n, count, 0.125)
    g = np.stack([omega_guess(s, 8, 1.0) * (1.0 - 0.3 * i / count) for i in range(count)])
    e = Engine([s] * count, FP64)
    e.density(w)
    grad = e.density_adjoint(g)
    e.close()
    for i in (0, count // 2, count - 1):
        e = Engine([s], FP64)
        e.density(w[i : i + 1])
        assert rel_err(grad[i], e.density_adjoint(g[i : i + 1])[0]) < 1e-12
        e.close()
