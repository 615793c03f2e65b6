"""The plane and z-line kernels of plane_rx.cuh against the FP64 oracle at
the edges of their shapes: odd and even extents, prime lines, every radix,
planes that do not divide the planes per CTA, tiles of columns that do not
divide the spectrum."""
import numpy as np
import pytest

from oracle import oracle as O
from pscf_b200.engine import CHECKPOINT, Engine, FP32, FP64
from tests.cases import diblock, omega_guess, rel_err, triblock

pytestmark = pytest.mark.gpu

# (2-D) both lines short and long, odd and even in either place
PLANES = [[2, 9], [7, 7], [8, 3], [9, 10], [10, 16], [12, 15], [15, 14], [25, 21], [27, 8], [64, 8], [8, 64], [50, 48],
          [63, 16], [64, 64]]
# (3-D) radices 2..16 along z, ragged planes per CTA
BOXES = [[8, 7, 9], [12, 10, 14], [15, 16, 12], [16, 15, 5], [9, 8, 25], [7, 2, 63], [20, 28, 27], [32, 32, 6],
         [64, 64, 3], [64, 128, 5], [10, 9, 112], [6, 5, 225], [32, 32, 32], [12, 12, 224]]


def check(s, precision, tol, seed=5):
    w = omega_guess(s, seed, 2.0)
    o = O.Oracle(s)
    rho_ref, q_ref = o.density(w)
    st_ref = np.asarray(o.stress())
    e = Engine([s, s], precision)
    rho, q = e.density(np.stack([w, w]))
    st = e.scf_stress()[1, : len(st_ref)]
    assert rel_err(q[1, :1], q_ref) < tol
    assert rel_err(rho[1], rho_ref) < tol
    qf_ref, qr_ref = o.propagators(0)
    qf, qr = e.propagators(1, 0)
    assert rel_err(qf, qf_ref) < tol and rel_err(qr, qr_ref) < tol
    assert np.max(np.abs(st - st_ref)) < 100 * tol * max(1.0, np.max(np.abs(st_ref)))
    e.close()


# FP64: rounding of six transforms a step, ~20 steps: 1e-12.  FP32: 6e-8 a
# value, transforms and ~20 steps: 2e-5.
@pytest.mark.parametrize("precision,tol", [(FP64, 1e-12), (FP32, 2e-5)])
@pytest.mark.parametrize("n", PLANES)
def test_planes_match_oracle(n, precision, tol):
    check(diblock(2, n, "rectangular", [1.6, 2.1], fA=0.35, ds=0.05, b=(1.0, 1.3)), precision, tol)


@pytest.mark.parametrize("precision,tol", [(FP64, 1e-12), (FP32, 2e-5)])
@pytest.mark.parametrize("n", BOXES)
def test_boxes_match_oracle(n, precision, tol):
    check(diblock(3, n, "orthorhombic", [1.6, 2.1, 1.9], fA=0.35, ds=0.1, b=(1.0, 1.3)), precision, tol)


@pytest.mark.parametrize("count", [37, 38, 75])
def test_planes_of_batches_match_single_ones(count):
    """The 2-D sweep's three forms (by the number of fields) agree to
    roundoff: 2 x 37 fields with two CTAs each, 2 x 38 with one, 2 x 75 with
    two CTAs to an SM."""
    for n in ([64, 64], [18, 15]):
        s = diblock(2, n, "rectangular", [1.6, 2.1], fA=0.35, ds=0.1)
        w = omega_guess(s, 4, 2.0)
        e1 = Engine([s], FP64)
        rho1, q1 = e1.density(w[None])
        e = Engine([s] * count, FP64)
        rho, q = e.density(np.stack([w] * count))
        for i in (0, count - 1):
            assert rel_err(rho[i], rho1[0]) < 1e-12 and rel_err(q[i, :1], q1[0, :1]) < 1e-12
        e.close()
        e1.close()


def test_stress_of_slices_of_very_different_size():
    """qf and qr of one slice differ by e^30 at the chain's ends: neither may
    carry the other's rounding (relative 1e-10, as for the older kernels)."""
    for dim, n, crystal, cell in ((2, [12, 10], "rectangular", [1.6, 2.1]),
                                  (3, [12, 10, 14], "orthorhombic", [1.6, 2.1, 1.9])):
        s = triblock(dim, n, crystal, cell, ds=0.02)
        w = omega_guess(s, 9, 2.0)
        w += 30.0
        o = O.Oracle(s)
        o.density(w)
        e = Engine([s], FP64)
        e.density(w[None])
        ref = np.asarray(o.stress())
        np.testing.assert_allclose(e.scf_stress()[0, : len(ref)], ref, rtol=1e-10, atol=1e-12)


@pytest.mark.parametrize("dim,n,crystal,cell", [(2, [15, 14], "rectangular", [1.6, 2.1]), (2, [12, 12], "hexagonal", [1.9]),
                                                (3, [9, 10, 7], "orthorhombic", [1.6, 2.1, 1.9])])
def test_single_steps_and_segments(dim, n, crystal, cell):
    """The step intermediates (adjoint) and checkpointed segments agree with
    the run-time shaped kernels and the stored sweep."""
    s = diblock(dim, n, crystal, cell, fA=0.35, ds=0.05)
    w = omega_guess(s, 7, 2.0)[None]
    g = omega_guess(s, 8, 1.0)[None]
    e = Engine([s], FP64)
    rho, _ = e.density(w)
    grad = e.density_adjoint(g)
    c = Engine([s], FP64 | CHECKPOINT)
    rho_c, _ = c.density(w)
    assert rel_err(rho_c, rho) < 1e-12
    assert rel_err(c.density_adjoint(g), grad) < 1e-12
    import os
    os.environ["PSCFG_GENERIC_KERNELS"] = "1"
    try:
        r = Engine([s], FP64)
    finally:
        del os.environ["PSCFG_GENERIC_KERNELS"]
    r.density(w)
    assert rel_err(r.density_adjoint(g), grad) < 1e-12
