"""1-D sweeps with the step as a dense matrix (up to 128 points) against the
FP64 oracle, at the edges of its size classes and of the class above."""
import numpy as np
import pytest

from oracle import oracle as O
from pscf_b200.engine import CHECKPOINT, Engine, FP32, FP64
from tests.cases import diblock, omega_guess, rel_err

pytestmark = pytest.mark.gpu


# FP64: a step's rounding is ~1e-16 N^(1/2) and ~100 steps add up: 1e-12.
# FP32 slabs: slices are rounded to 6e-8 once per step, ~100 steps: 2e-5.
@pytest.mark.parametrize("n", [2, 3, 7, 8, 30, 32, 35, 63, 64, 70, 125, 128, 135])
@pytest.mark.parametrize("precision,tol", [(FP64, 1e-12), (FP32, 2e-5)])
def test_dense_sweep_matches_oracle(n, precision, tol):
    ss = [diblock(1, [n], "lamellar", [1.5 + 0.2 * i], fA=0.3 + 0.1 * i, chiN=15.0, b=(1.0, 1.2)) for i in range(2)]
    w = np.stack([omega_guess(s, 3 + i, 2.0) for i, s in enumerate(ss)])
    e = Engine(ss, precision)
    rho, q = e.density(w)
    st = e.scf_stress()
    for i, s in enumerate(ss):
        o = O.Oracle(s)
        rho_ref, q_ref = o.density(w[i])
        st_ref = o.stress()
        assert rel_err(q[i, :1], q_ref) < tol
        assert rel_err(rho[i], rho_ref) < tol
        qf_ref, qr_ref = o.propagators(0)
        qf, qr = e.propagators(i, 0)
        assert rel_err(qf, qf_ref) < tol and rel_err(qr, qr_ref) < tol
        assert abs(st[i, 0] - st_ref[0]) < 100 * tol * max(1.0, abs(st_ref[0]))


def test_dense_sweep_segments_repeat_the_sweep():
    s = diblock(1, [40], "lamellar", [1.7], fA=0.35, chiN=18.0)
    w = omega_guess(s, 9, 2.0)[None]
    rho, q = Engine([s], FP64).density(w)
    rho_c, q_c = Engine([s], FP64 | CHECKPOINT).density(w)
    assert rel_err(rho_c, rho) < 1e-13 and rel_err(q_c[:, :1], q[:, :1]) < 1e-13
