"""Large orthogonal grids, whose k-space filters are products of 1-D factors,
against the FP64 oracle: odd and ragged extents, and a batch with cells of its
own (each with factors of its own)."""
import numpy as np
import pytest

from oracle import oracle as O
from pscf_b200.engine import CHECKPOINT, Engine, FP32, FP64
from tests.cases import diblock, omega_guess, rel_err

pytestmark = pytest.mark.gpu


# (FP64: rounding of six transforms a step, 8 steps: 1e-12; FP32: 2e-5)
@pytest.mark.parametrize("precision,tol", [(FP64, 1e-12), (FP32, 2e-5), (FP64 | CHECKPOINT, 1e-12), (FP32 | CHECKPOINT, 2e-5)])
@pytest.mark.parametrize("n", [[63, 70, 60], [64, 54, 80], [45, 75, 84]])
def test_large_orthogonal_grids_match_oracle(n, precision, tol):
    ss = [diblock(3, n, "orthorhombic", [1.6 + 0.1 * i, 2.1, 1.9 - 0.1 * i], fA=0.5, ds=0.125, b=(1.0, 1.3))
          for i in range(2)]
    w = np.stack([omega_guess(s, 5 + i, 2.0) for i, s in enumerate(ss)])
    e = Engine(ss, precision)
    rho, q = e.density(w)
    e.close()
    for i, s in enumerate(ss):
        rho_ref, q_ref = O.Oracle(s).density(w[i])
        assert rel_err(q[i, :1], q_ref) < tol
        assert rel_err(rho[i], rho_ref) < tol
