"""Solves of batches with more fields than a launch has blocks in y."""
import numpy as np
import pytest

from pscf_b200.engine import Engine, FP64
from pscf_b200.system import Chain, Solvent, System
from tests.cases import omega_guess, rel_err

pytestmark = pytest.mark.gpu


def test_solve_with_more_than_65535_fields():
    """16400 instances of four monomers, 65600 fields; one iteration, the
    first, a middle and the last instance as alone (rounding of sums over 4
    points and 4 steps: 1e-12)."""
    chi = np.array([[0, 12.0, 18.0, 9.0], [12.0, 0, 14.0, 20.0], [18.0, 14.0, 0, 11.0], [9.0, 20.0, 11.0, 0]])
    s = System(dim=1, ngrid=[4], crystal_system="lamellar", cell_param=[1.6], kuhn=[1.0, 1.1, 0.9, 1.2], chi=chi,
               chains=[Chain([0, 1], [0.5, 0.5], phi=0.7)],
               solvents=[Solvent(monomer=2, size=0.1, phi=0.2), Solvent(monomer=3, size=0.15, phi=0.1)], ds=0.25)
    count = 16400
    w = omega_guess(s, 5, 1.0)[None] * (1.0 + 0.2 * np.arange(count)[:, None, None] / count)
    kw = dict(error_max=1e-12, max_itr=1, n_hist=2)
    e = Engine([s] * count, FP64)
    om, rho, _ = e.iterate_am(w, **kw)
    e.close()
    e = Engine([s], FP64)
    for i in (0, count // 2, 16384, count - 1):
        om1, rho1, _ = e.iterate_am(w[i : i + 1], **kw)
        assert rel_err(om[i], om1[0]) < 1e-12 and rel_err(rho[i], rho1[0]) < 1e-12
    e.close()
