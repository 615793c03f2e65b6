"""Mixed-precision solves of a grid whose FP32 phase runs the plane kernels:
every solve of a batch ends in the basin of its FP64 one."""
import numpy as np
import pytest

from pscf_b200.engine import Engine, FP64, MIXED
from tests.cases import BCC_SITES, diblock, sphere_guess

pytestmark = pytest.mark.gpu


def test_mixed_solves_keep_their_basins():
    """24 BCC solves of 24^3.  Stopped at a field error of 1e-6, a free energy
    is off by less than the fields' size times it, some 1e-4; another basin is
    0.1 away."""
    ss = [diblock(3, [24] * 3, "cubic", [1.9], fA=0.25, chiN=18.0 + 0.25 * i, ds=0.05) for i in range(24)]
    w = np.stack([sphere_guess(s, 0.25, BCC_SITES, 0.08) for s in ss])
    out = []
    for precision, switch in ((FP64, 0.0), (MIXED, 1e-3)):
        e = Engine(ss, precision)
        out.append(e.iterate_am(w, error_max=1e-6, max_itr=300, switch_error=switch)[2])
        e.close()
    assert all(r["itr_fp32"] > 0 for r in out[1])
    for a, b in zip(*out):
        assert a["converged"] and b["converged"]
        assert abs(a["f_helmholtz"] - b["f_helmholtz"]) < 1e-3
