"""Planes per CTA of the register sweep: the measured choice of the grids that
run it (16^3; 32^3 in FP32), and what pscfg_sweep_planes reports."""
import numpy as np
import pytest

from pscf_b200.engine import Engine, FP32, FP64
from tests.cases import diblock, omega_guess

pytestmark = pytest.mark.gpu


def systems(n):
    ss = [diblock(3, [n] * 3, "cubic", [2.4], fA=0.25 + 0.02 * i, chiN=20.0, ds=0.02) for i in range(3)]
    return ss, np.stack([omega_guess(s, 40 + i, 2.0) for i, s in enumerate(ss)])


@pytest.mark.parametrize("n,precision,choices", [(16, FP64, (1, 2, 4, 8)), (16, FP32, (1, 2, 4, 8)), (32, FP32, (1, 2, 4))])
def test_every_density_comes_from_the_measured_count(n, precision, choices):
    """One timed trial sweep per candidate, then the chosen count: repeated
    calls are bit-identical."""
    ss, w = systems(n)
    e = Engine(ss, precision)
    outs = [e.density(w)[0] for _ in range(5)]
    p = e.sweep_planes(2 * len(ss), precision == FP32)
    e.close()
    assert p in choices
    for o in outs[1:]:
        assert np.array_equal(o, outs[0])


@pytest.mark.parametrize("n,forced", [(16, 8), (16, 2), (32, 4), (32, 1), (32, -1)])
def test_a_forced_count_is_reported(n, forced, monkeypatch):
    monkeypatch.setenv("PSCFG_PLANES", str(forced))
    ss, w = systems(n)
    e = Engine(ss, FP64)
    e.density(w)
    assert e.sweep_planes(2 * len(ss)) == forced
    e.close()
