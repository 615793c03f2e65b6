"""1-D chains of short blocks, where the dense step's matrix is not worth its
making: results against the FP64 oracle on both sides of the rule, and no
slower than the run-time shaped kernel."""
import numpy as np
import pytest

from oracle import oracle as O
from pscf_b200.engine import CHECKPOINT, Engine, FP64
from pscf_b200.system import Chain
from tests.cases import diblock, omega_guess, rel_err

pytestmark = pytest.mark.gpu


def multiblock(n, steps):
    """Eight alternating blocks of `steps` contour steps each."""
    s = diblock(1, [n], "lamellar", [1.6], ds=1.0 / (8 * steps), b=(1.0, 1.2))
    s.chains = [Chain([i % 2 for i in range(8)], [0.125] * 8)]
    return s


# rounding of a step ~1e-16 N^(1/2), at most 80 steps: 1e-12
@pytest.mark.parametrize("count", [1, 100])
@pytest.mark.parametrize("n,steps", [(30, 2), (64, 2), (64, 4), (70, 2), (70, 4), (128, 2), (128, 6), (128, 10)])
def test_short_blocks_match_oracle(n, steps, count):
    s = multiblock(n, steps)
    w = np.stack([omega_guess(s, 3 + (i > 0), 2.0) for i in range(count)])
    for precision in (FP64, FP64 | CHECKPOINT):
        e = Engine([s] * count, precision)
        rho, q = e.density(w)
        e.close()
        for i in {0, count - 1}:
            rho_ref, q_ref = O.Oracle(s).density(w[i])
            assert rel_err(q[i, :1], q_ref) < 1e-12
            assert rel_err(rho[i], rho_ref) < 1e-12


def sweep_ms(e, w):
    before = e.profile()["sweep_ms"]
    e.density(w)
    return e.profile()["sweep_ms"] - before


# A quarter above the other kernel is timing noise, of the least of both
# sides' sweeps, taken in turn; the dense step takes 2.2 (one instance) to 4
# times as long here (96).
@pytest.mark.parametrize("n,count", [(128, 1), (128, 96), (70, 96)])
def test_short_blocks_are_not_slower_than_the_general_kernel(n, count, monkeypatch):
    s = multiblock(n, 2)
    w = np.stack([omega_guess(s, 3, 2.0)] * count)
    e = Engine([s] * count, FP64)
    monkeypatch.setenv("PSCFG_GENERIC_KERNELS", "1")
    g = Engine([s] * count, FP64)
    times, general = [], []
    for x in (e, g):
        x.set_profiling(True)
        x.density(w)
    for _ in range(60):
        times.append(sweep_ms(e, w))
        general.append(sweep_ms(g, w))
        if len(times) >= 15 and min(times) < 1.25 * min(general):
            break
    e.close()
    g.close()
    assert min(times) < 1.25 * min(general)
