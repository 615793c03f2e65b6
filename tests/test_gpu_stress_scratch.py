"""Device memory that the stress of a large batch takes for its spectra."""
import numpy as np
import pytest

from pscf_b200.engine import Engine, FP64
from pscf_b200.system import Chain
from tests.cases import diblock, omega_guess, rel_err

pytestmark = pytest.mark.gpu


def test_stress_of_a_large_batch_keeps_to_its_scratch():
    """320 chains of 64^3: one slice's spectra of all of them are 1.4 GB, and
    the scratch at most 1 GB (the partial sums and the allocator's rounding:
    64 MB)."""
    import torch
    s = diblock(3, [64, 64, 64], "cubic", [1.9], ds=0.5)
    s.chains = [Chain([i % 2], [1.0], phi=0.25) for i in range(4)]
    w = np.stack([omega_guess(s, 5, 2.0) * (1.0 + 0.003 * i) for i in range(80)])
    e = Engine([s] * 80, FP64)
    e.density(w)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    st = e.scf_stress()
    taken = before - torch.cuda.mem_get_info()[0]
    e.close()
    assert taken < (1 << 30) + (64 << 20)
    for i in (0, 61, 62, 79):   # (a group holds the chains of 62 instances)
        e = Engine([s], FP64)
        e.density(w[i : i + 1])
        assert rel_err(st[i, :1], e.scf_stress()[0, :1]) < 1e-11
        e.close()
