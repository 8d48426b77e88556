"""Launches of several shot slots: the halves on two streams and the groups that stay in L2."""
import numpy as np
import pytest

import dsh
from test_gpu_parity import _case, engine_from

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nshots", [1, 3])
def test_launches_are_counted(nshots):
    """One slot: a velocity and a stress launch per step and a counter update per chunk of 32 steps, replayed from two
    graphs; three slots of this size run as halves of one and two, four launches per step."""
    nt = 70
    d, shots = _case(5100, nx=512, ny=260, nt=nt, fdo=4, L=1, fs=1, fw=10, nshots=nshots)
    shots = [dsh.Shot(s.srcpos, np.clip(s.recpos, 1, None)) for s in shots]      # inside the grid: no separate injection
    with engine_from(d, max_shots=nshots) as e:
        e.forward(shots)
        n = e.stats()["kernel_launches"]
    steps = (2 if nshots == 1 else 4) * nt
    assert steps + 4 <= n <= steps + 12          # + the counter (set, 3 updates) and the seismograms' way out
