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


def test_profile_of_more_steps_than_a_launch_word_counts():
    """dsh_profile_step over 66000 steps (a launch names its step in 16 bits beside its first slot), and of slots that run as
    halves; the next run is unaffected."""
    d, shots = _case(5200, nx=40, ny=32, nt=66000, fdo=4, L=1, fs=1, fw=6, nshots=2)
    d["dt"] = np.float32(1e-6)
    with engine_from(d, max_shots=2) as e:
        e.set_step_variant(0)
        ref = e.forward(shots)
        prof = e.profile_step("forward", 66000)
        again = e.forward(shots)
    assert prof["v_step"] > 0 and prof["s_step"] > 0
    assert all(np.array_equal(a, b) for a, b in zip(ref, again))
    d, shots = _case(5201, nx=512, ny=260, nt=40, fdo=4, L=1, fs=1, fw=10, nshots=3)
    with engine_from(d, max_shots=3) as e:
        seis = e.forward(shots)
        e.gradient(shots, seis)
        for name in ("forward", "forward_store", "forward_hessian", "adjoint"):
            prof = e.profile_step(name, 10)
            assert prof["v_step"] > 0 and prof["s_step"] > 0, name
        again = e.forward(shots)
    assert all(np.array_equal(a, b) for a, b in zip(seis, again))
