"""Several contexts on one device: a small grid's pass is one blocked launch while the device is its own, and the kernel
pair, whose launches overlap with the others', while another context's call is in flight."""
import threading

import numpy as np
import pytest

import dsh
from test_gpu_parity import _case, engine_from

pytestmark = pytest.mark.gpu


def _inside(d, shots):
    return [dsh.Shot(s.srcpos, np.clip(s.recpos, 1, None)) for s in shots]


@pytest.mark.parametrize("variant,nx,ny,nt", [(0, 160, 80, 100000), (5, 500, 200, 150000)])
def test_blocked_pass_beside_another_call(variant, nx, ny, nt):
    """The other call, some 0.4 s long: step kernels, then a blocked pass that leaves too few SMs."""
    d, shots = _case(5600, nx=160, ny=80, nt=90, fdo=4, L=0, fs=1, fw=10)
    shots = _inside(d, shots)
    other, oshots = _case(5601, nx=nx, ny=ny, nt=nt, fdo=4, L=0, fs=1, fw=10)
    oshots = _inside(other, oshots)
    seen = []
    with engine_from(d) as e, engine_from(other) as o:
        o.set_step_variant(variant)
        alone = e.forward(shots)[0]
        assert e.stats()["kernel_launches"] < 90
        t = threading.Thread(target=o.forward, args=(oshots,))
        t.start()
        while t.is_alive():
            assert np.array_equal(e.forward(shots)[0], alone)
            seen.append(e.stats()["kernel_launches"])
        t.join()
        assert np.array_equal(e.forward(shots)[0], alone)
        assert e.stats()["kernel_launches"] < 90          # the device is free again
    assert max(seen) >= 2 * 90
