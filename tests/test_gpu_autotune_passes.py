"""The autotuner times plain forward passes; its choice leaves the gradient's passes as they run without one."""
import numpy as np
import pytest

import dsh
from test_gpu_parity import _case, engine_from

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,fdo", [(720, 380, 4), (700, 400, 2), (160, 80, 4)])
def test_gradient_passes_after_autotuning(nx, ny, fdo):
    """Beyond 262144 points the storing and adjoint passes run the kernel pair, whatever was picked for forward passes; a
    small grid keeps the blocked pass where the tuner picked a launch that only serves forward passes."""
    nt = 64
    d, shots = _case(5300 + nx, nx=nx, ny=ny, nt=nt, fdo=fdo, L=0, fs=1, fw=10)
    i, j = int(shots[0].srcpos[0, 0]), int(shots[0].srcpos[1, 0])
    shots = [dsh.Shot(shots[0].srcpos, np.array([[i - 3, i - 1, i, i - 2], [j, j, j + 2, j + 3]], np.int32))]   # signals arrive
    out, launches = [], []
    for tune in (False, True):
        with engine_from(d) as e:
            if tune:
                choice, _ = e.autotune(shots, nsteps=nt)
            seis = e.forward(shots)
            obs = [s * np.float32(0.6) for s in seis]
            out.append((seis[0], e.gradient(shots, obs)))
            launches.append(e.stats()["kernel_launches"])
    assert np.array_equal(out[0][0], out[1][0]) and np.isfinite(out[0][1]["g_vs"]).all()
    assert all(np.array_equal(out[0][1][k], out[1][1][k]) for k in ("g_vs", "g_rho"))
    if choice in ("persistent launch", "cluster-resident launch", "temporally blocked launch"):
        assert launches[0] == launches[1]
    assert (launches[0] > 2 * 2 * nt) == (nx * ny > 1 << 18)
    print("picked", choice, "launches", launches)
