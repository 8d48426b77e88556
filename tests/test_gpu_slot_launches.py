"""Launches of several shot slots: the halves on two streams and the groups that stay in L2."""
import os
import subprocess
import sys

import numpy as np
import pytest

import dsh
import oracle as O
from conftest import oracle_model
from test_gpu_parity import _case, _oracle_gradient, engine_from
from test_gpu_qgrad import _oracle_q

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


# Halves and groups of slots of every size: DSH_SLOT_SPLIT and DSH_SLOT_GROUP_MB are read once per process, so the cases run
# in child processes that set them (and here as the sizes decide: all slots in one launch).
SPLITS = [(3, 4, 0), (5, 8, 2), (7, 6, 1)]          # slots, FDORDER, L


def _slots_case(n, fdo, L):
    d, _ = _case(5400 + n, nx=211, ny=151, nt=45, fdo=fdo, L=L, fs=n % 2, fw=8)
    shots = []
    for s in range(n):
        sp = np.array([[20 + 13 * s], [3 + s % 2], [0], [-0.01], [60.0], [1.0 + s], [0], [3]], np.float32)
        x = np.clip(20 + 13 * s + np.arange(-4, 5 + s % 3), 1, 211)
        shots.append(dsh.Shot(sp, np.array([x, 1 + np.arange(x.size) % 5], np.int32)))
    return d, shots


@pytest.mark.parametrize("n,fdo,L", SPLITS)
def test_every_pass_of_several_slots(n, fdo, L):
    """Forward modelling, gradients with full storage and with checkpoints, raw energies, Hessian sums and the Qs gradient:
    the values of each slot against the oracle's shot, bit for bit; a second launch of fewer slots too."""
    d, shots = _slots_case(n, fdo, L)
    m = oracle_model(d)
    seis, obs, ws, wr, hu, hr = [], [], [], [], [], []
    for sh in shots:
        o = O.Oracle(m, "port")
        seis.append(o.forward(sh.srcpos, sh.recpos))
        obs.append((seis[-1] * np.float32(0.7)).astype(np.float32))
        o.close()
        o = O.Oracle(m, "port")
        g = o.shot_gradient(sh.srcpos, sh.recpos, obs[-1])
        ws.append(g["Ws"]), wr.append(g["Wr"])
        o.close()
        o = O.Oracle(m, "port")
        o.forward(sh.srcpos, sh.recpos, hessian=True)
        hu.append(o.field("hess_u")), hr.append(o.field("hess_rho"))
        o.close()
    gv, gr, l2, _ = _oracle_gradient(d, shots, obs)
    with engine_from(d, max_shots=n) as e:
        e.set_step_variant(0)
        got = e.forward(shots)
        per_step = e.stats()["kernel_launches"] // d["nt"]
        fewer = e.forward(shots[1:3])
        out = e.gradient(shots, obs, want_energy=True)
        e.hessian_diag(shots)
        hess = [(e.field("hess_u", shot=s), e.field("hess_rho", shot=s)) for s in range(n)]
    assert all(np.array_equal(a, b) for a, b in zip(got, seis))
    assert all(np.array_equal(a, b) for a, b in zip(fewer, seis[1:3]))
    mb, split = os.environ.get("DSH_SLOT_GROUP_MB"), os.environ.get("DSH_SLOT_SPLIT") == "1"
    if mb is None or mb == "0":                      # launches per step: the pair, in each half or group
        assert per_step == (2 * n if mb == "0" else 4 if split else 2)
    assert np.isfinite(gv).all() and np.array_equal(out["g_vs"], gv) and np.array_equal(out["g_rho"], gr)
    assert all(np.array_equal(out["Ws"][s], ws[s]) and np.array_equal(out["Wr"][s], wr[s]) for s in range(n))
    assert all(np.array_equal(hess[s][0], hu[s]) and np.array_equal(hess[s][1], hr[s]) for s in range(n))
    with engine_from(d, max_shots=n, ckpt_every=11) as e:
        e.set_step_variant(0)
        out = e.gradient(shots, obs)
    assert np.array_equal(out["g_vs"], gv) and np.array_equal(out["g_rho"], gr)
    if L:
        q = []
        for slots, extra in ((1, {}), (n, {}), (n, {"ckpt_every": 11})):
            with engine_from(d, max_shots=slots, grad_q=1, **extra) as e:
                e.gradient(shots, obs)
                q.append(e.gradient_q())
        ref = sum(_oracle_q(d, [sh], [ob]) for sh, ob in zip(shots, obs))
        assert np.array_equal(q[0], q[1]) and np.array_equal(q[0], q[2])
        assert np.abs(q[0].astype(np.float64) - ref).max() <= 1e-5 * np.abs(ref).max()    # float sums over shots


@pytest.mark.parametrize("env", [{"DSH_SLOT_SPLIT": "1"}, {"DSH_SLOT_GROUP_MB": "0"},
                                 {"DSH_SLOT_GROUP_MB": "1", "DSH_SLOT_SPLIT": "1"},
                                 {"DSH_SLOT_GROUP_MB": "2", "DSH_SLOT_SPLIT": "1"},
                                 {"DSH_SLOT_GROUP_MB": "2", "DSH_SLOT_SPLIT": "0", "DSH_NO_GRAPHS": "1"}])
def test_halves_and_groups_in_subprocess(env):
    """Halves of an odd number of slots; groups of one slot; groups of up to 1 or 2 MB of fields (one to three slots, 127 KB
    per field and slot, a shorter last group among them), with and without halves."""
    code = ("import sys; sys.argv=['x']; import pytest; "
            "sys.exit(pytest.main(['-q', '-p', 'no:cacheprovider', '-m', 'gpu', "
            "'tests/test_gpu_slot_launches.py::test_every_pass_of_several_slots']))")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, **env), capture_output=True, text=True,
                         timeout=600)
    assert out.returncode == 0, out.stdout[-2000:] + out.stderr[-2000:]


def test_large_batch_model_equals_the_oracle():
    """A batch model of 786432 points or more over its shots runs through its context's own launches, here as two halves of
    one and two slots; the other model through the common ones."""
    members = [_case(5500, nx=655, ny=421, nt=30, fdo=4, L=2, fs=1, fw=10, nshots=3),
               _case(5501, nx=45, ny=37, nt=40, fdo=8, L=0, fs=0, fw=8, nshots=2)]
    members = [(d, [dsh.Shot(s.srcpos, np.array([s.srcpos[0, 0] + [-2, 0, 1], [1, 2, 4]], np.float32).clip(1, 45 if d["nx"] == 45 else 655)
                             .astype(np.int32)) for s in shots]) for d, shots in members]
    params = [dsh.make_params(nx=d["nx"], ny=d["ny"], nt=d["nt"], dh=d["dh"], dt=float(d["dt"]), fdorder=d["fdorder"],
                              fw=d["fw"], free_surf=d["free_surf"], l=d["l"], fl=tuple(float(x) for x in d["fl"]),
                              damping=float(d["damping"]), fpml=float(d["fpml"]), max_shots=len(s)) for d, s in members]
    with dsh.Batch(params) as b:
        for k, (d, _) in enumerate(members):
            b.set_model(k, d["vs"], d["rho"], d["qs"] if d["l"] else None)
        got = b.forward([s for _, s in members])
        assert b.stats()["kernel_launches"] > 4 * 30
    for (d, shots), seis in zip(members, got):
        for sh, s in zip(shots, seis):
            o = O.Oracle(oracle_model(d), "port")
            ref = o.forward(sh.srcpos, sh.recpos)
            o.close()
            assert np.abs(ref).max() > 0 and np.array_equal(s, ref)
