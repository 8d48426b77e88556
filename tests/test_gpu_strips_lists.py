"""CPML strips, divisions by DH, and the source / receiver lists of the step kernels where they can go wrong, against
the CPU oracle, bit for bit: strips that meet or overlap in a thread's four points (NX < 2 FW + 3, NY < 2 FW), stretching
factors K other than 1, DH that is no power of two, several sources at one point and at neighbouring points, more than 32
receivers in a row, receivers that share a point, several shots per launch with an idle slot, uneven batches."""
import numpy as np
import pytest

import dsh
import oracle as O

pytestmark = pytest.mark.gpu

CASES = [  # nx, ny, fw, fdorder, L, free_surf, dh, k_max, nrow
    (53, 41, 8, 4, 0, 0, 0.6, 1.0, 40),
    (45, 37, 22, 8, 2, 0, 0.6, 1.0, 20),
    (30, 26, 20, 6, 1, 0, 3.0, 1.0, 7),
    (61, 33, 10, 10, 0, 1, 1.1, 1.5, 33),
    (141, 21, 6, 4, 3, 0, 0.7, 2.0, 70),
    (262, 19, 5, 8, 0, 1, 0.5, 3.0, 131),
    (21, 10050, 4, 2, 0, 1, 0.5, 1.0, 9),   # more rows than one block of the vs / rho means holds
]


def _case(nx, ny, fw, fdo, L, fs, dh, k_max, nrow, seed):
    rng = np.random.default_rng(seed)
    vs = (200.0 + 40.0 * rng.standard_normal((ny, nx))).clip(120, 320).astype(np.float32)
    rho = (1800.0 + 80.0 * rng.standard_normal((ny, nx))).astype(np.float32)
    qs = rng.uniform(20.0, 60.0, (ny, nx)).astype(np.float32) if L else None
    kw = dict(nx=nx, ny=ny, nt=110, dh=dh, dt=float(np.float32(2e-4 * dh)), fdorder=fdo, fw=fw, free_surf=fs, l=L,
              fl=(7.5, 30.0, 120.0)[:L], damping=320.0, fpml=30.0, k_max_pml=k_max)
    shots = []
    for s in range(3):
        i = 6 + 7 * s
        src = np.zeros((8, 6), np.float32)
        src[7] = 3
        for k, (x, y, amp) in enumerate([(i, 3, 1.0), (i, 3, -0.5), (i + 1, 3, 0.3), (nx - 1, 3, 0.7), (2, ny - 1, 0.4),
                                         (i, 3, 0.2)]):
            src[:6, k] = [x, y, 0, -0.01 * k, 60.0 + 3 * k, amp]
        x = np.linspace(1, nx, nrow).round().astype(np.int32)
        rec = np.concatenate([[x, np.full(nrow, 2)], [x[:3], np.full(3, 2)], [[1, nx], [ny, ny]]], 1).astype(np.int32)
        shots.append(dsh.Shot(src, rec))
    return kw, vs, rho, qs, shots


def _model(kw, vs, rho, qs):
    return O.Model(vs=vs, rho=rho, qs=qs, **kw)


@pytest.mark.parametrize("case", CASES)
def test_forward_gradient_and_hessian(case):
    kw, vs, rho, qs, shots = _case(*case, seed=case[0])
    m = _model(kw, vs, rho, qs)
    ref, obs = [], []
    for sh in shots:
        o = O.Oracle(m, "port")
        ref.append(o.forward(sh.srcpos, sh.recpos))
        o.close()
        obs.append((ref[-1] * np.float32(0.6) + np.float32(1e-3)).astype(np.float32))
    su, sr = np.zeros((m.ny, m.nx), np.float32), np.zeros((m.ny, m.nx), np.float32)
    for sh, ob in zip(shots, obs):
        o = O.Oracle(m, "port")
        g = o.shot_gradient(sh.srcpos, sh.recpos, ob)
        su, sr = su + g["g_u"], sr + g["g_rho"]
        o.close()
    o = O.Oracle(m, "port")
    gv, gr = o.convert(su, sr)
    o.close()
    for extra, variant in (({}, 0), ({"ckpt_every": 17}, 0), ({}, 5), ({"ckpt_every": 17}, 5), ({}, -1)):
        with dsh.Engine(dsh.make_params(max_shots=2, **kw, **extra)) as e:
            e.set_model(vs, rho, qs)
            e.set_step_variant(variant)
            seis = e.forward(shots)
            out = e.gradient(shots, obs)
        assert all(np.array_equal(a, b) for a, b in zip(seis, ref))
        assert np.array_equal(out["g_vs"], gv) and np.array_equal(out["g_rho"], gr)


@pytest.mark.parametrize("variant", [1, 2, 3, 4, 5])
def test_variants_agree_with_the_pair(variant):
    """The opt-in step kernels on the case with neighbouring sources and K != 1 (4 and 5 serve elastic models only;
    where a variant does not apply the engine runs the pair)."""
    for case in (CASES[0], CASES[4], CASES[5]):
        kw, vs, rho, qs, shots = _case(*case, seed=11)
        with dsh.Engine(dsh.make_params(max_shots=3, **kw)) as e:
            e.set_model(vs, rho, qs)
            e.set_step_variant(0)
            ref = e.forward(shots)
            e.set_step_variant(variant)
            got = e.forward(shots)
        assert all(np.array_equal(a, b) for a, b in zip(got, ref))


@pytest.mark.parametrize("fdo,k,rows", [(4, 4, 8), (4, 4, 16), (4, 4, 40), (4, 4, 48), (8, 2, 8), (8, 2, 32), (2, 8, 8),
                                        (6, 3, 8), (6, 2, 48)])
def test_blocked_pass_of_each_block_size(fdo, k, rows, monkeypatch):
    """Blocks of 448, 576, 896, 1024 (FDORDER 4), 576, 960 (8), 288 (2), 608 and 960 (6) threads: the three builds in the
    forward, storing and adjoint modes against the kernel pair."""
    monkeypatch.setenv("DSH_TB_STEPS", str(k))
    monkeypatch.setenv("DSH_TB_ROWS", str(rows))
    kw, vs, rho, _, shots = _case(203, 97, 10, fdo, 0, 1, 0.6, 1.0, 40, seed=fdo)
    res = []
    with dsh.Engine(dsh.make_params(max_shots=1, **kw)) as e:
        e.set_model(vs, rho)
        for variant in (0, 5):
            e.set_step_variant(variant)
            seis = e.forward(shots)
            launches = e.stats()["kernel_launches"]
            g = e.gradient(shots, [x * np.float32(0.6) for x in seis])
            res.append((seis, g["g_vs"], g["g_rho"], g["l2"], launches))
    (s0, *g0, n0), (s5, *g5, n5) = res
    assert all(np.array_equal(a, b) for a, b in zip(s0, s5))
    assert all(np.array_equal(a, b) for a, b in zip(g0, g5))
    assert n5 < kw["nt"] < n0               # one launch per pass: the blocked pass ran


def test_uneven_batch():
    members = [_case(*c, seed=7) for c in (CASES[0], (45, 37, 18, 8, 2, 0, 0.6, 1.5, 20), (262, 19, 5, 8, 0, 1, 0.5, 3.0, 131))]
    with dsh.Batch([dsh.make_params(max_shots=3, **m[0]) for m in members]) as b:
        for k, m in enumerate(members):
            b.set_model(k, *m[1:4])
        got = b.forward([m[4] for m in members])
    for (kw, vs, rho, qs, shots), seis in zip(members, got):
        m = _model(kw, vs, rho, qs)
        for sh, s in zip(shots, seis):
            o = O.Oracle(m, "port")
            assert np.array_equal(o.forward(sh.srcpos, sh.recpos), s)
            o.close()


@pytest.mark.parametrize("dh", [0.6, 0.7, 1.1, 3.0, 6.0, 12.5])
def test_division_by_dh_over_magnitudes(dh):
    """One velocity step from a wavefield whose stresses span 1e-45 .. 1e30 (source amplitudes), free of strips: the
    increments DT (b s) / DH pass the product form, its limits and the denormal results."""
    nx, ny, nt = 96, 24, 40
    rng = np.random.default_rng(int(dh * 10))
    vs = np.full((ny, nx), 200.0, np.float32)
    rho = rng.uniform(0.5, 4000.0, (ny, nx)).astype(np.float32)
    kw = dict(nx=nx, ny=ny, nt=nt, dh=dh, dt=float(np.float32(2e-4 * dh)), fdorder=4, fw=0, free_surf=1, l=0, damping=200.0,
              fpml=30.0)
    for amp in (1e-40, 1e-36, 1e-30, 1e-20, 1e10, 1e28):
        src = np.zeros((8, 1), np.float32)
        src[:, 0] = [nx // 2, ny // 2, 0, -0.02, 70.0, amp, 0, 3]
        rec = np.array([np.arange(1, nx + 1), np.full(nx, ny // 2 + 1)], np.int32)
        o = O.Oracle(_model(kw, vs, rho, None), "port")
        ref = o.forward(src, rec)
        want = [o.field(f) for f in ("vy", "sxy", "syz")]
        o.close()
        with dsh.Engine(dsh.make_params(**kw)) as e:
            e.set_model(vs, rho)
            seis = e.forward([dsh.Shot(src, rec)])[0]
            got = [e.field(f) for f in ("vy", "sxy", "syz")]
        assert np.array_equal(seis, ref)
        assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_batch_of_small_and_large_models():
    """A model whose launches fill the device (2 shots of 655 x 607) is advanced alone, the other with the common
    launches; both equal their own contexts, also when the large one is left out of a later run."""
    members = [_case(655, 607, 10, 4, 2, 1, 0.5, 1.0, 40, seed=5), _case(45, 37, 10, 8, 0, 0, 0.6, 1.0, 20, seed=6)]
    groups = [members[0][4][:2], members[1][4]]
    ref = []
    for (kw, vs, rho, qs, _), shots in zip(members, groups):
        with dsh.Engine(dsh.make_params(max_shots=3, **kw)) as e:
            e.set_model(vs, rho, qs)
            ref.append(e.forward(shots))
    with dsh.Batch([dsh.make_params(max_shots=3, **m[0]) for m in members]) as b:
        for k, m in enumerate(members):
            b.set_model(k, *m[1:4])
        got = b.forward(groups)
        st = b.stats()
        again = b.forward([[], groups[1]])
    assert all(np.array_equal(x, y) for g, r in zip(got, ref) for x, y in zip(g, r))
    assert st["ms_total"] == max(st["model_ms"]) and st["kernel_launches"] > 0
    assert all(np.array_equal(x, y) for x, y in zip(again[1], ref[1]))


def test_blocked_passes_of_two_contexts_at_once():
    """Two small elastic contexts run their passes from two threads: launches whose blocks wait for one another."""
    import threading

    kw, vs, rho, _, shots = _case(203, 97, 10, 4, 0, 1, 0.5, 1.0, 40, seed=3)
    engines = [dsh.Engine(dsh.make_params(max_shots=3, **kw)) for _ in range(2)]
    out = [None, None]
    for e in engines:
        e.set_model(vs, rho)
        e.set_step_variant(5)
        e.set_wait_limits(device_polls=1 << 20)

    def work(k):
        out[k] = [engines[k].forward(shots) for _ in range(20)]

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    engines[0].set_step_variant(0)
    ref = engines[0].forward(shots)
    for k in range(2):
        engines[k].close()
        assert out[k] is not None
        assert all(np.array_equal(a, b) for o in out[k] for a, b in zip(o, ref))
