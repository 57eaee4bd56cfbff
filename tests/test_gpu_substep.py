"""The scalar work between the field kernels (channel3d_b200/csrc/ch3d_substep.cu) when
the time step changes from step to step (iCFL = 1), so that every substep's
coefficient tables are formed anew, against the oracle's steps: one block's partial
sums (up to 4096) and many blocks', the schemes with row tables and with periodic
factor blocks, a stage sequence after fused steps, and stages before any set-up.

Tolerance: whole steps 1e-10 as elsewhere; dt and the CFL number follow the
velocities, 1e-9; pressure 4 eps U (L / 2 pi) / (2/15 dt) over its rms where larger."""
import numpy as np
import pytest

from helpers import rel_l2, small_channel

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _cfg(scheme, shape):
    from channel3d_b200 import workloads
    nx, ny, nz = shape
    if scheme in ("explicit", "periodic", "periodic_adi"):
        cfg = workloads.taylor_green_periodic(16).copy(nxc=nx, nyc=ny, nzc=nz, nycSection=[ny])
        cfg = cfg.copy(IsImplicit=("explicit", "periodic", "periodic_adi").index(scheme))
    elif scheme == "wall":
        cfg = small_channel(nx, ny, nz)
    else:
        cfg, _ = workloads.get({"adi": "channel128_re5600_fimp", "4th": "channel128_re5600_4th"}[scheme])
        cfg = cfg.copy(nxc=nx, nyc=ny, nzc=nz, nycSection=[ny // 2, ny - ny // 2])
    return cfg.copy(iCFL=1, CFLc=0.3, dtMax=1.0)


def _partial_sums(cfg):
    """Partial sums of the projection (its tiles times its chunks of rows)."""
    import torch
    cols = -(-cfg.nxc // 32) * -(-cfg.nzc // 4)
    rows = 32
    while rows > 4 and cols * -(-cfg.nyc // rows) < 4 * torch.cuda.get_device_properties(0).multi_processor_count:
        rows //= 2
    return cols * -(-cfg.nyc // rows)


@pytest.mark.parametrize("scheme,shape", [("wall", (36, 17, 18)), ("adi", (36, 17, 18)), ("4th", (36, 17, 18)),
                                          ("explicit", (36, 17, 18)), ("periodic", (36, 17, 18)),
                                          ("periodic_adi", (36, 17, 18)), ("wall", (256, 16, 162)), ("adi", (768, 33, 192)),
                                          ("wall", (768, 9, 768)), ("adi", (768, 9, 768)), ("4th", (768, 9, 768))])
def test_variable_time_step(built, scheme, shape):
    from channel3d_b200 import ChannelSolver, initfield, mesh_y
    from oracle import oracle as O
    cfg = _cfg(scheme, shape)
    assert (_partial_sums(cfg) > 4096) == (shape == (768, 9, 768))
    yp = mesh_y(cfg)
    rng = np.random.default_rng(5)
    if cfg.BcOption[2] == 0:
        f = [a + 0.05 * rng.standard_normal(cfg.shape) for a in initfield.taylor_green(cfg, yp=yp)]
    else:
        f = list(initfield.laminar_noise(cfg, yp=yp, seed=5))
        f[3] = 0.01 * rng.standard_normal(cfg.shape)
    o = O.Oracle(cfg)
    o.set_state(*f)
    with ChannelSolver(cfg, yp=yp) as s:
        s.upload(*f)
        for _ in range(3):
            di, do = s.step(1), o.step(1)
            for k in ("cflmp", "uxm"):
                assert abs(di[k] - do[k]) <= 1e-9 * max(1.0, abs(do[k])), (k, di[k], do[k])
        gs, go = s.download(), o.get_state()
        for k in ("ux", "uy", "uz"):
            assert rel_l2(gs[k], go[k]) < 1e-10, (k, rel_l2(gs[k], go[k]))
        dt = di["dt"] if "dt" in di else 1e-3
        ptol = 4 * EPS * np.abs(go["ux"]).max() * cfg.xlx / (2 * np.pi) / (2 / 15 * dt) / np.sqrt(np.mean(go["p"] ** 2))
        assert rel_l2(gs["p"], go["p"]) < max(1e-10, ptol), rel_l2(gs["p"], go["p"])


def test_stages_after_steps(built):
    from channel3d_b200 import ChannelSolver, initfield, mesh_y
    from oracle import oracle as O
    cfg = small_channel(36, 17, 18)
    yp = mesh_y(cfg)
    f = initfield.laminar_noise(cfg, yp=yp, seed=6)
    o = O.Oracle(cfg)
    o.set_state(*f)
    with ChannelSolver(cfg, yp=yp) as s:
        s.upload(*f)
        s.step(2)
        o.step(2)
        for ns in (1, 2, 3):
            for q in range(7):
                s.stage(q, ns)
                o.stage(q, ns)
        s.step(1)
        o.step(1)
        gs, go = s.download(), o.get_state()
    for k in ("ux", "uy", "uz"):
        assert rel_l2(gs[k], go[k]) < 1e-10, (k, rel_l2(gs[k], go[k]))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("scheme", ["wall", "adi", "4th", "explicit", "periodic", "periodic_adi", "les"])
def test_stages_before_any_set_up(built, scheme, precision):
    """Right-hand sides and solves called first, or after an array was set (both leave the
    substep's coefficients zero): the right-hand sides are zero, Hist is the convective term
    of the state, and the solves return u* = u + Rhs, exactly."""
    from channel3d_b200 import ChannelSolver, initfield, mesh_y, workloads
    if precision == "mixed" and scheme in ("explicit", "periodic", "periodic_adi"):
        pytest.skip("periodic y runs in FP64")
    shape = (36, 17, 18)
    if scheme == "les":
        cfg, _ = workloads.get("channel48_les")
        cfg = cfg.copy(nxc=36, nyc=17, nzc=18, nycSection=[8, 9], LES_type=2, Cs=0.1)
    else:
        cfg = _cfg(scheme, shape)
    cfg = cfg.copy(precision=precision)
    yp = mesh_y(cfg)
    rng = np.random.default_rng(8)
    f = [rng.standard_normal(cfg.shape).astype(np.float32).astype(np.float64) for _ in range(4)]
    if cfg.BcOption[2] != 0:
        f[1][:, 0, :] = 0.0
    with ChannelSolver(cfg, yp=yp) as s, ChannelSolver(cfg, yp=yp) as ref:
        s.upload(*f)
        ref.upload(*f)
        ref.stage(0, 1)
        ref.stage(1, 1)
        s.stage(1, 1)
        for h in (s.HISTX, s.HISTY, s.HISTZ):
            assert np.array_equal(s.get_array(h), ref.get_array(h)), h
        for r in (s.RHSX, s.RHSY, s.RHSZ):
            assert not s.get_array(r).any(), r
        s.stage(0, 2)
        rhs = [rng.standard_normal(cfg.shape).astype(np.float32).astype(np.float64) for _ in range(3)]
        for q, r in zip((s.RHSX, s.RHSY, s.RHSZ), rhs):
            s.set_array(q, r)
        s.stage(2, 2)
        if cfg.BcOption[2] != 0 and cfg.IsImplicit != 0:
            rhs[1][:, 0, :] = 0.0  # the wall row of uy is held
        word = np.float32 if precision == "mixed" else np.float64
        for q in range(3):
            want = f[q].astype(word) + rhs[q].astype(word)
            assert np.array_equal(s.get_array(12 + q), want.astype(np.float64)), q
