"""The projection of every scheme as a march over chunks of rows, and the step
diagnostics that ride on the last one (channel3d_b200/csrc/ch3d_march.cu), on ragged
tiles and chunks: after steps of each scheme the reported divergence, velocity
maxima and bulk mean are those of the downloaded field (the sums in another order:
1e-12; the divergence, a difference of terms whose products may be contracted, 8 eps
of their sum), and fields and diagnostics match the oracle's steps (1e-10)."""
import numpy as np
import pytest

from helpers import rel_l2, small_channel

pytestmark = pytest.mark.gpu


def _cfg(scheme, nx, ny, nz):
    from channel3d_b200 import workloads
    if scheme == "wall":
        return small_channel(nx, ny, nz)
    if scheme == "free_slip_explicit":
        return workloads.taylor_green(16).copy(nxc=nx, nyc=ny, nzc=nz, nycSection=[ny])
    if scheme.startswith("periodic"):
        return workloads.taylor_green_periodic(16).copy(nxc=nx, nyc=ny, nzc=nz, nycSection=[ny], IsImplicit=int(scheme[-1]))
    cfg, _ = workloads.get({"adi": "channel128_re5600_fimp", "4th": "channel128_re5600_4th", "les": "channel48_les"}[scheme])
    if scheme == "les":
        cfg = cfg.copy(LES_type=2, Cs=0.1)
    return cfg.copy(nxc=nx, nyc=ny, nzc=nz, nycSection=[ny // 2, ny - ny // 2])


@pytest.mark.parametrize("shape", [(32, 4, 4), (36, 9, 18), (96, 33, 54)])
@pytest.mark.parametrize("scheme", ["wall", "adi", "4th", "les", "free_slip_explicit", "periodic0", "periodic1", "periodic2"])
def test_projection_and_diagnostics(built, scheme, shape):
    from channel3d_b200 import ChannelSolver, initfield, mesh_y
    from oracle import oracle as O
    nx, ny, nz = shape
    cfg = _cfg(scheme, nx, max(ny, 8) if scheme == "4th" else ny, max(nz, 8) if scheme == "4th" else nz)
    yp = mesh_y(cfg)
    rng = np.random.default_rng(nx)
    if cfg.nycSection[0] == cfg.nyc:
        f = [a + 0.05 * rng.standard_normal(cfg.shape) for a in initfield.taylor_green(cfg, yp=yp)]
    else:
        f = list(initfield.laminar_noise(cfg, yp=yp, seed=nx))
        f[3] = 0.01 * rng.standard_normal(cfg.shape)
    if cfg.BcOption[2] != 0:
        f[1][:, 0, :] = 0.0
    o = O.Oracle(cfg)
    o.set_state(*f)
    with ChannelSolver(cfg, yp=yp) as s:
        s.upload(*f)
        di = s.step(2)
        gs = s.download()
    do = o.step(2)
    go = o.get_state()
    for k in ("ux", "uy", "uz", "p"):
        assert rel_l2(gs[k], go[k]) < 1e-10, (k, rel_l2(gs[k], go[k]))
    for q, k in enumerate(("ux", "uy", "uz")):
        assert abs(di["vmax"][q] - np.abs(gs[k]).max()) <= 1e-14 * np.abs(gs[k]).max()
    dy = np.diff(yp)[None, :, None]
    uxm = (gs["ux"] * dy).sum() / (cfg.nxc * cfg.nzc) / cfg.yly
    assert abs(di["uxm"] - uxm) <= 1e-12 * max(1.0, abs(uxm))
    for k in ("uxm", "cflmp"):
        assert abs(di[k] - do[k]) <= 1e-9 * max(1.0, abs(do[k])), (k, di[k], do[k])
    assert di["divmax2"] < 1e-11


def _divergence(f, cfg, yp, word):
    """(div, sum of its terms' magnitudes) of the staggered field, with metrics of the field's precision."""
    m = lambda v: np.asarray(v, dtype=word).astype(np.float64)  # noqa: E731
    rdx, rdz, rdyp = m(cfg.nxc / cfg.xlx), m(cfg.nzc / cfg.zlz), m(1.0 / np.diff(yp))[None, :, None]
    v = f["uy"]
    vp = np.roll(v, -1, 1)
    if cfg.BcOption[2] != 0:
        vp[:, -1, :] = cfg.uyBcValue[3]

    def d(a, axis, r):
        u = lambda n: np.roll(a, -n, axis)  # noqa: E731
        if cfg.order == 4:
            return r * ((u(-1) - u(2)) / 24 + 1.125 * (u(1) - a)), abs(r) * (abs(u(-1)) + abs(u(2)) + abs(u(1)) + abs(a))
        return (u(1) - a) * r, (abs(u(1)) + abs(a)) * r

    (dx, sx), (dz, sz) = d(f["ux"], 2, rdx), d(f["uz"], 0, rdz)
    return dx + (vp - v) * rdyp + dz, sx + (abs(vp) + abs(v)) * rdyp + sz


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("scheme,shape", [(q, s) for q in ("wall", "adi", "4th", "les", "free_slip_explicit")
                                          for s in ((36, 9, 18), (96, 33, 54))] +
                         [("periodic%d" % q, (36, 9, 18)) for q in (0, 1, 2)] +
                         [("wall", (144, 9, 128)), ("wall", (256, 16, 162)), ("wall", (256, 16, 192)), ("wall", (128, 9, 486))])
def test_reported_divergence(built, scheme, shape, precision):
    """The divergence that the diagnostics report is that of the downloaded field: rows,
    twisted and substituting projections, ragged tiles and whole ones."""
    from channel3d_b200 import ChannelSolver, initfield, mesh_y
    if precision == "mixed" and scheme.startswith("periodic"):
        pytest.skip("periodic y runs in FP64")
    cfg = _cfg(scheme, *shape).copy(precision=precision)
    yp = mesh_y(cfg)
    f = initfield.taylor_green(cfg, yp=yp) if cfg.FlowType == 3 else initfield.laminar_noise(cfg, yp=yp, seed=4)
    with ChannelSolver(cfg, yp=yp) as s:
        s.upload(*f)
        di = s.step(2)
        gs = s.download()
    word = np.float32 if precision == "mixed" else np.float64
    div, terms = _divergence(gs, cfg, yp, word)
    want = np.abs(div).max()
    bound = 8 * np.finfo(np.float64).eps * terms.max()
    if scheme == "4th" and precision == "mixed":  # its divergence is formed in the field's precision
        bound = 8 * np.finfo(np.float32).eps * terms.max()
    assert want > 0 and di["divmax2"] > 0
    assert abs(di["divmax2"] - want) <= bound, (di["divmax2"], want, bound)
    if precision == "mixed" and scheme != "4th":
        assert want > 100 * bound  # far above what the comparison leaves open
