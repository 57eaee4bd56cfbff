"""The column march (right-hand sides fused with the y Crank-Nicolson solves,
channel3d_b200/csrc/ch3d_march.cu) in each of its launch layouts, whole steps
against the oracle within the 1e-10 relative bound:

- twisted blocks (few column tiles, more columns than the rows take: two thread
  groups per tile, the lower eliminating upwards and the upper downwards, meeting
  in the middle), with odd ny so the groups march different numbers of rows, even
  ny, ragged tiles in x and z, and the smallest ny the layout takes;
- grids of fewer columns, whose right-hand sides go by rows;
- one tile per plain block (more tiles than twisted blocks fit on the GPU, fewer
  than the resident persistent blocks), with a ragged last z tile;
- the 4th-order march both ways (128 column tiles twisted, 384 plain);
- the march that stops at g on grids with more tiles than twisted blocks fit
  (2nd order): the divergence and projection marches substitute u* from g
  themselves, and the last projection carries the step diagnostics."""
import numpy as np
import pytest

from helpers import rel_l2, small_channel

pytestmark = pytest.mark.gpu


def _run(cfg, nsteps, seed=11):
    from channel3d_b200 import ChannelSolver, initfield, mesh_y
    from oracle import oracle as O
    yp = mesh_y(cfg)
    ux, uy, uz, p = initfield.laminar_noise(cfg, yp=yp, seed=seed)
    p = 0.01 * np.random.default_rng(seed).standard_normal(cfg.shape)
    o = O.Oracle(cfg)
    o.set_state(ux, uy, uz, p)
    s = ChannelSolver(cfg, yp=yp)
    s.upload(ux, uy, uz, p)
    di = s.step(nsteps)
    o.step(nsteps)
    go, gs = o.get_state(), s.download(hist=True)
    s.close()
    return go, gs, di


def _check(go, gs, tol=1e-10):
    for k in ("ux", "uy", "uz", "p"):
        e = rel_l2(gs[k], go[k])
        assert e < tol, (k, e)


def _flags(cfg):
    from channel3d_b200 import ChannelSolver, mesh_y
    with ChannelSolver(cfg, yp=mesh_y(cfg)) as s:
        return s.path_flags()


@pytest.mark.parametrize("shape", [(144, 25, 162), (128, 5, 162), (96, 24, 192), (108, 4, 192), (144, 7, 128)])
def test_twisted_march(built, shape):
    cfg = small_channel(*shape)
    assert _flags(cfg) == {"march", "twisted"}
    go, gs, di = _run(cfg, 4)
    _check(go, gs)
    assert di["divmax2"] < 1e-12


@pytest.mark.parametrize("shape", [(48, 25, 18), (32, 5, 16), (64, 24, 48)])
def test_few_columns(built, shape):
    cfg = small_channel(*shape)
    assert not _flags(cfg)
    go, gs, di = _run(cfg, 4)
    _check(go, gs)
    assert di["divmax2"] < 1e-12


def test_plain_blocks_one_tile_each(built):
    # 8 x 41 = 328 tiles: above the 296 twisted FP64 blocks that fit, below the 592 persistent ones
    go, gs, _ = _run(small_channel(256, 16, 162), 3)
    _check(go, gs)


@pytest.mark.parametrize("shape,twisted", [((144, 25, 162), True), ((128, 5, 162), True), ((48, 25, 18), False)])
def test_twisted_march_mixed(built, shape, twisted):
    """FP32 twisted march (mixed path), and the rows of fewer columns, within the mixed
    path's 1e-4 bound."""
    cfg = small_channel(*shape, precision="mixed")
    assert ("twisted" in _flags(cfg)) == twisted
    go, gs, _ = _run(cfg, 4)
    for k in ("ux", "uy", "uz"):
        assert rel_l2(gs[k], go[k]) < 1e-4, (k, rel_l2(gs[k], go[k]))


@pytest.mark.parametrize("shape", [(128, 33, 128), (256, 16, 192)])
def test_march_4th(built, shape):
    from channel3d_b200 import workloads
    cfg, _ = workloads.get("channel128_re5600_4th")
    nx, ny, nz = shape
    cfg = cfg.copy(nxc=nx, nyc=ny, nzc=nz, nycSection=[ny // 2, ny - ny // 2])
    go, gs, di = _run(cfg, 3)
    _check(go, gs)
    assert di["divmax2"] < 1e-12


def test_gsub_step_info(built):
    """The diagnostics the last projection computes from g (divergence, velocity
    maxima, CFL, bulk mean) and the divergence before it, against the oracle's
    step, on a grid above the twisted threshold (8 x 41 = 328 tiles)."""
    go, gs, di = _run(small_channel(256, 16, 162), 3)
    _check(go, gs)
    from oracle import oracle as O
    from channel3d_b200 import initfield, mesh_y
    cfg = small_channel(256, 16, 162)
    yp = mesh_y(cfg)
    ux, uy, uz, p = initfield.laminar_noise(cfg, yp=yp, seed=11)
    p = 0.01 * np.random.default_rng(11).standard_normal(cfg.shape)
    o = O.Oracle(cfg)
    o.set_state(ux, uy, uz, p)
    do = o.step(3)
    for k in ("divmax1", "cflmp", "uxm", "PrGradAver"):
        assert abs(di[k] - do[k]) <= 1e-9 * max(1.0, abs(do[k])), (k, di[k], do[k])
    for q in range(3):
        assert abs(di["vmax"][q] - do["vmax"][q]) <= 1e-10 * abs(do["vmax"][q]), (q, di["vmax"], do["vmax"])
    assert di["divmax2"] < 1e-12


@pytest.mark.parametrize("shape", [(256, 16, 192), (128, 9, 486), (256, 33, 162)])
def test_gsub_projection_chunks(built, shape):
    """The substituting projection over whole columns (384 tiles, 0.86 of a wave) and over
    chunks of rows (488 and 328 tiles; ny below, at and above a chunk)."""
    cfg = small_channel(*shape)
    assert _flags(cfg) == {"march", "gsub"}
    go, gs, di = _run(cfg, 3)
    _check(go, gs)
    assert di["divmax2"] < 1e-12


def test_gsub_mixed(built):
    """Mixed path with the march stopping at g (8 x 81 = 648 tiles)."""
    go, gs, di = _run(small_channel(256, 24, 324, precision="mixed"), 3)
    for k in ("ux", "uy", "uz"):
        assert rel_l2(gs[k], go[k]) < 1e-4, (k, rel_l2(gs[k], go[k]))
    assert di["divmax2"] < 1e-4


@pytest.mark.parametrize("scheme,shape,flags", [
    ("rows", (64, 48, 48), set()), ("twisted", (144, 24, 128), {"march", "twisted"}),
    ("gsub", (256, 16, 162), {"march", "gsub"}), ("adi", (48, 32, 36), set()), ("4th", (48, 24, 36), {"march", "twisted"})])
def test_layout_flags(built, scheme, shape, flags):
    """The layout flags say which kernels run: no march where the right-hand sides go by rows."""
    from channel3d_b200 import ChannelSolver, mesh_y, workloads
    cfg = small_channel(*shape)
    if scheme in ("adi", "4th"):
        cfg, _ = workloads.get({"adi": "channel128_re5600_fimp", "4th": "channel128_re5600_4th"}[scheme])
        cfg = cfg.copy(nxc=shape[0], nyc=shape[1], nzc=shape[2], nycSection=[shape[1] // 2, shape[1] - shape[1] // 2])
    with ChannelSolver(cfg, yp=mesh_y(cfg)) as s:
        assert s.path_flags() == flags


@pytest.mark.parametrize("scheme,shape,fused", [
    ("rows", (64, 48, 48), False), ("twisted", (144, 24, 128), True), ("gsub", (256, 16, 162), True),
    ("adi", (48, 32, 36), False), ("4th", (48, 24, 36), True), ("explicit", (32, 24, 32), True),
    ("periodic", (32, 24, 32), False), ("les", (48, 24, 32), False), ("les_explicit", (48, 24, 32), False)])
def test_kernel_groups(built, scheme, shape, fused):
    """Group times keep right-hand sides and solves apart unless one kernel does both (then
    group 1 is 0), and the steps taken are steps."""
    from channel3d_b200 import ChannelSolver, initfield, mesh_y, workloads
    nx, ny, nz = shape
    if scheme in ("explicit", "periodic"):
        cfg = workloads.taylor_green_periodic(16).copy(nxc=nx, nyc=ny, nzc=nz, nycSection=[ny],
                                                       IsImplicit=0 if scheme == "explicit" else 1)
    elif scheme in ("rows", "twisted", "gsub"):
        cfg = small_channel(*shape)
    else:
        cfg, _ = workloads.get({"adi": "channel128_re5600_fimp", "4th": "channel128_re5600_4th"}.get(scheme, "channel48_les"))
        cfg = cfg.copy(nxc=nx, nyc=ny, nzc=nz, nycSection=[ny // 2, ny - ny // 2])
        if scheme.startswith("les"):
            cfg = cfg.copy(LES_type=2, Cs=0.1, IsImplicit=0 if scheme == "les_explicit" else 1)
    yp = mesh_y(cfg)
    f = initfield.taylor_green(cfg, yp=yp) if cfg.FlowType == 3 else initfield.laminar_noise(cfg, yp=yp, seed=3)
    with ChannelSolver(cfg, yp=yp) as s, ChannelSolver(cfg, yp=yp) as ref:
        s.upload(*f)
        ref.upload(*f)
        t = s.kernel_times(2)
        ref.step(2)
        a, b = s.download(), ref.download()
    assert (t[[0, 2, 3, 4, 5, 6]] > 0).all(), t
    assert (t[1] == 0) if fused else (t[1] > 0), t
    for k in ("ux", "uy", "uz", "p"):
        assert np.array_equal(a[k], b[k]), k
