"""Right-hand sides by chunks of rows (channel3d_b200/csrc/ch3d_rhs.cu) and the
line solves that follow them (ch3d_sweep.cu), whole steps against the oracle:

- ny at the edges of the chunks (8, 16, 32 rows) and of the march's ring, ragged
  tiles in x and z, walls and periodic y, the three implicit schemes;
- sweep lengths at the edges of their forms: 64, 128, 256, 384, 768, 2048, 6144 points
  of an x line, 128, 256, 384, 768, 1536, 3072, 6144 rows of a z or y line, and one
  thread per line beyond;
- grids with more columns than the rows take, where the march runs twisted
  (18432 columns, 160 tiles), FP64 and mixed.

Tolerance: 1e-10 relative for whole FP64 steps; with y systems of ny rows, whose
condition grows as ny^2, 16 eps ny^2 where that is larger (also for the
velocities, which the projection corrects with it).  Pressure: rounding of u*,
eps U, enters it as the potential of that difference over the substep's time
step, up to eps U (L / 2 pi) / (alpha dt) at the lowest wavenumber, alpha >= 2/15;
four times that over the pressure's rms where that is larger.  Mixed: 1e-4."""
import numpy as np
import pytest

from helpers import rel_l2, small_channel

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _fimp(nx, ny, nz):
    from channel3d_b200 import workloads
    cfg, _ = workloads.get("channel128_re5600_fimp")
    return cfg.copy(nxc=nx, nyc=ny, nzc=nz, nycSection=[ny // 2, ny - ny // 2])


def _periodic(nx, ny, nz, implicit):
    from channel3d_b200 import workloads
    return workloads.taylor_green_periodic(16).copy(nxc=nx, nyc=ny, nzc=nz, nycSection=[ny], IsImplicit=implicit)


def _check(cfg, nsteps=2, mixed=False):
    from channel3d_b200 import ChannelSolver, initfield, mesh_y
    from oracle import oracle as O
    rng = np.random.default_rng(cfg.nyc)
    yp = mesh_y(cfg)
    if cfg.BcOption[2] == 0:
        f = [a + 0.05 * rng.standard_normal(cfg.shape) for a in initfield.taylor_green(cfg, yp=yp)]
    else:
        f = list(initfield.laminar_noise(cfg, yp=yp, seed=3))
        f[3] = 0.01 * rng.standard_normal(cfg.shape)
    o = O.Oracle(cfg.copy(precision="fp64"))
    o.set_state(*f)
    with ChannelSolver(cfg, yp=yp) as s:
        s.upload(*f)
        s.step(nsteps)
        gs = s.download()
    o.step(nsteps)
    go = o.get_state()
    tol = 1e-4 if mixed else max(1e-10, 16 * EPS * cfg.nyc ** 2)
    for k in ("ux", "uy", "uz"):
        assert rel_l2(gs[k], go[k]) < tol, (k, rel_l2(gs[k], go[k]))
    if not mixed:
        ptol = 4 * EPS * np.abs(go["ux"]).max() * cfg.xlx / (2 * np.pi) / (2 / 15 * cfg.dtMax) / np.sqrt(np.mean(go["p"] ** 2))
        assert rel_l2(gs["p"], go["p"]) < max(tol, ptol), rel_l2(gs["p"], go["p"])


@pytest.mark.parametrize("ny", [4, 5, 8, 9, 17, 33, 65])
@pytest.mark.parametrize("scheme", ["wall", "adi", "explicit", "periodic", "periodic_adi"])
def test_chunk_edges(built, scheme, ny):
    nx, nz = 36, 18
    if scheme == "wall":
        cfg = small_channel(nx, ny, nz)
    elif scheme == "adi":
        cfg = _fimp(nx, ny, nz)
    elif scheme == "explicit":
        cfg = _periodic(nx, ny, nz, 0)
    else:
        cfg = _periodic(nx, ny, nz, 1 if scheme == "periodic" else 2)
    _check(cfg)


@pytest.mark.parametrize("ny", [5, 33, 65])
def test_chunk_edges_mixed(built, ny):
    _check(small_channel(36, ny, 18, precision="mixed"), mixed=True)


@pytest.mark.parametrize("shape", [(64, 6, 128), (72, 6, 144), (128, 6, 256), (144, 5, 288), (256, 6, 384), (288, 6, 432),
                                   (384, 6, 72), (432, 5, 54), (768, 6, 16), (864, 6, 12), (12, 6, 864)])
def test_sweep_lengths_xz(built, shape):
    _check(_fimp(*shape), 1)


@pytest.mark.parametrize("ny", [127, 128, 129, 256, 257, 384, 385, 768, 769])
@pytest.mark.parametrize("periodic", [False, True])
def test_sweep_lengths_y(built, ny, periodic):
    _check(_periodic(18, ny, 6, 2) if periodic else small_channel(18, ny, 6), 1)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_twisted_march_above_the_rows(built, precision):
    _check(small_channel(144, 25, 128, precision=precision), mixed=precision == "mixed")


@pytest.mark.parametrize("shape", [(2048, 4, 4), (2304, 5, 6), (6144, 4, 4), (6912, 4, 4), (8, 5, 1536), (8, 5, 1728),
                                   (6, 4, 3456)])
def test_long_sweeps_xz(built, shape):
    _check(_fimp(*shape), 1)


@pytest.mark.parametrize("ny", [1000, 1536, 1537, 3072, 3073, 6144, 6145])
@pytest.mark.parametrize("scheme", ["wall", "adi", "periodic", "periodic_adi"])
def test_long_sweeps_y(built, scheme, ny):
    if scheme.startswith("periodic"):
        cfg = _periodic(18, ny, 6, 2 if scheme == "periodic_adi" else 1)
    else:
        cfg = small_channel(18, ny, 6) if scheme == "wall" else _fimp(18, ny, 6)
    _check(cfg.copy(dtMax=cfg.dtMax * 769 / ny), 1)  # the convective limit of a shorter cell


def test_long_sweeps_y_mixed(built):
    cfg = small_channel(18, 1537, 6, precision="mixed")
    _check(cfg.copy(dtMax=cfg.dtMax / 2), 1, mixed=True)
