"""The Poisson y systems in their launch forms (channel3d_b200/csrc/ch3d_ysolve.cu):
the chunked solve at the edges of its rows per thread (4, 8, 12, 24 rows in up
to 32 chunks) and of its last chunk, and one thread per column beyond it, each
against the oracle's Poisson solve.

Tolerance: both sides eliminate the same systems in another order, so they
differ by rounding times the systems' condition number, which grows as ny^2
(the second difference in y); 16 eps ny^2 bounds it with the mesh stretching.
Mixed: FP32 transforms and sweeps of the higher modes, 1e-4."""
import numpy as np
import pytest

from helpers import rel_l2, small_channel

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _poisson(cfg):
    from channel3d_b200 import ChannelSolver, mesh_y
    from oracle import oracle as O
    src = np.random.default_rng(cfg.nyc).standard_normal(cfg.shape)
    src -= src.mean()
    o = O.Oracle(cfg)
    with ChannelSolver(cfg, yp=mesh_y(cfg)) as s:
        return s.poisson(src), o.poisson(src)


@pytest.mark.parametrize("ny", [4, 5, 31, 127, 128, 129, 255, 257, 384, 385, 768, 769])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_wall_systems(built, ny, precision):
    a, b = _poisson(small_channel(18, ny, 6, precision=precision))
    assert rel_l2(a, b) < (16 * EPS * ny * ny if precision == "fp64" else 1e-4), rel_l2(a, b)


@pytest.mark.parametrize("ny", [4, 5, 33, 128, 130, 257, 400, 770])
def test_cyclic_systems(built, ny):
    from channel3d_b200 import workloads
    cfg = workloads.taylor_green_periodic(16).copy(nxc=18, nyc=ny, nzc=6, nycSection=[ny])
    a, b = _poisson(cfg)
    assert rel_l2(a, b) < 16 * EPS * max(ny, 32) ** 2, rel_l2(a, b)
