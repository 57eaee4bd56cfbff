"""The generic FFT of the lines without a register plan
(channel3d_b200/csrc/fft.cuh, ch3d_fft.cu) against the oracle's Poisson solve:
x half-lengths and z lengths whose fewest-passes split uses each radix (2, 3,
4, 6, 8, 9, 12, 16) as the only, the first and the last pass, one to four
passes, powers of three, and the line counts that leave a block's last lines
empty.  nx / 2 and nz take the same lengths, in opposite order.

Tolerance: FP64 transforms differ by rounding (log2(n) eps) and the y systems by
eps ny^2 (16 eps ny^2 with the mesh stretching, ny = 6 or 7 here, below 1e-12);
mixed: FP32 transforms, 2e-5 as the lengths with plans."""
import numpy as np
import pytest

from helpers import rel_l2, small_channel

pytestmark = pytest.mark.gpu

LENGTHS = [4, 6, 8, 9, 12, 16, 18, 24, 27, 32, 36, 48, 54, 72, 81, 96, 108, 144, 162, 192, 216, 243, 324, 432, 486, 648]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("m,nz", list(zip(LENGTHS, LENGTHS[::-1])))
def test_generic_lengths(built, m, nz, precision):
    from channel3d_b200 import ChannelSolver, mesh_y
    from oracle import oracle as O
    cfg = small_channel(2 * m, 6 + m % 2, nz, precision=precision)
    src = np.random.default_rng(m).standard_normal(cfg.shape)
    o = O.Oracle(cfg.copy(precision="fp64"))
    with ChannelSolver(cfg, yp=mesh_y(cfg)) as s:
        e = rel_l2(s.poisson(src), o.poisson(src))
    assert e < (1e-12 if precision == "fp64" else 2e-5), (m, nz, e)
