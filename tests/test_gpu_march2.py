"""The FP32 march that stops at g (channel3d_b200/csrc/ch3d_march.cu, mixed path)
at its edges, whole steps against the
FP64 oracle within the mixed path's 1e-4: fewer rows than the march keeps in
flight, ragged tiles in z, several and single rounds of the persistent blocks,
and every x length with a register plan that the layout takes."""
import numpy as np
import pytest

from helpers import rel_l2, small_channel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(768, 4, 162), (768, 5, 216), (512, 9, 243), (256, 33, 486), (128, 8, 972)])
def test_two_column_march(built, shape):
    from channel3d_b200 import ChannelSolver, initfield, mesh_y
    from oracle import oracle as O
    cfg = small_channel(*shape, precision="mixed")
    yp = mesh_y(cfg)
    ux, uy, uz, p = initfield.laminar_noise(cfg, yp=yp, seed=17)
    p = 0.01 * np.random.default_rng(17).standard_normal(cfg.shape)
    o = O.Oracle(cfg.copy(precision="fp64"))
    o.set_state(ux, uy, uz, p)
    with ChannelSolver(cfg, yp=yp) as s:
        assert "gsub" in s.path_flags()
        s.upload(ux, uy, uz, p)
        s.step(2)
        gs = s.download()
    o.step(2)
    go = o.get_state()
    for k in ("ux", "uy", "uz"):
        assert rel_l2(gs[k], go[k]) < 1e-4, (k, rel_l2(gs[k], go[k]))
