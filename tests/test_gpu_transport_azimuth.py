"""FP64 passes against the oracle on the same random streams, for each branch of the
azimuth's update: isotropic, forward and backward scattering, reflecting faces of a
cube (mirrors and wraps), and a source whose azimuth is drawn by every packet."""
import numpy as np
import pytest

from test_gpu_parity import cfg_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("g", [0.0, 0.8, -0.5])
@pytest.mark.parametrize("n_medium", [1.0, 1.6])
def test_azimuth_follows_the_oracle(tam, orc, g, n_medium):
    mats = [(0.0, 0.0, 0.0, 1.0), (0.5, 40.0, g, n_medium)]
    ctx, d = cfg_pair(tam, orc, 9, 8, 7, 0.2, mats=mats, radius=0.05)
    grid = np.ones((9, 8, 7), dtype=np.uint8, order="F")
    n = 2000
    ctx.mc_pass(n, seed=17, stream=2)
    J = ctx.download(tam.TAM_F_JMEAN)
    Jo, to = orc.mc_transport(d, grid, n, seed=17, stream=2, nthreads=0)
    t = ctx.tallies()
    assert t["scatters"] == to["scatters"] and t["voxel_steps"] == to["voxel_steps"]
    # (a deflection near 0 or PI multiplies its cosine's last bit by up to 1e8)
    assert np.abs(J - Jo).sum() / np.abs(Jo).sum() < 1e-9
    ctx.close()
