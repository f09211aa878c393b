"""FP64 disk sources whose squared radius is subnormal, zero or the smallest normal: pencil
beams, every packet of which enters at the centre."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pass(tam, radius):
    p = tam.default_params(nxg=9, nyg=8, nzg=7, xmax=0.5, ymax=0.5, zmax=0.5, mode=1, precision=0)
    c = tam.default_config(nmat=2, source=tam._abi.TAM_SRC_DISK, source_radius=radius)
    tam.set_material(c, 0, 0.0, 0.0, 0.0, 1.0, 0.56, 1070.0, 3400.0)
    tam.set_material(c, 1, 0.5, 20.0, 0.8, 1.38, 0.56, 1070.0, 3400.0)
    with tam.Context(p, c) as ctx:
        ctx.mc_pass(4000, seed=3, stream=1)
        return ctx.download(tam.TAM_F_JMEAN), ctx.tallies()


# the square of 1e-170 is zero, those of 1e-162, 1e-158 and 1e-155 subnormal, that of 1.6e-154 normal,
# a random share of it subnormal
@pytest.mark.parametrize("radius", [1e-162, 1e-158, 1e-155, 1.6e-154, 1e-150])
def test_pencil_beam(tam, radius):
    J0, t0 = _pass(tam, 1e-170)
    J, t = _pass(tam, radius)
    assert t["missed"] == t0["missed"] == 0
    # the walks are the same to the last bit; the sums are taken in another order
    assert t["scatters"] == t0["scatters"] and t["voxel_steps"] == t0["voxel_steps"]
    assert np.abs(J - J0).sum() <= 4000 * 2.0**-53 * J0.sum()
