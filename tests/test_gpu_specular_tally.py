"""The specular tally: every packet that enters adds the normal reflectance of the material
it enters, with one material and with several, in both precisions, for passes smaller than
a warp and of many launches per warp, and where packets end after a few steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _refl(n):
    return ((1.0 - n) / (1.0 + n)) ** 2


@pytest.mark.parametrize("packets", [1, 33, 200_000])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("layout", ["one", "two"])
@pytest.mark.parametrize("mua", [0.5, 60.0])
def test_specular_weight(tam, orc, packets, precision, layout, mua):
    mats = [(0.0, 0.0, 0.0, 1.0), (mua, 10.0, 0.8, 1.5), (mua, 10.0, 0.8, 1.3)]
    p = tam.default_params(nxg=16, nyg=14, nzg=9, xmax=0.5, ymax=0.5, zmax=0.5, mode=1, precision=precision)
    kw = dict(source_radius=0.6)  # a part of the packets misses the grid
    c = tam.default_config(nmat=3, **kw)
    for i, m in enumerate(mats):
        tam.set_material(c, i, *m, 0.56, 1070.0, 3400.0)
    grid = np.ones((16, 14, 9), dtype=np.uint8, order="F")
    if layout == "two":
        grid[7:] = 2
    with tam.Context(p, c) as ctx:
        ctx.upload(tam.TAM_F_MATERIAL, grid)
        ctx.mc_pass(packets, seed=6, stream=4)
        t = ctx.tallies()
    if layout == "one":
        # per packet: the reflectance of those that enter
        want = (1.0 - t["missed"]) * _refl(1.5)
    else:
        d = orc.mc_desc(16, 14, 9, 0.5, 0.5, 0.5, materials=mats, **kw)
        want = orc.mc_transport(d, grid, packets, seed=6, stream=4)[1]["specular"] / packets
    # FP32 rounds the reflectance (a few operations) and, at an entry point within an ulp
    # of the two materials' border, may enter the other one
    tol = 1e-12 if precision == 0 else 1e-6 + (0 if layout == "one" or packets < 1000 else 3.0 / packets)
    assert abs(t["specular"] - want) <= tol * max(want, 1e-3)
