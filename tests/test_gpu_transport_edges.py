"""Edges of the transport's launch and flight: passes smaller than the GPU's
lanes (the packets of a warp follow from the pass size) and packets that end
at their step cap (tested per voxel step only near the cap), against the
oracle on the same Philox streams."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pair(tam, orc, edge=24, precision=0, mua=2.0, mus=40.0, **kw):
    p = tam.default_params(nxg=edge, nyg=edge, nzg=edge, xmax=0.5, ymax=0.5, zmax=0.5, mode=1, precision=precision)
    c = tam.default_config(nmat=2, **kw)
    tam.set_material(c, 0, 0.0, 0.0, 0.0, 1.0, 0.56, 1070.0, 3400.0)
    tam.set_material(c, 1, mua, mus, 0.8, 1.38, 0.56, 1070.0, 3400.0)
    d = orc.mc_desc(edge, edge, edge, 0.5, 0.5, 0.5, materials=[(0.0, 0.0, 0.0, 1.0), (mua, mus, 0.8, 1.38)], **kw)
    return tam.Context(p, c), d, np.ones((edge, edge, edge), dtype=np.uint8, order="F")


# one packet, part of a warp, and around the sizes at which a warp of the
# spread pass (8 warps on each of 152 SMs) takes one packet more, or all 32
@pytest.mark.parametrize("n", [1, 31, 1215, 1217, 2433, 4863, 37697, 40000])
def test_pass_sizes(tam, orc, n):
    ctx, d, grid = _pair(tam, orc)
    with ctx:
        ctx.mc_pass(n, seed=9, stream=2)
        J, t = ctx.download(tam.TAM_F_JMEAN), ctx.tallies()
    Jo, to = orc.mc_transport(d, grid, n, seed=9, stream=2)
    assert t["scatters"] == to["scatters"] and t["voxel_steps"] == to["voxel_steps"]
    assert np.abs(J - Jo).sum() <= 1e-9 * np.abs(Jo).sum()
    # FP32, alone and in the batched launch: every packet launched once (each
    # adds the same specular weight), and the same walks both ways
    c32, _, _ = _pair(tam, orc, precision=1)
    with c32:
        c32.mc_pass(n, seed=9, stream=2)
        J32, t32 = c32.download(tam.TAM_F_JMEAN), c32.tallies()
        tam.batch_mc_pass([c32], [9], nphotons=[n], streams=[2])
        Jb, tb = c32.download(tam.TAM_F_JMEAN), c32.tallies()
    assert t32["specular"] == pytest.approx((0.38 / 2.38) ** 2, rel=1e-6)
    for k in ("voxel_steps", "scatters"):
        assert t32[k] == tb[k]
    assert np.abs(J32 - Jb).sum() <= 1e-12 * np.abs(J32).sum()


# caps below, around and above the number of faces a flight can cross (3 x 24)
@pytest.mark.parametrize("cap", [1, 2, 40, 73, 74, 75, 120])
def test_step_caps(tam, orc, cap):
    n = 3000
    ctx, d, grid = _pair(tam, orc, mua=0.3, max_steps=cap)
    with ctx:
        with pytest.raises(tam.TamError):
            ctx.mc_pass(n, seed=4, stream=1)
        J, t = ctx.download(tam.TAM_F_JMEAN), ctx.tallies()
    Jo, to = orc.mc_transport(d, grid, n, seed=4, stream=1)
    assert t["overflow"] > 0 and t["voxel_steps"] == to["voxel_steps"] and t["scatters"] == to["scatters"]
    assert np.abs(J - Jo).sum() <= 1e-9 * np.abs(Jo).sum()
    c32, _, _ = _pair(tam, orc, mua=0.3, precision=1, max_steps=cap)
    with c32:
        with pytest.raises(tam.TamError):
            c32.mc_pass(n, seed=4, stream=1)
        t32, J32 = c32.tallies(), c32.download(tam.TAM_F_JMEAN)
        try:
            tam.batch_mc_pass([c32], [4], nphotons=[n], streams=[1])
        except tam.TamError:
            pass
        tb, Jb = c32.tallies(), c32.download(tam.TAM_F_JMEAN)
    assert t32["overflow"] == tb["overflow"] and t32["voxel_steps"] == tb["voxel_steps"]
    assert np.abs(J32 - Jb).sum() <= 1e-12 * np.abs(J32).sum()
