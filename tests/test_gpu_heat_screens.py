"""Damage windows that begin at or below 0 K: the screen in front of the rare work then
lies below 0 and lists every voxel, so damage, ablation and the latent-heat clamp of the
quad, line and FP64 class forms equal those of the per-voxel step ("heat.cls" 0)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MATS = [(0.0, 0.0, 0.0, 1.0, 0.56, 1070.0, 3400.0), (1.0, 20.0, 0.8, 1.4, 0.21, 1200.0, 3590.0),
        (0.3, 12.0, 0.9, 1.4, 0.37, 1200.0, 3300.0), (0.1, 8.0, 0.9, 1.4, 0.16, 1000.0, 2674.0)]
DT, T_HI, T_ABL = 1e-4, 390.0, 400.0


def _step(tam, shape, grid, prec, T_lo, cls):
    nx, ny, nz = shape
    p = tam.default_params(nxg=nx, nyg=ny, nzg=nz, xmax=0.01 * nx / 2, ymax=0.012 * ny / 2, zmax=0.008 * nz / 2, mode=1,
                           precision=prec, pulse_type=1, power=2.0, energy_per_pixel=1e9, total_time=1e6)
    c = tam.default_config(nmat=len(MATS), retrace_fraction=0.0, dt=DT, T_lo=T_lo, T_hi=T_HI, T_abl=T_ABL)
    for i, m in enumerate(MATS):
        tam.set_material(c, i, *m)
    rng = np.random.default_rng(11)
    g = rng.integers(1, 4, size=shape).astype(np.uint8) if grid == "random" else np.full(shape, 2, dtype=np.uint8)
    T = np.full(tuple(n + 2 for n in shape), 310.15, order="F")
    # A step conducts at most 1.1 K and heats by about 2 K: below, in and above the window,
    # at boiling (all of it heated, so every one takes up latent heat) and, its latent heat
    # spent, at ablation, each more than 1 K from the next threshold
    T[1:-1, 1:-1, 1:-1] = rng.choice([312.0, 345.0, 380.0, 420.0], size=shape)
    with tam.Context(p, c) as ctx:
        ctx.upload(tam.TAM_F_MATERIAL, g)
        ctx.upload(tam.TAM_F_TEMP, T)
        ctx.upload(tam.TAM_F_JMEAN_GLOBAL, np.full(shape, 3.6e10))
        spent = T[1:-1, 1:-1, 1:-1] == 420.0
        ctx.upload(tam.TAM_F_Q, np.where(spent, 1.0, 0.0))
        ctx.set_tuning("heat.cls", cls)
        ctx.heat_steps(1)
        assert ctx.device_errors() == 0
        out = [ctx.download(f) for f in (tam.TAM_F_TEMP, tam.TAM_F_TISSUE, tam.TAM_F_MATERIAL, tam.TAM_F_Q)]
        assert (out[3][spent] == 1.0).all()
        out[3][spent] = 0.0
        return out


# whole quads (FP32: quad form), other rows (line form), both at the ends of blocks,
# row pairs and runs of planes
@pytest.mark.parametrize("shape", [(4, 1, 1), (36, 9, 6), (33, 8, 7), (43, 3, 33), (128, 2, 5), (129, 3, 17)])
@pytest.mark.parametrize("grid", ["one", "random"])
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("T_lo", [0.0, 0.005, -5.0])
def test_window_from_zero(tam, shape, grid, prec, T_lo):
    T0, O0, m0, Q0 = _step(tam, shape, grid, prec, T_lo, 0)
    T, O, m, Q = _step(tam, shape, grid, prec, T_lo, 1)
    # a voxel's step sums differences of at most 108 K, rounded about ten times
    eps = 2.0 ** (-24 if prec else -53)
    assert np.abs(T - T0).max() <= 10 * eps * 420.0
    assert np.array_equal(m, m0) and np.array_equal(O > 0, O0 > 0)
    assert (O0 > 0).sum() == (T0[1:-1, 1:-1, 1:-1] < T_HI).sum()
    if O0.size > 4:
        assert (m0 == 0).any() and (m0 != 0).any() and (Q0 > 0).any()
    # the damage rate's logarithm changes by less than 1 per K; its exponent near 200 in
    # FP64 (or in two floats) adds 200 ulp
    assert np.abs(O - O0).max() <= 1e-300 or (np.abs(O - O0) <= (10 * 420.0 + 1000) * eps * O0).all()
    # the energy taken up: the source plus a conducted part of at most half of it
    assert np.abs(Q - Q0).max() <= 1000 * eps * max(Q0.max(), 1e-300)
