"""Batched heat steps of grids one voxel thick along an axis (both faces of that axis belong
to the same voxels) against each instance's FP64 steps, in every form of the batched step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MATS = [(0.0, 0.0, 0.0, 1.0, 0.56, 1070.0, 3400.0), (1.0, 20.0, 0.8, 1.4, 0.21, 1200.0, 3590.0),
        (0.3, 12.0, 0.9, 1.4, 0.37, 1200.0, 3300.0)]
SHAPES = [(37, 1, 9), (12, 1, 40), (1, 11, 9), (14, 13, 1), (1, 1, 1), (2, 1, 1), (33, 9, 8)]
STEPS = 30


def _ctx(tam, shape, several, robin, prec):
    nx, ny, nz = shape
    p = tam.default_params(nxg=nx, nyg=ny, nzg=nz, xmax=0.01 * nx / 2, ymax=0.012 * ny / 2, zmax=0.008 * nz / 2, mode=1,
                           precision=prec, pulse_type=1, power=2.0, energy_per_pixel=1e9, total_time=1e6)
    c = tam.default_config(nmat=len(MATS), retrace_fraction=0.0)
    for i, m in enumerate(MATS):
        tam.set_material(c, i, *m)
    for f in range(6):
        c.bc_type[f] = robin >> f & 1
        c.bc_h[f] = 100.0 * (f + 1)
        c.bc_T[f] = 305.0 + 2 * f
    rng = np.random.default_rng(nx + 10 * ny)
    ctx = tam.Context(p, c)
    ctx.upload(tam.TAM_F_MATERIAL, rng.integers(1, 3, size=shape).astype(np.uint8) if several else np.full(shape, 2, dtype=np.uint8))
    T = np.full(tuple(n + 2 for n in shape), 310.15, order="F")
    T[1:-1, 1:-1, 1:-1] = rng.uniform(300.0, 345.0, size=shape)
    ctx.upload(tam.TAM_F_TEMP, T)
    ctx.upload(tam.TAM_F_JMEAN_GLOBAL, rng.uniform(0.0, 1e3, size=shape))
    return ctx


@pytest.mark.parametrize("staged", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("several", [False, True])
@pytest.mark.parametrize("robin", [0, 0b111111, 0b001000])
def test_thin_grids(tam, staged, several, robin):
    ctxs = [_ctx(tam, s, several, robin, 1) for s in SHAPES]
    try:
        ctxs[0].set_tuning("batch.staged", staged)
        tam.batch_heat_steps(ctxs, STEPS)
        for s, ctx in zip(SHAPES, ctxs):
            with _ctx(tam, s, several, robin, 0) as ref:
                ref.heat_steps(STEPS)
                T0 = ref.download(tam.TAM_F_TEMP)
            # a step adds at most the 45 K spread, rounded about ten times
            assert np.abs(ctx.download(tam.TAM_F_TEMP) - T0).max() <= STEPS * 10 * 2.0**-24 * 45.0, s
            assert ctx.device_errors() == 0
    finally:
        for c in ctxs:
            c.close()
