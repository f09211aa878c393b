"""The quad form of the FP32 heat step against the voxel-pair form ("heat.slab" 0)
and the FP64 step: the smallest grids, rows and planes that end inside a warp, a
block or a run of planes, one and several classes, convective and fixed faces, with
and without a source."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MATS = [(0.0, 0.0, 0.0, 1.0, 0.56, 1070.0, 3400.0), (1.0, 20.0, 0.8, 1.4, 0.21, 1200.0, 3590.0),
        (0.3, 12.0, 0.9, 1.4, 0.37, 1200.0, 3300.0), (0.1, 8.0, 0.9, 1.4, 0.16, 1000.0, 2674.0)]
STEPS = 20


def _run(tam, shape, grid, robin, on, prec, slab, zchunk=0):
    nx, ny, nz = shape
    p = tam.default_params(nxg=nx, nyg=ny, nzg=nz, xmax=0.01 * nx / 2, ymax=0.012 * ny / 2, zmax=0.008 * nz / 2, mode=1,
                           precision=prec, pulse_type=1, power=2.0, energy_per_pixel=1e9 if on else 1e-12, total_time=1e6)
    c = tam.default_config(nmat=len(MATS), retrace_fraction=0.0)
    for i, m in enumerate(MATS):
        tam.set_material(c, i, *m)
    for f in range(6):
        c.bc_type[f] = 1 if robin >> f & 1 else 0
        c.bc_h[f] = 10.0 * (f + 1)
    rng = np.random.default_rng(5)
    with tam.Context(p, c) as ctx:
        g = np.ones(shape, dtype=np.uint8)
        if grid == "random":
            g = rng.integers(1, 4, size=shape).astype(np.uint8)
        elif grid == "ball":  # runs of one class, mixed runs and quads beside another class
            r = sum(((np.arange(n) - 0.4 * n) ** 2).reshape([-1 if i == k else 1 for i in range(3)]) for k, n in enumerate(shape))
            g[r < (0.2 * max(shape)) ** 2] = 3
        ctx.upload(tam.TAM_F_MATERIAL, g)
        T = np.full(tuple(n + 2 for n in shape), 310.15, order="F")
        # through the damage window; neither boiling nor ablation, whose switch is not a rounding error
        T[1:-1, 1:-1, 1:-1] = rng.uniform(305.0, 350.0, size=shape)
        ctx.upload(tam.TAM_F_TEMP, T)
        ctx.upload(tam.TAM_F_JMEAN_GLOBAL, rng.uniform(0.0, 1e3, size=shape))
        ctx.set_tuning("heat.slab", slab)
        ctx.set_tuning("heat.zchunk", zchunk)
        ctx.heat_steps(STEPS)
        return ctx.download(tam.TAM_F_TEMP), ctx.download(tam.TAM_F_TISSUE), ctx.device_errors()


def _check(T, O, T0, O0):
    # a step adds at most the 45 K spread, rounded about ten times; the damage rate
    # doubles in less than 1 K, so its relative error is that of the temperature in K
    tol = STEPS * 10 * 2.0**-24 * 45.0
    assert np.abs(T - T0).max() <= tol
    assert np.abs(O - O0).max() <= (2 * tol + 1e-5) * max(np.abs(O0).max(), 1e-300)


@pytest.mark.parametrize("shape", [(4, 1, 1), (4, 3, 2), (8, 2, 1), (36, 9, 6), (128, 1, 5), (132, 5, 7), (64, 8, 41), (508, 3, 9)])
@pytest.mark.parametrize("grid", ["one", "ball", "random"])
@pytest.mark.parametrize("robin,on", [(0, True), (0b111111, False), (0b100110, True)])
def test_quad_step(tam, shape, grid, robin, on):
    T0, O0, _ = _run(tam, shape, grid, robin, on, 0, 0)
    T, O, err = _run(tam, shape, grid, robin, on, 1, 1)
    Tp, Op, _ = _run(tam, shape, grid, robin, on, 1, 0)
    assert err == 0
    _check(T, O, T0, O0)
    _check(T, O, Tp, Op)


@pytest.mark.parametrize("zchunk", [1, 2, 3, 5, 8, 13])
def test_quad_step_planes_per_block(tam, zchunk):
    shape = (68, 9, 13)
    T0, O0, _ = _run(tam, shape, "ball", 0b111111, True, 0, 0)
    _check(*_run(tam, shape, "ball", 0b111111, True, 1, 1, zchunk)[:2], T0, O0)


def test_quad_step_one_class_is_independent_of_the_planes_per_block(tam):
    shape = (132, 9, 23)
    a = _run(tam, shape, "one", 0b111111, True, 1, 1, 1)
    for zchunk in (0, 3, 8):
        b = _run(tam, shape, "one", 0b111111, True, 1, 1, zchunk)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
