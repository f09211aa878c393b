"""The two ways in which the quad form takes the voxels beside another class -- listed
where few quads are, in their plane where more than one in twenty is -- against each other
bit for bit, against the FP64 step, and on a context whose material grid changes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MATS = [(0.0, 0.0, 0.0, 1.0, 0.56, 1070.0, 3400.0), (1.0, 20.0, 0.8, 1.4, 0.21, 1200.0, 3590.0),
        (0.3, 12.0, 0.9, 1.4, 0.37, 1200.0, 3300.0), (0.1, 8.0, 0.9, 1.4, 0.16, 1000.0, 2674.0)]


def _ctx(tam, shape, robin, on=True, prec=1):
    nx, ny, nz = shape
    p = tam.default_params(nxg=nx, nyg=ny, nzg=nz, xmax=0.01 * nx / 2, ymax=0.012 * ny / 2, zmax=0.008 * nz / 2, mode=1,
                           precision=prec, pulse_type=1, power=2.0, energy_per_pixel=1e9 if on else 1e-12, total_time=1e6)
    c = tam.default_config(nmat=len(MATS), retrace_fraction=0.0)
    for i, m in enumerate(MATS):
        tam.set_material(c, i, *m)
    for f in range(6):
        c.bc_type[f] = 1 if robin >> f & 1 else 0
        c.bc_h[f] = 10.0 * (f + 1)
    return tam.Context(p, c)


def _fill(tam, ctx, shape, grid, hi=350.0):
    rng = np.random.default_rng(5)
    T = np.full(tuple(n + 2 for n in shape), 310.15, order="F")
    # through the damage window; neither boiling nor ablation, whose switch is not a rounding error
    T[1:-1, 1:-1, 1:-1] = rng.uniform(305.0, hi, size=shape)
    ctx.upload(tam.TAM_F_MATERIAL, grid)
    ctx.upload(tam.TAM_F_TEMP, T)
    ctx.upload(tam.TAM_F_JMEAN_GLOBAL, rng.uniform(0.0, 1e3, size=shape))


def _share(g):
    """Share of quads with another class in or beside them."""
    p = np.pad(g, 1, mode="edge")
    n = [slice(1, -1)] * 3
    d = np.zeros(g.shape, dtype=bool)
    for ax in range(3):
        for o in (0, 2):
            s = list(n)
            s[ax] = slice(o, o + g.shape[ax])
            d |= p[tuple(s)] != g
    return d.reshape(g.shape[0] // 4, 4, *g.shape[1:]).any(axis=1).mean()


SHAPE, DENSE = (68, 41, 44), slice(18, 28)


def _grids(shape):
    rng = np.random.default_rng(9)
    few = np.ones(shape, dtype=np.uint8)
    few[:8, :5, :7] = rng.integers(1, 4, size=(8, 5, 7))             # at the corner, where the faces' ghosts are
    few[-9:-3, -4:, -2:] = rng.integers(1, 4, size=(6, 4, 2))
    many = few.copy()
    many[:, :, DENSE] = rng.integers(1, 4, size=many[:, :, DENSE].shape)
    return few, many




@pytest.mark.parametrize("robin", [0, 0b111111])
@pytest.mark.parametrize("zchunk", [0, 3, 8])
def test_listed_and_in_plane_agree_bitwise(tam, robin, zchunk):
    few, many = _grids(SHAPE)
    assert 0 < _share(few) < 0.04 and _share(many) > 0.2
    same = np.ones(SHAPE, dtype=bool)  # voxels with equal surroundings: a step reaches one plane, a run of one class 8
    same[:, :, DENSE.start - 9:DENSE.stop + 9] = False
    out = []
    for g in (few, many):
        with _ctx(tam, SHAPE, robin) as ctx:
            ctx.set_tuning("heat.zchunk", zchunk)
            _fill(tam, ctx, SHAPE, g)
            ctx.heat_steps(1)
            out.append([ctx.download(f) for f in (tam.TAM_F_TEMP, tam.TAM_F_TISSUE)])
    (T, O), (T2, O2) = out
    assert np.array_equal(T[1:-1, 1:-1, 1:-1][same], T2[1:-1, 1:-1, 1:-1][same])
    assert np.array_equal(O[same], O2[same]) and same.sum() == 68 * 41 * 16


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("robin,on", [(0, True), (0b100110, False), (0b111111, True)])
def test_against_fp64(tam, kind, robin, on):
    steps = 20
    out = []
    for prec in (0, 1):
        with _ctx(tam, SHAPE, robin, on, prec) as ctx:
            _fill(tam, ctx, SHAPE, _grids(SHAPE)[kind])
            ctx.heat_steps(steps)
            assert ctx.device_errors() == 0
            out.append([ctx.download(f) for f in (tam.TAM_F_TEMP, tam.TAM_F_TISSUE)])
    (T0, O0), (T, O) = out
    # a step adds at most the 45 K spread, rounded about ten times; the damage rate
    # doubles in less than 1 K
    tol = steps * 10 * 2.0**-24 * 45.0
    assert np.abs(T - T0).max() <= tol
    assert np.abs(O - O0).max() <= (2 * tol + 1e-5) * O0.max()


def test_follows_the_material_grid(tam):
    """Steps replayed from graphs after each new grid: the same as on a context that only had that grid."""
    few, many = _grids(SHAPE)
    with _ctx(tam, SHAPE, 0b100000) as ctx:
        for g in (few, many, few, np.full(SHAPE, 2, dtype=np.uint8), many):
            _fill(tam, ctx, SHAPE, g, 315.0)
            ctx.heat_steps(40)
            with _ctx(tam, SHAPE, 0b100000) as fresh:
                _fill(tam, fresh, SHAPE, g, 315.0)
                fresh.heat_steps(40)
                assert np.array_equal(ctx.download(tam.TAM_F_TEMP), fresh.download(tam.TAM_F_TEMP))


def test_no_slower_on_grids_full_of_boundaries(tam):
    """A grid of random classes takes at most 2.2 times the step of one class (listed: 4.4 times)."""
    shape, us = (192, 192, 192), []
    for g in (np.ones(shape, dtype=np.uint8), np.random.default_rng(1).integers(1, 4, size=shape).astype(np.uint8)):
        with _ctx(tam, shape, 0, False) as ctx:
            ctx.upload(tam.TAM_F_MATERIAL, g)
            best = []
            for _ in range(5):
                ctx.heat_steps(96)
                best.append(ctx.timing()[1])
            us.append(min(best))
    assert us[1] <= 2.2 * us[0]
