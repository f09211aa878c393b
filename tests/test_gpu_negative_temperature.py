"""A step that takes a voxel from an ordinary temperature to a negative one reports it, in
every form of the heat step.  The time step lies far beyond the stability limit, so one
voxel 4 K above a uniform field swings below 0 K while all the others warm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MATS = [(0.0, 0.0, 0.0, 1.0, 0.56, 1070.0, 3400.0), (1.0, 20.0, 0.8, 1.4, 0.21, 1200.0, 3590.0),
        (0.3, 12.0, 0.9, 1.4, 0.37, 1200.0, 3300.0)]


def _ctx(tam, shape, at, mixed, prec):
    nx, ny, nz = shape
    p = tam.default_params(nxg=nx, nyg=ny, nzg=nz, xmax=0.01 * nx / 2, ymax=0.012 * ny / 2, zmax=0.008 * nz / 2, mode=1,
                           precision=prec, pulse_type=1, power=2.0, energy_per_pixel=1e9, total_time=1e6)
    c = tam.default_config(nmat=len(MATS), retrace_fraction=0.0, dt=5.0)
    for i, m in enumerate(MATS):
        tam.set_material(c, i, *m)
    ctx = tam.Context(p, c)
    g = np.full(shape, 2, dtype=np.uint8)
    if mixed:  # one class in the first tiles' runs, another from x = 60 on
        g[60:] = 1
    ctx.upload(tam.TAM_F_MATERIAL, g)
    T = np.full(tuple(n + 2 for n in shape), 310.15, order="F")
    if at is not None:
        T[tuple(i + 1 for i in at)] = 314.15
    ctx.upload(tam.TAM_F_TEMP, T)
    return ctx


def _check(tam, ctxs, step, places):
    if not any(places):
        step()
    else:
        with pytest.raises(tam.TamError, match="negative temperature"):
            step()
    for ctx, at in zip(ctxs, places):
        T = ctx.download(tam.TAM_F_TEMP)[1:-1, 1:-1, 1:-1]
        assert (T < 0).sum() == (0 if at is None else 1) and (at is None or T[at] < 0)
        assert ctx.device_errors() == (0 if at is None else tam._abi.TAM_DEVERR_NEG_T)


# x = 59 and 60: beside another class; 45: in a mixed run, all of one class around
PLACES = [None, (5, 4, 6), (0, 0, 0), (45, 3, 12), (59, 4, 6), (60, 0, 3), (67, 8, 12)]


# quad form (68 wide), line form (69), FP64 class form, and the per-voxel forms ("heat.cls" 0)
@pytest.mark.parametrize("at", PLACES)
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("nx,prec", [(68, 1), (69, 1), (68, 0)])
@pytest.mark.parametrize("cls", [1, 0])
def test_single(tam, at, mixed, nx, prec, cls):
    with _ctx(tam, (nx, 9, 13), at, mixed, prec) as ctx:
        ctx.set_tuning("heat.cls", cls)
        _check(tam, [ctx], lambda: ctx.heat_steps(1), [at])


@pytest.mark.parametrize("at", PLACES)
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("staged", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("hot", [0, 1])
def test_batch(tam, at, mixed, staged, hot):
    places = [at if k == hot else None for k in range(2)]
    ctxs = [_ctx(tam, (nx, 9, 13), a, mixed, 1) for nx, a in zip((68, 69), places)]
    try:
        ctxs[0].set_tuning("batch.staged", staged)
        _check(tam, ctxs, lambda: tam.batch_heat_steps(ctxs, 1), places)
    finally:
        for c in ctxs:
            c.close()
