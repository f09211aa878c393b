"""The autotuner against the settings in force before it: its choice is never slower, and
the choice that it returns gives the same speed on another context."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ctx(tam, shape, prec):
    nx, ny, nz = shape
    p = tam.default_params(nxg=nx, nyg=ny, nzg=nz, xmax=0.005 * nx, ymax=0.005 * ny, zmax=0.005 * nz, mode=1, precision=prec,
                           pulse_type=1, power=2.0, energy_per_pixel=1e-12, total_time=1e9)
    return tam.Context(p, tam.default_config(retrace_fraction=0.0))


def _us(ctx, steps=320):
    best = []
    for _ in range(5):
        ctx.heat_steps(steps)
        best.append(ctx.timing()[1] * 1e3 / steps)
    return min(best)


# one plane per column is the fastest on the first two (quad and line form: two planes
# take 1.17 and 1.5 times as long); FP64 form; the last has no choice of length at all
@pytest.mark.parametrize("shape,prec", [((64, 64, 64), 1), ((63, 64, 64), 1), ((60, 50, 55), 0), ((64, 64, 1), 1)])
def test_no_slower_than_before(tam, shape, prec):
    with _ctx(tam, shape, prec) as ctx, _ctx(tam, shape, prec) as other:
        before = _us(ctx)
        chosen = ctx.autotune(packets=0, steps=480)
        assert _us(ctx) <= 1.15 * before
        for k, v in chosen.items():
            other.set_tuning(k, v)
        assert _us(other) <= 1.15 * before


def test_settings_in_force_count(tam):
    """A setting that is set before the call is timed with the others, and the fields stay as they were."""
    with _ctx(tam, (64, 64, 64), 1) as ctx:
        T = np.full((66, 66, 66), 310.15, order="F")
        T[1:-1, 1:-1, 1:-1] = np.random.default_rng(3).uniform(305.0, 315.0, (64, 64, 64))
        ctx.upload(tam.TAM_F_TEMP, T)
        T = ctx.download(tam.TAM_F_TEMP)
        ctx.set_tuning("heat.zchunk", 1)
        before = _us(ctx)
        ctx.upload(tam.TAM_F_TEMP, T)
        chosen = ctx.autotune(packets=0, steps=480)
        assert np.array_equal(ctx.download(tam.TAM_F_TEMP), T)
        assert (chosen["heat.zchunk"], chosen["heat.zauto"]) == (1, 0)
        assert _us(ctx) <= 1.15 * before


@pytest.mark.parametrize("value", [-1, 2])
def test_zauto_is_a_switch(tam, value):
    with _ctx(tam, (8, 8, 8), 1) as ctx:
        with pytest.raises(tam.TamError):
            ctx.set_tuning("heat.zauto", value)
