"""Results written into a caller's new pages while the GPU works (heat_steps and mc_pass
with `want`) equal the ones fetched afterwards, below and above the size at which the
pages are made present ahead of the copy (4 MiB: 80^3 values)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [24, 79, 81, 120])
def test_wanted_results_equal_downloads(tam, n):
    p = tam.default_params(nxg=n, nyg=n, nzg=n, xmax=0.5, ymax=0.5, zmax=0.5, mode=1, precision=1, nphotons=2000, pulse_type=1,
                           power=2.0, energy_per_pixel=1e9, total_time=1e6)
    c = tam.default_config(nmat=2, retrace_fraction=0.0)
    tam.set_material(c, 0, 0.0, 0.0, 0.0, 1.0, 0.56, 1070.0, 3400.0)
    tam.set_material(c, 1, 1.0, 20.0, 0.8, 1.4, 0.21, 1200.0, 3590.0)
    with tam.Context(p, c) as ctx:
        J = ctx.mc_pass(2000, seed=3, want=True)
        assert np.array_equal(J, ctx.download(tam.TAM_F_JMEAN_GLOBAL)) and J.max() > 0
        for steps in (0, 1, 40):
            T = ctx.heat_steps(steps, want=True)
            assert np.array_equal(T, ctx.download(tam.TAM_F_TEMP))
