"""The reference loop's step that normalises the pass's tally itself (replayed and
launched) against a pass and a step of their own calls: grids of even and odd rows
and several blocks, both precisions, absorbed weight included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(9, 8, 7), (40, 40, 40), (33, 41, 26)])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("graph", [0, 1])
def test_loop_equals_its_calls(tam, shape, precision, graph):
    iters = 20
    out = []
    for loop in (True, False):
        p = tam.default_params(nxg=shape[0], nyg=shape[1], nzg=shape[2], power=2.0, pulse_type=tam._abi.TAM_PULSE_TOPHAT,
                               precision=precision, nphotons=20000)
        with tam.Context(p) as ctx:
            ctx.init_thermal()
            ctx.set_tuning("heat.graph", graph)
            if loop:
                ctx.step_coupled(iters, seed=5)
            else:
                for k in range(iters):
                    ctx.mc_pass(20000, seed=5, stream=k)
                    ctx.heat_steps(1)
                    ctx.arrhenius()
                    ctx.update_props(p.ablate_temp)
            out.append([ctx.download(f) for f in (tam.TAM_F_JMEAN_GLOBAL, tam.TAM_F_JMEAN, tam.TAM_F_TEMP)] + [ctx.tallies()])
    (J0, j0, T0, t0), (J1, j1, T1, t1) = out
    # atomic additions come in another order: 2e4 packets, 2^-53 each
    tol = 2e4 * 2.0**-53
    assert J0.max() > 0
    assert np.abs(J1 - J0).max() <= tol * J0.max() and np.abs(j1 - j0).max() <= tol * j0.max()
    assert abs(t1["absorbed"] - t0["absorbed"]) <= tol * t0["absorbed"]
    assert np.abs(T1 - T0).max() <= iters * (tol if precision == 0 else 2.0**-22) * T0.max()
