"""The reference-mode FP64 step on grids large enough for columns of several planes, where
skin and cells with properties of their own alternate along them (a face's coefficient is
carried from plane to plane): every voxel bit for bit against numpy's IEEE operations."""
import numpy as np
import pytest

from test_gpu_ref_classes import _step

pytestmark = pytest.mark.gpu


# 25 and 27 blocks of row pairs: columns of 2 and 3 planes, a last one of 1 or 2
@pytest.mark.parametrize("shape", [(80, 79, 47), (81, 85, 80), (80, 80, 61)])
@pytest.mark.parametrize("kind", ["all", "planes", "spots", "none"])
def test_bitwise_along_columns(tam, shape, kind):
    F = tam
    rng = np.random.default_rng(sum(shape))
    with tam.Context(tam.default_params(nxg=shape[0], nyg=shape[1], nzg=shape[2])) as ctx:
        ctx.update_props(500.0)
        K, D, C = (ctx.download(f) for f in (F.TAM_F_KAPPA, F.TAM_F_DENSITY, F.TAM_F_HEATCAP))
        own = np.zeros(shape, dtype=bool)
        if kind == "all":
            own[:] = True
        elif kind == "planes":  # whole warps change from plane to plane
            own[:, :, rng.random(shape[2]) < 0.5] = True
        elif kind == "spots":
            own = rng.random(shape) < 0.02
        for f, A in ((F.TAM_F_KAPPA, K), (F.TAM_F_DENSITY, D), (F.TAM_F_HEATCAP, C)):
            A[1:-1, 1:-1, 1:-1][own] *= rng.uniform(0.9, 1.1, own.sum())
            ctx.upload(f, A)
        T = ctx.download(F.TAM_F_TEMP)
        T[1:-1, 1:-1, 1:-1] += rng.uniform(0.0, 5.0, shape)
        J, Q = rng.uniform(0.0, 1e9, shape), np.zeros(shape)
        ctx.upload(F.TAM_F_TEMP, T)
        ctx.upload(F.TAM_F_JMEAN_GLOBAL, J)
        for _ in range(2):
            st, cf = ctx.state(), ctx.download(F.TAM_F_COEFF)
            T, Q = _step(T, K, D, C, cf, J, Q, st)
            got = ctx.heat_steps(1, want=True)
            assert np.array_equal(got.view(np.uint64), T.view(np.uint64))


def test_no_slower_with_properties_of_their_own(tam):
    """A grid of per-voxel conductivities takes about 3.7 times the step of unheated skin (4.5 times
    with every coefficient formed twice)."""
    us = []
    for own in (False, True):
        with tam.Context(tam.default_params(nxg=128, nyg=128, nzg=128)) as ctx:
            if own:
                K = ctx.download(tam.TAM_F_KAPPA)
                ctx.upload(tam.TAM_F_KAPPA, K * np.random.default_rng(1).uniform(0.9, 1.1, K.shape))
            best = []
            for _ in range(6):
                ctx.heat_steps(48)
                best.append(ctx.timing()[1])
            us.append(min(best))
    assert us[1] <= 4.1 * us[0]
