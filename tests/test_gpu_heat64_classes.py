"""The FP64 heat step on thermal classes against the per-voxel FP64 step
("heat.cls" 0, the form the oracle tests cover) on grids of one and of several
materials, at the edges of its 32 x 8 tiles and with convective faces."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MATS = [(0.0, 0.0, 0.0, 1.0, 0.56, 1070.0, 3400.0), (1.0, 20.0, 0.8, 1.4, 0.21, 1200.0, 3590.0),
        (0.3, 12.0, 0.9, 1.4, 0.37, 1200.0, 3300.0), (0.1, 8.0, 0.9, 1.4, 0.16, 1000.0, 2674.0)]


def _ctx(tam, shape, grid, robin, seed):
    nx, ny, nz = shape
    p = tam.default_params(nxg=nx, nyg=ny, nzg=nz, xmax=0.01 * nx / 2, ymax=0.012 * ny / 2, zmax=0.008 * nz / 2, mode=1,
                           precision=0, pulse_type=1, power=2.0, energy_per_pixel=1e9, total_time=1e6)
    c = tam.default_config(nmat=len(MATS), retrace_fraction=0.0)
    for i, m in enumerate(MATS):
        tam.set_material(c, i, *m)
    for f in range(6):
        c.bc_type[f] = 1 if robin >> f & 1 else 0
        c.bc_h[f] = 10.0 * (f + 1)
    ctx = tam.Context(p, c)
    rng = np.random.default_rng(seed)
    if grid:
        ctx.upload(tam.TAM_F_MATERIAL, rng.integers(1, 4, size=shape).astype(np.uint8))
    T = np.full(tuple(n + 2 for n in shape), 310.15, order="F")
    T[1:-1, 1:-1, 1:-1] = rng.uniform(305.0, 380.0, size=shape)  # through the damage window, boiling and ablation
    ctx.upload(tam.TAM_F_TEMP, T)
    ctx.upload(tam.TAM_F_JMEAN_GLOBAL, rng.uniform(0.0, 1e7, size=shape))
    return ctx


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 3, 5), (31, 7, 17), (32, 8, 16), (33, 9, 33), (70, 20, 6)])
@pytest.mark.parametrize("grid", [False, True])
@pytest.mark.parametrize("robin", [0, 0b100000, 0b111111])
def test_matches_per_voxel_step(tam, shape, grid, robin):
    F = tam
    out = []
    for cls in (1, 0):
        with _ctx(tam, shape, grid, robin, 7) as ctx:
            ctx.set_tuning("heat.cls", cls)
            ctx.heat_steps(20)
            out.append([ctx.download(f) for f in (F.TAM_F_TEMP, F.TAM_F_Q, F.TAM_F_TISSUE, F.TAM_F_MATERIAL)])
    (T, Q, O, m), (T0, Q0, O0, m0) = out
    # both round each of ~20 operations per step differently: 20 steps x 20 x 1.1e-16 relative
    assert np.abs(T / T0 - 1).max() < 1e-12
    assert np.array_equal(m, m0)
    assert np.abs(Q - Q0).max() <= 1e-9 * max(1e-300, np.abs(Q0).max())
    assert np.abs(O - O0).max() <= 1e-9 * max(1e-300, np.abs(O0).max())


def test_follows_material_and_state(tam, tmp_path):
    """A new material grid, a loaded state and per-voxel properties each reach the next step."""
    shape, F = (24, 10, 9), tam
    with _ctx(tam, shape, True, 0, 3) as ctx, _ctx(tam, shape, True, 0, 3) as ref:
        ref.set_tuning("heat.cls", 0)
        g = np.ones(shape, dtype=np.uint8)
        g[5:9, 2:7, 1:4] = 3
        for c in (ctx, ref):
            c.heat_steps(2)
            c.upload(F.TAM_F_MATERIAL, g)
            c.heat_steps(3)
            c.save_state(str(tmp_path / f"s{c is ref}"))
            c.upload(F.TAM_F_MATERIAL, np.full(shape, 2, dtype=np.uint8))
            c.heat_steps(2)
            c.load_state(str(tmp_path / f"s{c is ref}"))
            c.heat_steps(4)
            c.upload(F.TAM_F_KAPPA, np.full(tuple(n + 2 for n in shape), 0.4))
            c.heat_steps(2)
        assert np.abs(ctx.download(F.TAM_F_TEMP) / ref.download(F.TAM_F_TEMP) - 1).max() < 1e-12
