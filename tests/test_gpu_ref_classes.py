"""The reference-mode FP64 step where most cells hold unheated skin (known face
coefficients, shared products) next to heated ones and the halo: every voxel
bit for bit against numpy's IEEE operations, at the edges of the kernel's row
pairs, warps and z columns, with the property update between the steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _step(T, K, D, C, coeff, J, Q, st):
    """src/3dFD.f90:113-187 in float64, in the Fortran's order of operations."""
    c = (slice(1, -1),) * 3

    def sh(A, ax, o):
        idx = [slice(1, -1)] * 3
        idx[ax] = slice(1 + o, A.shape[ax] - 1 + o)
        return A[tuple(idx)]

    u = []
    for ax, dd in enumerate((st.dx, st.dy, st.dz)):
        id2 = 1.0 / (dd * dd)
        a, d = ((0.5 * ((0.5 * (K[c] + sh(K, ax, o))) / ((0.5 * (D[c] + sh(D, ax, o))) * (0.5 * (C[c] + sh(C, ax, o)))))) * id2
                for o in (-1, 1))
        u.append(((a * sh(T, ax, -1)) - ((2.0 * (0.5 * (a + d))) * T[c])) + (d * sh(T, ax, 1)))
    inc = st.delt * ((u[0] + u[1]) + u[2])
    energy = (((st.laser_on * J) * st.delt) * st.volume_voxel) + ((C[c] * st.mass_voxel) * inc)
    heat = (T[c] + inc) + ((st.laser_on * coeff[c]) * J)
    boil = (T[c] >= 373.0) & (Q < st.qvapor) & (energy > 0.0)
    qn = Q + energy
    out = T.copy()
    out[c] = np.where(boil, 373.0, heat)
    return out, np.where(boil, np.where(qn < st.qvapor, qn, st.qvapor), Q)


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 3), (5, 4, 3), (31, 3, 4), (32, 2, 9), (33, 7, 17), (64, 5, 2), (40, 40, 33)])
@pytest.mark.parametrize("heated", [False, True])
def test_bitwise_with_skin_and_heated_cells(tam, shape, heated):
    F = tam
    nx, ny, nz = shape
    rng = np.random.default_rng(nx * 100 + ny)
    with tam.Context(tam.default_params(nxg=nx, nyg=ny, nzg=nz)) as ctx:
        ctx.update_props(500.0)
        T = ctx.download(F.TAM_F_TEMP)
        T[1:-1, 1:-1, 1:-1] += rng.uniform(0.0, 5.0, shape)
        J, Q = np.zeros(shape, order="F"), np.zeros(shape, order="F")
        if heated:
            hot = (slice(nx // 3, nx // 3 + max(1, nx // 4)), slice(ny // 2, ny), slice(max(0, nz - 3), nz))
            J[hot] = rng.uniform(0.0, 5e9, J[hot].shape)
            Q[hot] = ctx.state().qvapor * rng.uniform(0.0, 0.9, J[hot].shape)
            T[1:-1, 1:-1, 1:-1][hot] = 374.0
        for f, A in ((F.TAM_F_TEMP, T), (F.TAM_F_JMEAN_GLOBAL, J), (F.TAM_F_Q, Q)):
            ctx.upload(f, A)
        for n in range(4):
            K, D, C, cf = (ctx.download(f) for f in (F.TAM_F_KAPPA, F.TAM_F_DENSITY, F.TAM_F_HEATCAP, F.TAM_F_COEFF))
            T, Q = ctx.download(F.TAM_F_TEMP), ctx.download(F.TAM_F_Q)
            st = ctx.state()
            Tn, Qn = _step(T, K, D, C, cf, J, Q, st)
            got = ctx.heat_steps(1, want=True)
            assert np.array_equal(got.view(np.uint64), Tn.view(np.uint64)), (n, np.argwhere(got != Tn)[:4])
            assert np.array_equal(ctx.download(F.TAM_F_Q).view(np.uint64), Qn.view(np.uint64))
            ctx.update_props(500.0)
            if heated and n:  # the property update reached the heated cells
                assert (ctx.download(F.TAM_F_KAPPA)[1:-1, 1:-1, 1:-1] != K[1, 1, 1]).any() or nx * ny * nz == 1
