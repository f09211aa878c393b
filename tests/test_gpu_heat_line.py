"""The line form of the FP32 heat step (rows of any width) against the FP64 step: the
smallest grids, rows and planes that end inside a warp, a block or a run of planes,
one and several classes, convective and fixed faces, with and without a source."""
import numpy as np
import pytest

from test_gpu_heat_quad import _check, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 1, 2), (1, 5, 3), (7, 3, 2), (31, 9, 6), (33, 8, 7), (127, 2, 5), (129, 2, 9), (257, 3, 4)])
@pytest.mark.parametrize("grid", ["one", "ball", "random"])
@pytest.mark.parametrize("robin,on", [(0, True), (0b111111, False), (0b100110, True)])
def test_line_step(tam, shape, grid, robin, on):
    T0, O0, _ = _run(tam, shape, grid, robin, on, 0, 0)
    T, O, err = _run(tam, shape, grid, robin, on, 1, 1)
    assert err == 0
    _check(T, O, T0, O0)


@pytest.mark.parametrize("grid", ["one", "ball"])
def test_line_step_is_independent_of_the_planes_per_block(tam, grid):
    shape = (37, 15, 19)
    a = _run(tam, shape, grid, 0b111111, True, 1, 1, 1)
    for zchunk in (0, 2, 3, 5, 8, 19):
        b = _run(tam, shape, grid, 0b111111, True, 1, 1, zchunk)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
