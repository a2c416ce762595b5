"""The plane Jacobi kernel with three groups of four points per thread (planes of 8196 to 12288 points) against the
grid-barrier kernel: identical grids and sweep counts."""
import pytest

from qmtools import _native as N
from test_gpu_jacobi_plane import _solve

pytestmark = pytest.mark.gpu


# three groups of four points per thread: whole, with a last group partly filled and rows that straddle warps, and the
# fewest planes that the automatic choice gives this kernel (550,000 points)
@pytest.mark.parametrize("fn", ["qmt_jacobi", "qmt_jacobi_dirichlet"])
@pytest.mark.parametrize("shape", [(96, 96, 64), (100, 100, 60), (96, 128, 45), (92, 92, 148)])
def test_three_groups_identical_to_grid_barrier_kernel(fn, shape):
    import torch
    groups = -(-(shape[0] // 4 * shape[1]) // 1024)
    assert groups == 3 and shape[0] * shape[1] * shape[2] >= 550000 and shape[2] <= 148
    a = _solve(fn, shape, 30, 0)
    b = _solve(fn, shape, 30, 1)
    assert a[:2] == b[:2] == (N.OK, 30)
    assert torch.equal(a[3], b[3])
    assert a[2] == pytest.approx(b[2], rel=1e-12)      # the residual's order of summation differs
