"""Weights with more row-blocks than a launch has grid rows."""
import pytest

from gpu_util import cuda, seeded_normal

pytestmark = pytest.mark.gpu


def test_more_row_blocks_than_a_grid_has_rows():
    """A K-major product of a weight with 65536 row-blocks and one chunk of columns is served."""
    from sten_b200 import _native as nat, ops
    rows, cols, tokens = 262144, 64, 1040
    w = seeded_normal((rows, cols), 1).to(cuda())
    val, idx = ops.sparsify(w.unsqueeze(0), 1, 4, 16)
    dense = ops.densify(val, idx, 1, rows, cols, 1, 4, 16)[0]
    x = seeded_normal((cols, tokens), 2).to(cuda())
    y = ops.spmm(val, idx, rows, cols, 1, 4, 16, x, layout=nat.NMG_ACT_K_MAJOR)
    for r in (0, 131000, rows - 512):
        want, sums = dense[r:r + 512].double() @ x.double(), dense[r:r + 512].double().abs() @ x.double().abs()
        assert bool(((y[r:r + 512].double() - want).abs() <= 1e-5 * sums).all())
    assert ops.read_status() == 0
