"""Edges of the conversion kernels' tiles: partly filled warps, remainder tiles, unaligned rows, ties and zeros."""
import math

import numpy as np
import pytest
import torch

from gpu_util import cuda, np_of, seeded_normal
from oracle import nmg_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,m,g", [(1, 4, 1), (1, 4, 16), (2, 4, 3), (2, 4, 16), (2, 4, 300), (1, 8, 16), (2, 8, 2), (2, 8, 16),
                                   (1, 16, 16), (2, 8, 100), (1, 4, 2000)])
def test_sparsify_and_densify_at_tile_edges(n, m, g, dtype):
    """One tile, tiles that do not fill a warp, cut tiles in both directions, rows without 16-byte alignment; few distinct
    values (ties) with many zeros, and random weights."""
    from sten_b200 import ops
    cc = g * math.comb(m, n)
    for M, K, off in [(m, cc, 0), (3 * m + 1, cc, 1), (2 * m, 2 * cc + cc // 2 + 1, 0)]:
        for ties in (False, True):
            w = seeded_normal((M, K + off), M + K)
            if ties:
                w = w.round()
            w = w.to(dtype)[:, off:]
            val_o, idx_o = orc.sparsify(w.float().numpy(), n, m, g)
            val, idx = ops.sparsify(w.to(cuda())[None], n, m, g)
            assert np.array_equal(np_of(idx), idx_o) and np.array_equal(np_of(val.float()), val_o)
            assert np.array_equal(np_of(ops.densify(val, idx, 1, M, K, n, m, g).float())[0], orc.densify(val_o, idx_o, (M, K), n, m, g))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,m,g", [(1, 4, 16), (2, 4, 3), (2, 4, 16), (2, 8, 16), (1, 16, 16), (3, 6, 4)])
@pytest.mark.parametrize("B,K,off,tail", [(1, 96, 8, 0), (1, 96, 1, 0), (1, 500, 0, 3), (2, 448, 8, 8), (2, 451, 1, 2), (3, 40, 0, 0)])
def test_densify_into_rows_of_a_wider_matrix(B, K, off, tail, n, m, g, dtype):
    """A pitch larger than the row, aligned and unaligned bases: the rows are the dense weight, what lies between them stays."""
    from sten_b200 import _native as nat, ops
    M = 2 * m + 1
    val, idx = ops.sparsify(seeded_normal((B, M, K), M + K).to(dtype).to(cuda()), n, m, g)
    pitch = off + K + tail
    d = torch.full((B, M, pitch), 7.0, dtype=dtype, device=cuda())
    code = nat.NMG_F32 if dtype == torch.float32 else nat.NMG_BF16
    nat.check(nat.lib().nmg_densify(val.data_ptr(), idx.data_ptr(), B, M, K, n, m, g, code, d[:, :, off:].data_ptr(), pitch, M * pitch,
                                    torch.cuda.current_stream().cuda_stream))
    assert torch.equal(d[:, :, off:off + K], ops.densify(val, idx, B, M, K, n, m, g))
    assert bool((d[:, :, :off] == 7.0).all()) and bool((d[:, :, off + K:] == 7.0).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,m,g,B,M,K,off", [(2, 4, 16, 1, 64, 1152, 0), (1, 8, 16, 2, 130, 1000, 3), (2, 8, 16, 1, 24, 449, 0), (1, 16, 4, 1, 17, 700, 0),
                                              (1, 4, 4, 3, 36, 40, 0), (2, 4, 3, 1, 20, 100, 1), (1, 4, 512, 1, 9, 5000, 0)])
def test_gather_at_tile_edges(n, m, g, B, M, K, off, dtype):
    """Values of another tensor at a layout's positions, against the densified mask: whole and cut items, unaligned rows."""
    from sten_b200 import ops
    w = seeded_normal((B, M, K), 1).to(dtype).to(cuda())
    val, idx = ops.sparsify(w, n, m, g)
    other = seeded_normal((B, M, K + off), 2).to(dtype).to(cuda())[:, :, off:]
    got = ops.gather_layout(other, idx, n, m, g)
    mask = ops.densify(torch.ones_like(val), idx, B, M, K, n, m, g)
    assert torch.equal(ops.densify(got, idx, B, M, K, n, m, g), torch.where(mask != 0, other, torch.zeros_like(other)))
    assert torch.equal(ops.gather_layout(w, idx, n, m, g), val)


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-6), (torch.bfloat16, 4e-3), (torch.float16, 5e-4)])
@pytest.mark.parametrize("rows,cols,off", [(1, 1, 0), (31, 8, 0), (33, 257, 0), (4096, 1000, 0), (1000, 4096, 3), (5000, 40, 0), (70000, 16, 8)])
def test_column_sums(rows, cols, off, dtype, tol):
    from sten_b200 import _native as nat
    x = seeded_normal((rows, cols + off), 3).to(dtype).to(cuda())[:, off:]
    got, want = nat.host().column_sum(x), x.double().sum(0)
    assert got.dtype == dtype and float((got.double() - want).norm() / want.norm()) <= tol
    assert torch.equal(nat.host().column_sum(x), got)


@pytest.mark.parametrize("rows", [1, 100, 1000, 4096, 70000])
def test_fp32_column_sums_err_no_more_than_a_torch_reduction(rows):
    from sten_b200 import _native as nat
    for x in (seeded_normal((rows, 512), 5) + 0.3, seeded_normal((rows, 512), 6), seeded_normal((rows, 512), 7).abs()):
        x = x.to(cuda())
        got, want = nat.host().column_sum(x).double(), x.double().sum(0)
        assert float((got - want).norm()) <= float((x.sum(0).double() - want).norm())
    for bad, expect in ((float("inf"), float("inf")), (-float("inf"), -float("inf")), (float("nan"), float("nan"))):
        y = x.clone()
        y[rows // 2, 7] = bad
        s = nat.host().column_sum(y)
        assert torch.equal(s[8:], nat.host().column_sum(x)[8:]) and np.array_equal(np_of(s[7:8]), np.float32([expect]), equal_nan=True)
