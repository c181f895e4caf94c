"""Edges of the two-pass fp32 product: tile widths, chunks of the reduction, ragged rows, columns and reductions."""
import pytest
import torch

from gpu_util import cuda, seeded_normal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,tokens", [(100, 700, 1024), (3072, 40, 1500), (640, 513, 1031), (1028, 1100, 2049), (130, 4096, 1100), (2000, 520, 5000)])
@pytest.mark.parametrize("n,m", [(1, 4), (2, 4)])
def test_fp32_two_pass_tiles(n, m, M, K, tokens):
    from sten_b200 import _native as nat, ops
    dev = cuda()
    w = (seeded_normal((M, K), 1) * K ** -0.5).to(dev)
    val, idx = ops.sparsify(w.unsqueeze(0), n, m, 4)
    dense = ops.densify(val, idx, 1, M, K, n, m, 4)[0].double()
    rel = lambda a, b: float((a.double() - b).norm() / b.norm())  # noqa: E731
    x, b, dy = seeded_normal((tokens, K), 2).to(dev), seeded_normal((M,), 3).to(dev), seeded_normal((tokens, M), 4).to(dev)
    res = seeded_normal((tokens, M), 5).to(dev)
    want = x.double() @ dense.t() + b.double()
    y = ops.spmm(val, idx, M, K, n, m, 4, x, bias=b, algo=nat.NMG_ALGO_TENSOR)
    assert rel(y, want) <= 5e-6
    yt = ops.spmm(val, idx, M, K, n, m, 4, x, bias=b, layout=nat.NMG_ACT_TOKEN_MAJOR_OUT_ROWS, algo=nat.NMG_ALGO_TENSOR)
    assert torch.equal(yt.t(), y)  # the operands' roles are exchanged, the sums are not
    fused = ops.spmm(val, idx, M, K, n, m, 4, x, bias=b, activation="gelu", residual=res, algo=nat.NMG_ALGO_TENSOR)
    assert rel(fused, torch.nn.functional.gelu(want) + res.double()) <= 5e-6
    assert rel(ops.spmm_t(val, idx, M, K, n, m, 4, dy, algo=nat.NMG_ALGO_TENSOR), dy.double() @ dense) <= 5e-6
    assert ops.read_status() == 0
