"""Edges of the two-pass product: tile widths, rows of narrow tiles, chunks of the reduction, ragged rows, columns and reductions."""
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


# rows of tiles (256 tokens) x columns whose last wave is filled with narrow tiles: 128 and 192 wide, the ragged last row and column
# among them; then one wave, where there are none
@pytest.mark.parametrize("M,tokens", [(2816, 7 * 256), (2813, 9 * 256 - 3), (2500, 10 * 256 - 100), (5000, 8 * 256 - 1), (4096, 5 * 256), (1000, 1600)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_16bit_rows_of_narrow_tiles(dtype, M, tokens):
    from sten_b200 import _native as nat, ops
    dev = cuda()
    K = 200
    w = (seeded_normal((M, K), 1) * K ** -0.5).to(dev)
    val, idx = ops.sparsify(w.unsqueeze(0), 2, 4, 4)
    val = val.to(dtype)
    dense = ops.densify(val, idx, 1, M, K, 2, 4, 4)[0].double()
    x, b = seeded_normal((tokens, K), 2).to(dev, dtype), seeded_normal((M,), 3).to(dev, dtype)
    res = seeded_normal((tokens, M), 5).to(dev, dtype)
    want = x.double() @ dense.t() + b.double()
    rounding = 2.0 ** (-11 if dtype == torch.float16 else -8)  # of one result; the sums are fp32

    def close(got, ref):
        assert float(((got.double() - ref).abs() / (ref.abs() + 1)).max()) <= rounding

    close(ops.spmm(val, idx, M, K, 2, 4, 4, x, bias=b, algo=nat.NMG_ALGO_TENSOR), want)
    close(ops.spmm(val, idx, M, K, 2, 4, 4, x, bias=b, layout=nat.NMG_ACT_TOKEN_MAJOR_OUT_ROWS, algo=nat.NMG_ALGO_TENSOR).t(), want)
    close(ops.spmm(val, idx, M, K, 2, 4, 4, x, bias=b, activation="gelu", residual=res, algo=nat.NMG_ALGO_TENSOR), torch.nn.functional.gelu(want) + res.double())
    assert ops.read_status() == 0
