"""The fused tensor-core matmul where its tiling changes: tile widths in steps of 32 tokens, one and several ranges of the
reduction axis (partial tiles exchanged between the CTAs of a cluster), ragged last tiles in every direction, one k-block per
range, and the fp32 mode's accumulation chunks.  Reference: float64 matmul of the rounded operands."""
import pytest
import torch

from gpu_util import cuda, seeded_normal

pytestmark = pytest.mark.gpu

CASES = [
    # n, m, g, M, K, tokens
    (2, 4, 16, 128, 64, 1),       # one tile, one k-block
    (2, 4, 16, 129, 72, 33),      # a second feature tile with one row, a ragged second k-block, 33 of 64 token columns
    (1, 8, 16, 1000, 1032, 31),   # ranges of the reduction with a ragged last one
    (1, 16, 4, 384, 4160, 97),    # eight ranges, an odd token count in the exchange
    (2, 8, 16, 136, 4104, 257),   # two token tiles of 160, many k-blocks per CTA
    (1, 4, 8, 4096, 520, 96),     # as many tiles as SMs: no exchange
    (2, 4, 4, 260, 1000, 200),    # rows that are not 4-byte pairs apart in the output are covered by M = 129 and 1000
]


@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 1e-2), (torch.float16, 2e-3), (torch.float32, 1e-5)])
@pytest.mark.parametrize("n,m,g,M,K,tokens", CASES)
def test_fused_matmul_tiles(n, m, g, M, K, tokens, dtype, tol):
    from sten_b200 import _native as nat, ops
    dev = cuda()
    w = (seeded_normal((M, K), 1) * K ** -0.5).to(dtype).to(dev)
    val, idx = ops.sparsify(w.unsqueeze(0), n, m, g)
    dense = ops.densify(val, idx, 1, M, K, n, m, g)[0].double()
    x = seeded_normal((tokens, K), 2).to(dtype).to(dev)
    bias, res = seeded_normal((M,), 3).to(dtype).to(dev), seeded_normal((tokens, M), 4).to(dtype).to(dev)
    rel = lambda a, b: float((a.double() - b).norm() / b.norm())  # noqa: E731
    product = x.double() @ dense.t()
    y = ops.spmm(val, idx, M, K, n, m, g, x, algo=nat.NMG_ALGO_TENSOR)
    assert rel(y, product) <= tol
    assert torch.equal(y, ops.spmm(val, idx, M, K, n, m, g, x, algo=nat.NMG_ALGO_TENSOR))  # ranges are added in a fixed order
    fused = ops.spmm(val, idx, M, K, n, m, g, x, bias=bias, activation="gelu", residual=res, algo=nat.NMG_ALGO_TENSOR)
    assert rel(fused, torch.nn.functional.gelu(product + bias.double()) + res.double()) <= tol
    rows = ops.spmm(val, idx, M, K, n, m, g, x, bias=bias, layout=nat.NMG_ACT_TOKEN_MAJOR_OUT_ROWS, algo=nat.NMG_ALGO_TENSOR)
    assert rel(rows, (product + bias.double()).t()) <= tol
    if M % 8 == 0 or dtype == torch.float32:
        dy = seeded_normal((tokens, M), 5).to(dtype).to(dev)
        assert rel(ops.spmm_t(val, idx, M, K, n, m, g, dy, algo=nat.NMG_ALGO_TENSOR), dy.double() @ dense) <= tol
    assert ops.read_status() == 0


@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 1e-2), (torch.float16, 2e-3)])
@pytest.mark.parametrize("n,m,g,M,K,tokens", [(1, 8, 16, 1023, 777, 333), (2, 4, 16, 130, 250, 1), (2, 4, 4, 66, 1031, 1500)])
def test_rows_tma_cannot_read_are_laid_out_again(n, m, g, M, K, tokens, dtype, tol):
    """Odd reduction lengths, and aligned ones behind an odd offset, on both products; every token count's kernel."""
    from sten_b200 import ops
    dev = cuda()
    w = (seeded_normal((M, K), 1) * K ** -0.5).to(dtype).to(dev)
    val, idx = ops.sparsify(w.unsqueeze(0), n, m, g)
    dense = ops.densify(val, idx, 1, M, K, n, m, g)[0].double()
    rel = lambda a, b: float((a.double() - b).norm() / b.norm())  # noqa: E731
    for pad in (0, 3):
        x = seeded_normal((tokens, K + pad), 2).to(dtype).to(dev)[:, pad:]
        assert rel(ops.spmm(val, idx, M, K, n, m, g, x), x.double() @ dense.t()) <= tol
        dy = seeded_normal((tokens, M + pad), 5).to(dtype).to(dev)[:, pad:]
        assert rel(ops.spmm_t(val, idx, M, K, n, m, g, dy), dy.double() @ dense) <= tol
    assert ops.read_status() == 0


@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 1e-2), (torch.float32, 1e-5)])
@pytest.mark.parametrize("tokens", [1, 33, 63, 64, 200, 700])
def test_k_major_columns(tokens, dtype, tol):
    """torch.mm through the plugin: a handful of columns, and the fp32 mode's transposing split at ragged tile edges."""
    import sten_b200 as sten
    sten.set_dispatch_failure("raise")
    dev, M, K = cuda(), 200, 333
    lin = torch.nn.Linear(K, M, bias=False).to(dev).to(dtype)
    sb = sten.SparsityBuilder()
    sb.set_weight("weight", initial_sparsifier=sten.GroupedNMSparsifier(2, 4, 16), out_format=sten.GroupedNMTensor)
    w = sb.get_sparse_model(lin).weight
    b = seeded_normal((K, tokens), 7).to(dtype).to(dev)
    with torch.no_grad():
        c = torch.mm(w, b)
    want = w.wrapped_tensor.to_dense().double() @ b.double()
    assert float((c.double() - want).norm() / want.norm()) <= tol


@pytest.mark.parametrize("n,m", [(1, 4), (2, 4), (1, 8), (2, 8), (1, 16)])
@pytest.mark.parametrize("K,tokens", [(256, 1), (256, 63), (1000, 8), (4096, 33), (16384, 63)])
def test_few_fp32_columns_are_summed_as_accurately_as_by_fp32_fmas(n, m, K, tokens):
    """torch.mm of a handful of columns runs on the tensor cores when a packed copy is there, and on fp32 FMAs when it is not."""
    from sten_b200 import _native as nat, ops
    dev, M = cuda(), 256
    w = (seeded_normal((M, K), 1) * K ** -0.5).to(dev)
    val, idx = ops.sparsify(w.unsqueeze(0), n, m, 4)
    b = seeded_normal((K, tokens), 2).to(dev)
    want = ops.densify(val, idx, 1, M, K, n, m, 4)[0].double() @ b.double()
    err = lambda c: float((c.double() - want).norm() / want.norm())  # noqa: E731
    packed = ops.pack(val, idx, M, K, n, m, 4)
    tensor = ops.spmm(val, idx, M, K, n, m, 4, b, layout=nat.NMG_ACT_K_MAJOR, packed=packed)
    fma = ops.spmm(val, idx, M, K, n, m, 4, b, layout=nat.NMG_ACT_K_MAJOR, algo=nat.NMG_ALGO_SIMT)
    assert not torch.equal(tensor, fma)
    assert err(tensor) <= err(fma)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("tokens", [3, 300, 2000])
def test_gelu_of_infinities_and_nan(tokens, dtype):
    """As torch's exact GELU has them: infinity stays, minus infinity and NaN give NaN; large finite values pass through."""
    from sten_b200 import _native as nat, ops
    M, K = 256, 128
    w = (seeded_normal((M, K), 1) * K ** -0.5).to(dtype).to(cuda())
    val, idx = ops.sparsify(w.unsqueeze(0), 2, 4, 16)
    x = seeded_normal((tokens, K), 2).to(dtype).to(cuda())
    bias = torch.zeros(M, dtype=dtype, device=cuda())
    big = 6e4 if dtype == torch.float16 else 3e38
    bias[:5] = torch.tensor([float("inf"), -float("inf"), float("nan"), big, -big], dtype=dtype)
    for algo in (nat.NMG_ALGO_AUTO, nat.NMG_ALGO_SIMT):
        y = ops.spmm(val, idx, M, K, 2, 4, 16, x, bias=bias, activation="gelu", algo=algo)[:, :5].float()
        want = torch.nn.functional.gelu(bias[:5].double()).float().expand(tokens, 5)
        assert torch.equal(y.isnan(), want.isnan())
        assert torch.equal(y[:, 0], want[:, 0]) and float((y[:, 3] / want[:, 3] - 1).abs().max()) < 1e-2 and float(y[:, 4].abs().max()) == 0
