"""fp32 products on the tensor cores keep every value's own precision: values far below the largest of their row, in the activation or in
the weight, count as much as they do in plain fp32 arithmetic, wherever an output meets only those."""
import pytest
import torch

from gpu_util import cuda, seeded_normal

pytestmark = pytest.mark.gpu

# Relative to the sum of magnitudes of an output.  An accumulator takes 96 steps before it is added up in fp32; a step aligns its 16 products and
# the accumulator to the largest of them and cuts each off, at 2^-25 of the sum of magnitudes or below.  The operands are exact sums of three
# pieces; of the nine products of pieces the three smallest, each at most 2^-24 of the whole, are left out.
BOUND = 96 * 17 * 2.0 ** -25 + 3 * 2.0 ** -24

M, K = 512, 1024


def _spread(bits):
    """Powers of two over 2^bits, one per column."""
    return torch.exp2(torch.randint(-bits // 2, bits // 2 + 1, (K,), generator=torch.Generator().manual_seed(5)).float())


def _operands(kind, bits, tokens):
    """Weight (before magnitude selection), activation, gradient of the output."""
    w, x, dy = seeded_normal((M, K), 1), seeded_normal((tokens, K), 2), seeded_normal((tokens, M), 3)
    cols = torch.arange(K)
    if kind == "scales":  # features of different scales, weights that compensate
        s = _spread(bits)
        w, x = w / s, x * s
        r = s[:M].clone()
        return w, x, dy * r
    if kind == "tiny":  # a third of the features far below the others, every fourth output meets only those
        small = cols % 10 < 3
        x[:, small] *= 2.0 ** -bits
        w[::4, ~small] = 0
        w[:, cols % 20 < 3] *= 2.0 ** bits
        dy[:, torch.arange(M) % 3 == 0] *= 2.0 ** -bits
        return w, x, dy
    if kind == "half":  # the same with half of the features and no weights that compensate
        small = cols % 2 == 0
        x[:, small] *= 2.0 ** -bits
        w[1::4, ~small] = 0
        dy[:, torch.arange(M) % 2 == 0] *= 2.0 ** -bits
        w[1::2, ::8] = 0
        return w, x, dy
    assert kind == "outlier"  # one weight per row (and some columns) far above the others, over features that are zero
    big = (torch.arange(M) * 37) % 64
    w[torch.arange(M), big] = 2.0 ** bits
    x[:, :64] = 0
    x[:, 1] = 2.0 ** -bits
    dy[:, :3] = 0
    w[:3, 64:] = 2.0 ** bits
    return w, x, dy


def _close(got, a, b):
    err, ref = (got.double() - a @ b.t()).abs(), a.abs() @ b.abs().t()
    bad = err > BOUND * ref + 2.0 ** -148
    assert not bool(bad.any()), (int(bad.sum()), float((err / ref.clamp(min=2.0 ** -140)).max()))


def _products(n, m, g, w, x, dy):
    """The three products through the tensor-core kernels, each with what it should be close to."""
    from sten_b200 import _native as nat, ops
    w = w.to(cuda())
    val, idx = ops.sparsify(w.unsqueeze(0), n, m, g)
    dense = ops.densify(val, idx, 1, M, K, n, m, g)[0]
    copy = ops.pack(val, idx, M, K, n, m, g) if (n, m) != (3, 6) else None
    x, dy = x.to(cuda()), dy.to(cuda())
    d = dense.double()
    yield ops.spmm(val, idx, M, K, n, m, g, x, packed=copy, algo=nat.NMG_ALGO_TENSOR), x.double(), d
    yield (ops.spmm(val, idx, M, K, n, m, g, x.t().contiguous(), layout=nat.NMG_ACT_K_MAJOR, packed=copy, algo=nat.NMG_ALGO_TENSOR).t(), x.double(), d)
    yield ops.spmm_t(val, idx, M, K, n, m, g, dy, packed=copy, algo=nat.NMG_ALGO_TENSOR), dy.double(), d.t()
    assert ops.read_status() == 0


@pytest.mark.parametrize("tokens", [1100, 300, 70, 40])  # two passes, fused, few columns
@pytest.mark.parametrize("n,m,g", [(1, 4, 16), (2, 4, 1), (3, 6, 3)])
@pytest.mark.parametrize("kind,bits", [("scales", 24), ("scales", 32), ("scales", 40), ("tiny", 24), ("tiny", 28), ("tiny", 40), ("half", 30),
                                       ("half", 40), ("outlier", 20), ("outlier", 30), ("outlier", 40)])
def test_far_apart(kind, bits, n, m, g, tokens):
    for got, a, b in _products(n, m, g, *_operands(kind, bits, tokens)):
        _close(got, a, b)


@pytest.mark.parametrize("tokens", [1100, 300, 70])
def test_mask_beside_small_values(tokens):
    """A masked feature of the type's largest magnitude over weights that are zero."""
    w, x, dy = seeded_normal((M, K), 1), seeded_normal((tokens, K), 2) * 1e-8, seeded_normal((tokens, M), 3) * 1e-8
    top = torch.finfo(torch.float32).max
    w[:, :8], w[:8] = 0, 0
    x[:, 3], x[::2, 5], dy[:, 2] = -top, top, -top
    for got, a, b in _products(2, 4, 4, w, x, dy):
        _close(got, a, b)


@pytest.mark.parametrize("tokens", [1024, 1025])  # fused with a copy, two passes
def test_unit_columns_return_the_weight(tokens):
    """Rows of the identity, scaled by powers of two: products of one term, which are exact."""
    from sten_b200 import _native as nat, ops
    n, m, g = 2, 4, 8
    w = (seeded_normal((M, K), 1) * _spread(60)).to(cuda())
    val, idx = ops.sparsify(w.unsqueeze(0), n, m, g)
    dense = ops.densify(val, idx, 1, M, K, n, m, g)[0]
    s = _spread(20).to(cuda())
    x = torch.zeros(tokens, K, device=cuda())
    x[:K] = torch.diag(s)
    copy = ops.pack(val, idx, M, K, n, m, g)
    y = ops.spmm(val, idx, M, K, n, m, g, x, packed=copy, algo=nat.NMG_ALGO_TENSOR)
    assert torch.equal(y[:K], (dense * s).t())
    y = ops.spmm(val, idx, M, K, n, m, g, x.t().contiguous(), layout=nat.NMG_ACT_K_MAJOR, packed=copy, algo=nat.NMG_ALGO_TENSOR)
    assert torch.equal(y[:, :K], dense * s)


@pytest.mark.parametrize("tokens", [1100, 300, 70, 40])
@pytest.mark.parametrize("n,m,g", [(2, 4, 1), (3, 6, 3)])
def test_tiny_rows(n, m, g, tokens):
    """Rows (and parts of rows, which the split pass looks at one by one) below the magnitudes that three pieces hold."""
    x, dy = seeded_normal((tokens, K), 2), seeded_normal((tokens, M), 3)
    for t in (x, dy):
        t[0::5] *= 2.0 ** -90         # a whole row
        t[1::5] *= 2.0 ** -130        # denormals
        t[2::5, :300] *= 2.0 ** -100  # some parts of a row, its others settle that it is not tiny
        t[3::5, :500] = 0             # parts of zeros and one of tiny values
        t[3::5, 400] = 2.0 ** -95
        t[3::10, 500:] = 0
        t[14] = 0
    for got, a, b in _products(n, m, g, seeded_normal((M, K), 1), x, dy):
        _close(got, a, b)
        assert bool((got[14] == 0).all())


def test_tiny_rows_longer_than_the_registers():
    """Token-major rows of which the split pass reads a part again."""
    from sten_b200 import _native as nat, ops
    rows, cols = 256, 9000
    w = seeded_normal((rows, cols), 1).to(cuda())
    val, idx = ops.sparsify(w.unsqueeze(0), 2, 4, 4)
    dense = ops.densify(val, idx, 1, rows, cols, 2, 4, 4)[0].double()
    x = seeded_normal((70, cols), 2)
    x[1] *= 2.0 ** -120
    x[2, :8990] *= 2.0 ** -120
    x[3, :8990] = 0
    x[4] = 0
    x = x.to(cuda())
    wide = torch.zeros(70, cols + 1, device=cuda())
    wide[:, 1:] = x
    for a in (x, wide[:, 1:]):  # the second: rows that take no 16-byte loads
        _close(ops.spmm(val, idx, rows, cols, 2, 4, 4, a, algo=nat.NMG_ALGO_TENSOR), a.double(), dense)


@pytest.mark.parametrize("m_rows,k_cols,tokens", [(512, 1000, 1025), (517, 1032, 1030), (203, 5003, 1040), (512, 1000, 70), (517, 1032, 513), (203, 5003, 200)])
@pytest.mark.parametrize("n,m,g", [(1, 4, 16), (2, 4, 1), (2, 8, 4), (3, 6, 3)])
def test_rows_of_different_magnitude(n, m, g, m_rows, k_cols, tokens):
    """Rows of both operands over many binades, some columns apart from the others, rows that take no 16-byte loads: the plain bound holds."""
    from sten_b200 import _native as nat, ops
    gen = lambda seed: torch.Generator().manual_seed(seed)  # noqa: E731
    w = seeded_normal((m_rows, k_cols), 1) * k_cols ** -0.5 * torch.exp2(torch.randint(-40, 40, (m_rows, 1), generator=gen(7)).float())
    w[:, 1::7] *= 2.0 ** -9
    w = w.to(cuda())
    val, idx = ops.sparsify(w.unsqueeze(0), n, m, g)
    dense = ops.densify(val, idx, 1, m_rows, k_cols, n, m, g)[0].double()
    x, dy = seeded_normal((tokens, k_cols + 3), 2), seeded_normal((tokens, m_rows + 1), 3)
    x = x * torch.exp2(torch.randint(-60, 60, (tokens, 1), generator=gen(8)).float())
    x[5] = 0
    dy[:, 2] *= 2.0 ** 14
    x, dy = x.to(cuda())[:, 1:k_cols + 1], dy.to(cuda())[:, :m_rows]
    copy = ops.pack(val, idx, m_rows, k_cols, n, m, g) if (n, m) != (3, 6) else None
    _close(ops.spmm(val, idx, m_rows, k_cols, n, m, g, x, packed=copy, algo=nat.NMG_ALGO_TENSOR), x.double(), dense)
    y = ops.spmm(val, idx, m_rows, k_cols, n, m, g, x.t().contiguous(), layout=nat.NMG_ACT_K_MAJOR, packed=copy, algo=nat.NMG_ALGO_TENSOR)
    _close(y.t(), x.double(), dense)
    _close(ops.spmm_t(val, idx, m_rows, k_cols, n, m, g, dy, packed=copy, algo=nat.NMG_ALGO_TENSOR), dy.double(), dense.t())
    assert ops.read_status() == 0


@pytest.mark.parametrize("features,tokens,fused", [(4736, 512, True), (4737, 512, True), (3712, 513, True), (3713, 513, False), (3712, 640, True), (3200, 641, False),
                                                   (3072, 768, True), (3073, 768, False), (2304, 1024, True), (2305, 1024, False), (64, 1024, True), (64, 1025, False)])
@pytest.mark.parametrize("transposed", [False, True])
def test_both_sides_of_the_line(transposed, features, tokens, fused):
    """With a kept copy: the fused kernel while its tiles of 128 x 128 fit the chip at once, two passes from there on; with aligned rows, rows that
    take no 16-byte loads and K-major ones."""
    from sten_b200 import _native as nat, ops
    n, m, g, red = 2, 4, 4, 200
    rows, cols = (red, features) if transposed else (features, red)
    val, idx = ops.sparsify(seeded_normal((rows, cols), 1).to(cuda()).unsqueeze(0), n, m, g)
    dense = ops.densify(val, idx, 1, rows, cols, n, m, g)[0].double()
    copy = ops.pack(val, idx, rows, cols, n, m, g)
    assert ops.uses_packed(rows, cols, tokens, n, m, g, torch.float32, transposed=transposed) == fused
    wide = seeded_normal((tokens, red + 1), 2).to(cuda())
    for a in (wide[:, :red].contiguous(), wide[:, 1:]):
        if transposed:
            _close(ops.spmm_t(val, idx, rows, cols, n, m, g, a, packed=copy), a.double(), dense.t())
            continue
        _close(ops.spmm(val, idx, rows, cols, n, m, g, a, packed=copy), a.double(), dense)
        _close(ops.spmm(val, idx, rows, cols, n, m, g, a.t().contiguous(), layout=nat.NMG_ACT_K_MAJOR, packed=copy).t(), a.double(), dense)
    assert ops.read_status() == 0
