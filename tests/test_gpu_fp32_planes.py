"""fp32 operands as two fp16 planes with an exponent per row, in both tensor-core kernels: the rows' scales, lengths that the pass holds
in registers or shared memory and those it reads again, both orientations, values at the ends of the range."""
import pytest
import torch

from gpu_util import cuda, seeded_normal

pytestmark = pytest.mark.gpu

# An accumulator takes 8 k-blocks x 4 steps x 3 products before it is added up in fp32.  A step aligns its 16 products and the
# accumulator to the largest of them and cuts each off, at 2^-25 of the sum of magnitudes or below; two operands are off by up to 2^-22
# each and one product of 2^-22 is dropped.
BOUND = 96 * 17 * 2.0 ** -25 + 3 * 2.0 ** -22


def _weight(n, m, M, K, g, spread):
    from sten_b200 import ops
    w = seeded_normal((M, K), 1) * K ** -0.5
    if spread:  # rows of very different magnitude, a few columns much smaller
        w = w * torch.exp2(torch.randint(-40, 40, (M, 1), generator=torch.Generator().manual_seed(7)).float())
        w[:, 1::7] *= 2.0 ** -9
    w = w.to(cuda())
    val, idx = ops.sparsify(w.unsqueeze(0), n, m, g)
    return val, idx, ops.densify(val, idx, 1, M, K, n, m, g)[0].double()


def _packed(val, idx, M, K, n, m, g):
    """The copy that the fused kernel reads (fewer tokens), where the pattern has one."""
    from sten_b200 import ops
    return ops.pack(val, idx, M, K, n, m, g) if (n, m) in ((1, 4), (2, 4), (1, 8), (2, 8), (1, 16)) else None


def _close(got, a, b, spread=False):
    """got against the fp64 product a b^T, by the sum of magnitudes of every element.  spread: values may lie further below the largest
    of their row than two planes reach, and are then off by up to 2^-39 of that (half of the smallest fp16 step, 2^-25, against 2^14)."""
    err, bound = (got.double() - a @ b.t()).abs(), BOUND * (a.abs() @ b.abs().t()) + 2.0 ** -148
    if spread:
        top = lambda v: v.abs().amax(1, keepdim=True)  # noqa: E731
        bound += 2.0 ** -39 * (top(a) * b.abs().sum(1) + (a.abs() @ (b != 0).double().t()) * top(b).t())
    assert bool((err <= bound).all()), float((err / bound).max())


@pytest.mark.parametrize("K,tokens", [(256, 1100), (1000, 1025), (1032, 1030), (4096, 1100), (5003, 1040),  # two passes
                                      (192, 64), (256, 300), (1000, 70), (1032, 513), (4096, 1024), (5003, 200)])  # fused
@pytest.mark.parametrize("n,m,g", [(1, 4, 16), (2, 4, 1), (2, 8, 4), (1, 16, 3), (3, 6, 3), (1, 3, 5)])
@pytest.mark.parametrize("spread", [False, True])
def test_products(n, m, g, K, tokens, spread):
    from sten_b200 import _native as nat, ops
    M = 203 if K > 4000 else 517 if K != 1000 else 512  # output rows that take no 16-byte stores, and some that do
    val, idx, dense = _weight(n, m, M, K, g, spread)
    x, dy = seeded_normal((tokens, K + 3), 2), seeded_normal((tokens, M + 1), 3)
    if spread:
        x = x * torch.exp2(torch.randint(-60, 60, (tokens, 1), generator=torch.Generator().manual_seed(8)).float())
        x[5] = 0
        dy[:, 2] *= 2.0 ** 14
    x, dy = x.to(cuda())[:, 1:K + 1], dy.to(cuda())[:, :M]  # rows that take no 16-byte loads
    copy = _packed(val, idx, M, K, n, m, g)
    _close(ops.spmm(val, idx, M, K, n, m, g, x, packed=copy, algo=nat.NMG_ALGO_TENSOR), x.double(), dense, spread)
    _close(ops.spmm(val, idx, M, K, n, m, g, x.t().contiguous(), layout=nat.NMG_ACT_K_MAJOR, packed=copy, algo=nat.NMG_ALGO_TENSOR).t(), x.double(), dense, spread)
    _close(ops.spmm_t(val, idx, M, K, n, m, g, dy, packed=copy, algo=nat.NMG_ALGO_TENSOR), dy.double(), dense.t(), spread)
    assert ops.read_status() == 0


@pytest.mark.parametrize("M", [768, 1001])
@pytest.mark.parametrize("K,tokens", [(600, 1030), (1500, 2100), (4500, 1100), (600, 300), (300, 1000), (4500, 90)])
def test_wide_rows(K, tokens, M):
    """Rows with a few values far above all others: what they do not reach keeps the precision of the rest."""
    from sten_b200 import _native as nat, ops
    val, idx, dense = _weight(2, 8, M, K, 4, False)
    x, dy = seeded_normal((tokens, K), 2), seeded_normal((tokens, M), 3)
    for i, r in enumerate(range(3, tokens, 257)):
        for t, c in ((x, 7), (dy, 11)):
            t[r, c + i] = 2.0 ** (20 + 9 * i)
            t[r, 2 * c] = -2.0 ** (10 + 9 * i)
    x[9], dy[9] = 0, 0
    x[9, 5], dy[9, 5] = -2.0 ** 100, 2.0 ** 90
    x[9, 6], dy[9, 6] = 2.0 ** -20, 2.0 ** -30
    x, dy = x.to(cuda()), dy.to(cuda())
    copy = _packed(val, idx, M, K, 2, 8, 4)
    _close(ops.spmm(val, idx, M, K, 2, 8, 4, x, packed=copy, algo=nat.NMG_ALGO_TENSOR), x.double(), dense)
    _close(ops.spmm(val, idx, M, K, 2, 8, 4, x.t().contiguous(), layout=nat.NMG_ACT_K_MAJOR, packed=copy, algo=nat.NMG_ALGO_TENSOR).t(), x.double(), dense)
    _close(ops.spmm_t(val, idx, M, K, 2, 8, 4, dy, packed=copy, algo=nat.NMG_ALGO_TENSOR), dy.double(), dense.t())
    assert ops.read_status() == 0


@pytest.mark.parametrize("tokens", [1100, 600, 70])
@pytest.mark.parametrize("k_major", [False, True])
def test_ends_of_the_range(k_major, tokens):
    """Rows of zeros, of denormals, of the largest values; infinities and NaN stay in their own rows."""
    from sten_b200 import _native as nat, ops
    M, K = 256, 512
    val, idx, dense = _weight(2, 4, M, K, 4, False)
    x = seeded_normal((tokens, K), 2)
    x[3] = 0
    x[4] *= 2.0 ** -130
    x[5] *= 2.0 ** 120
    x[6] = torch.finfo(torch.float32).max * x[6].sign() * 2.0 ** -10
    x[7, 9] = -torch.finfo(torch.float32).max
    x[8, 10] = float("inf")
    x[9, 11] = float("nan")
    x = x.to(cuda())
    y = ops.spmm(val, idx, M, K, 2, 4, 4, x.t().contiguous() if k_major else x, layout=nat.NMG_ACT_K_MAJOR if k_major else nat.NMG_ACT_TOKEN_MAJOR,
                 packed=_packed(val, idx, M, K, 2, 4, 4), algo=nat.NMG_ALGO_TENSOR)
    y = y.t() if k_major else y
    assert bool((y[3] == 0).all())
    _close(y[5:8], x[5:8].double(), dense)
    _close(torch.cat([y[:4], y[10:]]), torch.cat([x[:4], x[10:]]).double(), dense)
    # results around 2^-130 are rounded to multiples of 2^-149
    err, ref = (y[4].double() - dense @ x[4].double()).abs(), dense.abs() @ x[4].double().abs()
    assert bool((err <= BOUND * ref + 2.0 ** -148).all())
    assert not bool(y[8].isfinite().any()) and bool(y[9].isnan().all())
    assert ops.read_status() == 0
