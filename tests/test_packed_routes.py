"""Which calls read a packed copy, which are served without one, and when the host makes one."""
import pytest
import torch

from sten_b200 import _native as nat
from sten_b200 import ops
from sten_b200.grouped_nm_tensor import GroupedNMTensor

AUTO, TM = nat.NMG_ALGO_AUTO, nat.NMG_ACT_TOKEN_MAJOR


@pytest.mark.parametrize("dtype,transposed,without,kept", [(nat.NMG_F32, 0, 513, 1025), (nat.NMG_F32, 1, 513, 1025), (nat.NMG_BF16, 0, 1280, 1536),
                                                           (nat.NMG_F16, 0, 1280, 1536), (nat.NMG_F16, 1, 1280, 1280)])
def test_thresholds(dtype, transposed, without, kept):
    L = nat.lib()
    uses = lambda tokens: L.nmg_spmm_uses_packed(512, 512, tokens, 2, 4, 16, dtype, TM, AUTO, transposed)  # noqa: E731
    assert uses(1) == uses(without - 1) == 1
    if kept > without:
        assert uses(without) == uses(kept - 1) == 2
    assert uses(kept) == 0
    if not transposed:  # a call without a copy: the workspace holds the copy below `without`, the expanded weight from there on
        ws = lambda tokens, have: L.nmg_spmm_workspace_bytes(512, 512, tokens, 2, 4, 16, dtype, TM, AUTO, have)  # noqa: E731
        assert ws(without - 1, 0) - ws(without - 1, 1) >= L.nmg_packed_bytes(512, 512, 2, 4, 16, dtype)
        assert ws(without, 0) - ws(without, 1) >= 512 * 512 * (6 if dtype == nat.NMG_F32 else 2)
        assert ws(kept, 0) == ws(kept, 1)


@pytest.mark.parametrize("dtype", [nat.NMG_F16, nat.NMG_BF16])
@pytest.mark.parametrize("tokens", [8, 16384])
def test_workspace_holds_the_activation_only_when_its_rows_are_unaligned(dtype, tokens):
    """Two passes over a 16384 x 16384 weight and 16384 tokens: the expanded weight, 512 MB, and not as much again."""
    L, size, again = nat.lib(), 16384, tokens * 16384 * 2
    for given in (0, 1):
        any_rows = L.nmg_spmm_workspace_bytes(size, size, tokens, 2, 8, 16, dtype, TM, AUTO, given)
        aligned = L.nmg_spmm_workspace_bytes(size, size, tokens, 2, 8, 16, dtype, TM, AUTO, given | 2)
        assert any_rows - aligned >= again
        if tokens == 16384:
            assert aligned <= size * size * 2 + 4096
        any_rows, aligned = (L.nmg_spmm_t_workspace_bytes(size, size, tokens, 2, 8, 16, dtype, AUTO, g) for g in (given, given | 2))
        assert any_rows - aligned >= again


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tol,first", [(torch.float32, 5e-6, 513), (torch.bfloat16, 1e-2, 1280)])
def test_a_copy_is_made_when_the_same_contents_are_used_again(dtype, tol, first):
    dev, M, K = torch.device("cuda", 0), 200, 328
    rel = lambda a, b: float((a.double() - b).norm() / b.norm())  # noqa: E731
    w = GroupedNMTensor.from_dense(torch.randn(M, K, device=dev).to(dtype), 2, 4, 0, 16, 1)
    h = w.native()
    for tokens in (first - 1, first, 1024 if first == 513 else 1535, 1025 if first == 513 else 1536):
        x = torch.randn(tokens, K, device=dev).to(dtype)
        for update in range(2):
            w.val.mul_(1.25)
            want = x.double() @ w.to_dense().double().t()
            if first <= tokens < (1025 if first == 513 else 1536):
                w.__dict__.pop("_packed_cache", None)
                assert rel(h.linear(w, x, None, 0, None), want) <= tol
                assert w.__dict__.get("_packed_cache") is None
                assert rel(h.mm(w, x.t()), want.t()) <= tol  # the second use
                assert w.__dict__.get("_packed_cache") is not None
            for _ in range(2):
                assert rel(h.linear(w, x, None, 0, None), want) <= tol
                assert rel(h.mm(w, x.t()), want.t()) <= tol
                assert rel(ops.spmm(w.val, w.idx, M, K, 2, 4, 16, x), want) <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("off,pitch", [(0, 0), (1, 0), (0, 3), (8, 8)])
@pytest.mark.parametrize("tokens", [40, 1300])
def test_scratch_of_a_call_fits_its_rows(off, pitch, tokens):
    """The host asks for what the call needs: aligned rows, an odd offset, an odd pitch; peak memory shows the difference."""
    dev, M, K = torch.device("cuda", 0), 512, 2048
    w = GroupedNMTensor.from_dense(torch.randn(M, K, device=dev).bfloat16(), 2, 4, 0, 16, 1)
    x = torch.randn(tokens, K + off + pitch, device=dev).bfloat16()[:, off:off + K]
    want = x.double() @ w.to_dense().double().t()
    for _ in range(3):
        y = w.native().linear(w, x, None, 0, None)
    assert float((y.double() - want).norm() / want.norm()) < 1e-2
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    w.native().linear(w, x, None, 0, None)
    scratch = torch.cuda.max_memory_allocated() - before - y.numel() * 2
    assert (scratch >= tokens * K * 2) == (off % 8 != 0 or pitch % 8 != 0)
