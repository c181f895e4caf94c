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
