"""val and idx that do not hold a weight of the stated geometry are refused on the host."""
import pytest
import torch

from sten_b200 import _native as nat


@pytest.mark.parametrize("n,m,g,M,K", [(2, 4, 2, 8, 24), (2, 4, 2, 5, 13), (1, 8, 4, 16, 64), (3, 6, 1, 7, 41)])
def test_smaller_tensors_are_refused(n, m, g, M, K):
    cc = nat.lib().nmg_num_patterns(n, m) * g
    slots = -(-M // m) * -(-K // cc) * cc
    check = lambda v, i: nat.host().check_weight(torch.zeros(v), torch.zeros(i, dtype=torch.int16), M, K, n, m, g)  # noqa: E731
    check(slots * n, slots)
    check(slots * n + 3, slots + 1)  # more than that is never read
    with pytest.raises(ValueError, match="smaller"):
        check(slots * n - 1, slots)
    with pytest.raises(ValueError, match="smaller"):
        check(slots * n, slots - 1)
    with pytest.raises(TypeError, match="int16"):
        nat.host().check_weight(torch.zeros(slots * n), torch.zeros(slots), M, K, n, m, g)


@pytest.mark.gpu
def test_every_entry_point_checks():
    from sten_b200 import ops
    from sten_b200.grouped_nm_tensor import GroupedNMTensor
    dev, M, K = torch.device("cuda", 0), 96, 200
    w = GroupedNMTensor.from_dense(torch.randn(M, K, device=dev).bfloat16(), 2, 4, 0, 8, 1)
    x, dy, val, idx = torch.randn(16, K, device=dev).bfloat16(), torch.randn(16, M, device=dev).bfloat16(), w.val, w.idx
    a = (M, K, 2, 4, 8)
    for v, i in ((val[1:], idx), (val, idx[1:])):
        w.val, w.idx = v, i
        for call in (lambda: w.native().linear(w, x, None, 0, None), lambda: w.native().mm(w, x.t()), lambda: w.native().linear_t(w, dy, ops.SP24_MIN_TOKENS),
                     w.to_dense, w.packed, w.packed_sp24, w.expanded, lambda: ops.spmm(v, i, *a, x), lambda: ops.spmm_t(v, i, *a, dy),
                     lambda: ops.spmm_replicated(v, i, *a, x, [x.data_ptr()], 16)):
            with pytest.raises(ValueError, match="smaller"):
                call()
