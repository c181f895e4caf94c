"""Operands that a kernel would read past their end are refused on the host, before any launch."""
import pytest
import torch

from gpu_util import cuda

pytestmark = pytest.mark.gpu
M, K, TOKENS = 96, 200, 32


def _weight(dtype=torch.bfloat16):
    from sten_b200.grouped_nm_tensor import GroupedNMTensor
    return GroupedNMTensor.from_dense(torch.randn(M, K, device=cuda()).to(dtype), 2, 4, 0, 8, 1)


@pytest.mark.parametrize("shape", [(M - 1,), (M + 1,), (1,), (M, 1), (2, M), ()])
def test_a_bias_of_another_size_is_refused(shape):
    import sten_b200 as sten
    from sten_b200 import ops
    w, x, bias = _weight(), torch.randn(TOKENS, K, device=cuda()).bfloat16(), torch.zeros(shape, device=cuda(), dtype=torch.bfloat16)
    wrapped, good = sten.SparseTensorWrapper.wrapped_from_dense(w, w.to_dense()), torch.zeros(M, device=cuda(), dtype=torch.bfloat16)
    with torch.no_grad():
        for _ in range(3):  # the general route, then the repeated one
            torch.nn.functional.linear(x, wrapped, good)
            with pytest.raises(ValueError, match="bias"):
                torch.nn.functional.linear(x, wrapped, bias)
        with pytest.raises(ValueError, match="bias"):
            sten.sparse_linear_fused(x, w, bias, activation="gelu")
    for kernel_layout in (0, 1, 2):
        act = x.t().contiguous() if kernel_layout == 1 else x
        with pytest.raises(ValueError, match="bias"):
            ops.spmm(w.val, w.idx, M, K, 2, 4, 8, act, bias=bias, layout=kernel_layout)
    with pytest.raises(ValueError, match="bias"):
        ops.spmm_expanded(w.expanded(), M, K, x, bias=bias)
    out = torch.zeros(M, TOKENS, device=cuda(), dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="bias"):
        ops.spmm_replicated(w.val, w.idx, M, K, 2, 4, 8, x, [out.data_ptr()], TOKENS, bias=bias)


def test_a_bias_with_a_leading_dimension_is_served():
    w, x, bias = _weight(), torch.randn(TOKENS, K, device=cuda()).bfloat16(), torch.randn(1, M, device=cuda()).bfloat16()
    assert torch.equal(w.native().linear(w, x, bias, 0, None), w.native().linear(w, x, bias[0], 0, None))
