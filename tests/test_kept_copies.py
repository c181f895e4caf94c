"""Copies derived from a weight are made again whenever the weight is no longer what they were made from."""
import numpy as np
import pytest
import torch

from sten_b200 import ops
from sten_b200.grouped_nm_tensor import GroupedNMTensor


def _weight(val, idx):
    return GroupedNMTensor(val, idx, {"dense_shape": [4, 8], "sparse_dim": 0, "group_dim": 1, "n": 2, "m": 4, "group_size": 1})


def _replaced_at_the_same_address(gnm, buf):
    gnm.val = None
    gnm.val = torch.from_numpy(buf)


def _data_set_to_the_same_address(gnm, buf):
    gnm.val.data = torch.zeros(2)
    gnm.val.data = torch.from_numpy(buf)


def _detached_with_its_own_version(gnm, buf):
    gnm.val = gnm.val.data  # same storage, address and version number, another counter


@pytest.mark.parametrize("change", [_replaced_at_the_same_address, _data_set_to_the_same_address, _detached_with_its_own_version,
                                    lambda gnm, buf: gnm.val.mul_(2), lambda gnm, buf: gnm.idx.add_(0)])
def test_a_changed_weight_is_packed_again(change, monkeypatch):
    made = []
    monkeypatch.setattr(ops, "pack", lambda val, *a: made.append(val) or torch.zeros(1))
    buf = np.arange(12, dtype=np.float32)
    gnm = _weight(torch.from_numpy(buf), torch.zeros(6, dtype=torch.int16))
    first = gnm.packed()
    assert gnm.packed().data_ptr() == first.data_ptr() and len(made) == 1
    made.clear()
    change(gnm, buf)
    gnm.packed()
    assert len(made) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tokens", [16, 300, 1500])
def test_products_after_two_replacements_of_the_values(tokens, dtype):
    """The allocator hands the third tensor the first one's address."""
    dev, M, K = torch.device("cuda", 0), 256, 512
    rel = lambda a, b: float((a.double() - b).norm() / b.norm())  # noqa: E731
    w = GroupedNMTensor.from_dense(torch.randn(M, K, device=dev).to(dtype), 2, 4, 0, 16, 1)
    x, dy = torch.randn(tokens, K, device=dev).to(dtype), torch.randn(tokens, M, device=dev).to(dtype)
    for _ in range(4):
        w.native().linear(w, x, None, 0, None)
        w.native().mm(w, x[:8].t())
        w.native().linear_t(w, dy, ops.SP24_MIN_TOKENS)
        w.expanded()
        w.val = w.val * 2
        w.val = w.val * 0.25
        dense = w.to_dense().double()
        assert rel(w.native().linear(w, x, None, 0, None), x.double() @ dense.t()) < 1e-2
        assert rel(w.native().mm(w, x[:8].t()), dense @ x[:8].double().t()) < 1e-2
        assert rel(w.native().linear_t(w, dy, ops.SP24_MIN_TOKENS), dy.double() @ dense) < 1e-2
        if dtype != torch.float32:
            assert rel(ops.spmm_expanded(w.expanded(), M, K, x), x.double() @ dense.t()) < 1e-2
