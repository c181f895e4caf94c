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


def test_nothing_is_kept_of_inference_tensors(monkeypatch):
    """They have no version counter: a write between two calls would go unseen."""
    made = []
    monkeypatch.setattr(ops, "pack", lambda val, *a: made.append(val) or torch.zeros(1))
    with torch.inference_mode():
        gnm = _weight(torch.zeros(12), torch.zeros(6, dtype=torch.int16))
    for _ in range(2):
        gnm.packed()
    assert len(made) == 2


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tokens", [16, 300, 1400])
def test_products_of_a_weight_made_under_inference_mode(tokens, dtype):
    dev, M, K = torch.device("cuda", 0), 256, 512
    with torch.inference_mode():
        w = GroupedNMTensor.from_dense(torch.randn(M, K, device=dev).to(dtype), 2, 4, 0, 16, 1)
        x = torch.randn(tokens, K, device=dev).to(dtype)
        for _ in range(3):
            w.val.mul_(1.5)
            want = x.double() @ w.to_dense().double().t()
            assert _rel(w.native().linear(w, x, None, 0, None), want) < 1e-2
            assert _rel(w.native().mm(w, x[:8].t()), want[:8].t()) < 1e-2
            assert _rel(w.native().mm(w, x.t()), want.t()) < 1e-2


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm())


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


def _captured(fn, device=torch.device("cuda", 0)):
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        out = fn()
    return graph, out


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tokens,op", [(torch.float32, 300, "linear"), (torch.float32, 600, "linear"), (torch.float32, 300, "mm"), (torch.float32, 600, "linear_t"),
                                             (torch.bfloat16, 1400, "linear"), (torch.bfloat16, 8, "mm"), (torch.float32, 8, "mm")])
def test_replays_see_what_was_written_into_the_weight(dtype, tokens, op):
    dev, M, K = torch.device("cuda", 0), 256, 512
    w = GroupedNMTensor.from_dense(torch.randn(M, K, device=dev).to(dtype), 2, 4, 0, 16, 1)
    h = w.native()
    x = torch.randn(tokens, M if op == "linear_t" else K, device=dev).to(dtype)
    b = x.t().contiguous()
    fn = {"linear": lambda: h.linear(w, x, None, 0, None), "mm": lambda: h.mm(w, b), "linear_t": lambda: h.linear_t(w, x, ops.SP24_MIN_TOKENS)}[op]
    want = lambda: {"linear": lambda d: x.double() @ d.t(), "mm": lambda d: d @ b.double(), "linear_t": lambda d: x.double() @ d}[op](w.to_dense().double())  # noqa: E731
    for _ in range(3):
        fn()
    graph, out = _captured(fn)
    w.val.mul_(2)
    graph.replay()
    assert _rel(out, want()) < 1e-2


@pytest.mark.gpu
@pytest.mark.parametrize("op", ["linear", "linear_t"])
def test_a_copy_made_inside_a_graph_is_not_kept(op):
    dev, M, K = torch.device("cuda", 0), 256, 512
    w, warm = (GroupedNMTensor.from_dense(torch.randn(M, K, device=dev).bfloat16(), 2, 4, 0, 16, 1) for _ in range(2))
    for tokens in (16, 1300):
        x = torch.randn(tokens, K if op == "linear" else M, device=dev).bfloat16()
        fn = lambda t: t.native().linear(t, x, None, 0, None) if op == "linear" else t.native().linear_t(t, x, ops.SP24_MIN_TOKENS)  # noqa: E731
        fn(warm)
        graph, out = _captured(lambda: fn(w))
        assert not {"_packed_cache", "_sp24_cache"} & set(w.__dict__)
        d = w.to_dense().double()
        want = x.double() @ (d.t() if op == "linear" else d)
        graph.replay()
        assert _rel(out, want) < 1e-2
    del graph
    assert _rel(fn(w), want) < 1e-2


@pytest.mark.gpu
def test_a_graph_keeps_the_copy_that_it_reads():
    """A captured call of few tokens reads the copy of the contents it was captured with; a later change of the weight does not
    give that memory to somebody else."""
    dev, M, K = torch.device("cuda", 0), 256, 512
    w = GroupedNMTensor.from_dense(torch.randn(M, K, device=dev).bfloat16(), 2, 4, 0, 16, 1)
    x = torch.randn(16, K, device=dev).bfloat16()
    fn = lambda: w.native().linear(w, x, None, 0, None)  # noqa: E731
    fn()
    graph, out = _captured(fn)
    graph.replay()
    before = out.clone()
    keep = (w.val, w.idx)  # what the graph was captured with
    nbytes = w.packed().numel()
    for _ in range(2):
        w.val = w.val * 3
        fn()
        filler = [torch.full((nbytes,), 0x55, dtype=torch.uint8, device=dev) for _ in range(4)]
    graph.replay()
    assert torch.equal(out, before)
    del filler, keep


_CALLS = {"linear": lambda w, x: w.native().linear(w, x, None, 0, None), "linear_t": lambda w, x: w.native().linear_t(w, x, ops.SP24_MIN_TOKENS),
          "expanded": lambda w, x: ops.spmm_expanded(w.expanded(), x.shape[1], x.shape[1], x)}


@pytest.mark.gpu
@pytest.mark.parametrize("tokens", [16, 1300])
@pytest.mark.parametrize("op", sorted(_CALLS))
def test_another_stream_waits_for_the_copy(op, tokens):
    """The copy is made on one stream behind 100 ms of other work; a call on another stream uses it meanwhile."""
    dev, M = torch.device("cuda", 0), 512
    w = GroupedNMTensor.from_dense(torch.randn(M, M, device=dev).bfloat16(), 2, 4, 0, 16, 1)
    x = torch.randn(tokens, M, device=dev).bfloat16()
    dense = w.to_dense().double()
    want = x.double() @ (dense if op == "linear_t" else dense.t())
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(one):
        torch.cuda._sleep(200_000_000)
        for _ in range(2):
            _CALLS[op](w, x)
    with torch.cuda.stream(two):
        out = _CALLS[op](w, x)
    torch.cuda.synchronize()
    assert _rel(out, want) < 1e-2


@pytest.mark.gpu
@pytest.mark.parametrize("op", sorted(_CALLS))
def test_a_replaced_copy_stays_until_other_streams_have_read_it(op):
    dev, M, tokens = torch.device("cuda", 0), 512, 1300
    w = GroupedNMTensor.from_dense(torch.randn(M, M, device=dev).bfloat16(), 2, 4, 0, 16, 1)
    x = torch.randn(tokens, M, device=dev).bfloat16()
    dense = w.to_dense().double()
    want = x.double() @ (dense if op == "linear_t" else dense.t())
    for _ in range(3):
        _CALLS[op](w, x)
    nbytes = {n: k.get(w.val, w.idx).numel() for n, k in w.__dict__.items() if n.endswith("_cache")}
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    keep = (w.val, w.idx)
    with torch.cuda.stream(side):
        torch.cuda._sleep(200_000_000)
        out = _CALLS[op](w, x)
    w.val = w.val * 3
    for _ in range(3):
        _CALLS[op](w, x)
    filler = [torch.full((n,), 0x55, dtype=torch.uint8, device=dev) for n in nbytes.values() for _ in range(6)]
    torch.cuda.synchronize()
    assert _rel(out, want) < 1e-2
    del keep, filler
