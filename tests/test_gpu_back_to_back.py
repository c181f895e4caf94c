"""Calls queued behind one another without a host synchronisation: inputs written right before a call, results of one call as inputs of the
next, memory of one call reused by the next, on one stream and on two."""
import pytest
import torch

from gpu_util import cuda, seeded_normal

pytestmark = pytest.mark.gpu


def _weight(dtype, n, m, g, M, K, seed):
    from sten_b200 import ops
    w = (seeded_normal((M, K), seed) * K ** -0.5).to(dtype).to(cuda())
    return ops.sparsify(w.unsqueeze(0), n, m, g)


class _Call:
    """One entry point, its weight and its input buffer; run() queues the writes of weight and input, then the call."""

    def __init__(self, kind, dtype, fmt, M, K, tokens, packed):
        from sten_b200 import _native as nat, ops
        self.ops, self.nat, self.kind, self.shape, self.fmt = ops, nat, kind, (M, K), fmt
        self.weights = [_weight(dtype, *fmt, M, K, s) for s in (1, 2)]
        self.val, self.idx = (t.clone() for t in self.weights[0])
        self.packed = packed
        size = {"tm": (tokens, K), "ragged": (tokens, K + 1), "km": (K, tokens), "t": (tokens, M), "densify": (1, 1)}[kind]
        self.inputs = [seeded_normal(size, s).to(dtype).to(cuda()) for s in (3, 4)]
        self.x = torch.empty_like(self.inputs[0])

    def run(self, i, load):
        ops, (M, K), (n, m, g) = self.ops, self.shape, self.fmt
        load()  # the writes below wait for it, and run just ahead of the call
        self.val.copy_(self.weights[i % 2][0])
        self.idx.copy_(self.weights[i % 2][1])
        self.x.copy_(self.inputs[i // 2 % 2])
        if self.kind == "densify":
            return ops.densify(self.val, self.idx, 1, M, K, n, m, g)
        packed = ops.pack(self.val, self.idx, M, K, n, m, g) if self.packed else None
        x = self.x[:, 1:] if self.kind == "ragged" else self.x
        if self.kind == "t":
            return ops.spmm_t(self.val, self.idx, M, K, n, m, g, x, packed=packed)
        layout = self.nat.NMG_ACT_K_MAJOR if self.kind == "km" else self.nat.NMG_ACT_TOKEN_MAJOR
        return ops.spmm(self.val, self.idx, M, K, n, m, g, x, layout=layout, packed=packed)


def _calls():
    f16, bf16, f32 = torch.float16, torch.bfloat16, torch.float32
    yield _Call("tm", f16, (2, 4, 16), 512, 768, 40, True)        # fused
    yield _Call("ragged", bf16, (1, 8, 8), 512, 760, 300, True)   # rows laid out first
    yield _Call("km", f16, (2, 4, 16), 512, 768, 200, True)       # transposed first
    yield _Call("tm", bf16, (2, 4, 16), 1024, 1024, 2000, False)  # expansion and matmul
    yield _Call("t", f16, (2, 4, 16), 1024, 1024, 4096, False)    # structured-sparse form
    yield _Call("t", bf16, (3, 6, 4), 504, 600, 700, False)
    yield _Call("tm", f32, (2, 4, 16), 512, 768, 300, True)       # split and fused
    yield _Call("km", f32, (2, 4, 16), 512, 768, 40, True)
    yield _Call("tm", f32, (1, 4, 16), 512, 5000, 1100, False)    # split, expansion and matmul
    yield _Call("km", f32, (1, 4, 16), 512, 768, 1100, False)
    yield _Call("t", f32, (2, 4, 16), 512, 768, 1100, False)
    yield _Call("densify", bf16, (2, 8, 16), 2048, 2048, 1, False)


def _load():
    """Work that keeps the chip busy for some tens of microseconds."""
    a = torch.ones(4096, 4096, device=cuda())

    def load():
        a.mul_(1.0)
    return load


def test_inputs_written_right_before_the_call():
    from sten_b200 import ops
    calls, load = list(_calls()), _load()
    want = {}
    for c, call in enumerate(calls):
        for i in range(4):
            want[c, i] = call.run(i, load)
            torch.cuda.synchronize()
    for rounds in range(3):
        got = {(c, i): call.run(i, load) for i in range(4) for c, call in enumerate(calls)}
        torch.cuda.synchronize()
        for key, y in got.items():
            assert torch.equal(y, want[key]), (key, rounds)
    assert ops.read_status() == 0


def test_two_streams():
    from sten_b200 import ops
    sides = [list(_calls()) for _ in range(2)]
    loads = [_load() for _ in range(2)]
    want = {}
    for c, call in enumerate(sides[0]):
        for i in range(4):
            want[c, i] = call.run(i, loads[0])
            torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    got = []
    for i in range(4):
        for c in range(len(sides[0])):
            for s in range(2):
                with torch.cuda.stream(streams[s]):
                    j = (i + s) % 4
                    got.append(((c, j), sides[s][c].run(j, loads[s])))
    torch.cuda.synchronize()
    for key, y in got:
        assert torch.equal(y, want[key]), key
    assert ops.read_status() == 0


@pytest.mark.parametrize("dtype,tokens", [(torch.float16, 24), (torch.bfloat16, 2500), (torch.float32, 200), (torch.float32, 1500)])
def test_results_feed_the_next_call(dtype, tokens):
    """A chain of products, each reading what the one before wrote: the same with a synchronisation between all of them."""
    from sten_b200 import ops
    n, m, g, size = 2, 4, 16, 768
    weights = [_weight(dtype, n, m, g, size, size, s) for s in range(4)]
    packed = [ops.pack(v, i, size, size, n, m, g) for v, i in weights]
    x0 = seeded_normal((tokens, size), 9).to(dtype).to(cuda())

    def chain(sync):
        x = x0
        for k in range(12):
            v, i = weights[k % 4]
            step = ops.spmm if k % 3 else ops.spmm_t
            x = step(v, i, size, size, n, m, g, x, packed=packed[k % 4])
            x = x / x.abs().amax().clamp(min=1e-3) if k % 4 == 3 else x  # a kernel of another library in between
            if sync:
                torch.cuda.synchronize()
        return x

    want = chain(True)
    for _ in range(5):
        assert torch.equal(chain(False), want)
    assert ops.read_status() == 0
