"""A backward pass that is recorded itself (create_graph)."""
import pytest
import torch

from gpu_util import cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(32, 128), (2, 16, 128)])
def test_the_bias_gradient_depends_on_the_output_gradient(shape):
    import sten_b200 as sten
    lin = torch.nn.Linear(128, 64).to(cuda())
    sb = sten.SparsityBuilder()
    sb.set_weight("weight", initial_sparsifier=sten.GroupedNMSparsifier(2, 4, 4), out_format=sten.GroupedNMTensor)
    lin = sb.get_sparse_model(lin)
    x = torch.randn(*shape, device=cuda())
    y = lin(x)
    dy = torch.randn_like(y).requires_grad_(True)
    (db,) = torch.autograd.grad(y, [lin.bias], dy, create_graph=True)
    scale = torch.randn(64, device=cuda())
    (back,) = torch.autograd.grad((db * scale).sum(), [dy])
    assert torch.equal(back, scale.expand_as(dy))
    (plain,) = torch.autograd.grad(lin(x), [lin.bias], dy.detach())
    assert not plain.requires_grad and float((plain - db).norm() / db.norm()) < 1e-6
