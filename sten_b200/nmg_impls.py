"""The grouped n:m plugin: sparsifier and operator registrations (reference: src/sten/grouped_nm/sten_impls.py).

Registered here, all backed by ``libnmg_b200.so``:

* ``GroupedNMSparsifier`` : ``torch.Tensor -> GroupedNMTensor``                    (reference sten_impls.py:13-37)
* ``F.linear``  forward for ``(Tensor, GroupedNMTensor, Tensor)`` -- the reference's only operator (:143-174) -- and for
  ``(Tensor, GroupedNMTensor)``: a bias-free linear has two tensor inputs and would otherwise miss the registration
  and silently densify;
* ``torch.mm`` / ``torch.matmul`` forward for ``(GroupedNMTensor, Tensor)``;
* the matching backward entries (``dX = dY W`` through the transposed kernel); the reference has none and installs a
  failing stub (sten.py:1690-1693).

Unlike the reference (sten_impls.py:53, which derives the transpose flag from contiguity and ends up reading a
contiguous ``[tokens, K]`` activation as ``[K, tokens]``), the activation layout is stated explicitly:
``F.linear`` is ``y = x W^T + b`` on ``x[tokens, K]``.
"""
import torch

from . import _native as nat
from . import dispatch as sten
from . import ops
from .grouped_nm_tensor import GroupedNMTensor


class GroupedNMSparsifier:
    def __init__(self, n, m, g):
        self.n = n
        self.m = m
        self.g = g


class WeightLayoutSparsifier:
    """Inline gradient sparsifier of a grouped n:m weight: the gradient keeps the weight's own layout (same ``idx``),
    only the kept positions are stored.  Declared per weight with::

        sb.set_weight_grad(name, inline_sparsifier=WeightLayoutSparsifier(), tmp_format=GroupedNMTensor,
                           external_sparsifier=KeepAll(), out_format=GroupedNMTensor)

    The reference leaves this open (``clone_layout`` is disabled, grouped_nm_tensor.py:904-951; its linear backward
    returns dense gradients only).  With it the gradient, the optimizer's view of it and the bytes a data-parallel
    all-reduce moves are n/m of the dense size, and the layout is identical on every rank."""


@sten.register_sparsifier_implementation(sparsifier=GroupedNMSparsifier, inp=torch.Tensor, out=GroupedNMTensor)
def dense_to_grouped_nm(sparsifier, tensor, grad_fmt=None):
    gnm = GroupedNMTensor.from_dense(tensor, sparsifier.n, sparsifier.m, sparse_dim=tensor.ndim - 2,
                                     group_size=sparsifier.g, group_dim=tensor.ndim - 1)
    return sten.SparseTensorWrapper.wrapped_from_dense(gnm, tensor, grad_fmt)


@sten.register_sparsifier_implementation(sparsifier=sten.SameFormatSparsifier, inp=torch.Tensor, out=GroupedNMTensor)
def dense_to_same_grouped_nm(sparsifier, tensor, grad_fmt=None):
    """Re-sparsify a dense result with the (n, m, g, dims) of the reference tensor (fresh magnitude selection)."""
    ref = sparsifier.ref_sp_ten
    s = ref.wrapped_tensor.nm_strides
    gnm = GroupedNMTensor.from_dense(tensor, s["n"], s["m"], sparse_dim=s["sparse_dim"], group_size=s["group_size"],
                                     group_dim=s["group_dim"])
    return sten.SparseTensorWrapper.wrapped_from_dense(gnm, tensor, grad_fmt if grad_fmt is not None else ref.grad_fmt)


def _wants_expanded(gnm, x2d, tokens):
    """The opt-in of ``set_spmm_opt(kernel="sm100-expanded")`` applies: 16-bit weight, token-major activation whose rows TMA
    can read, and a batch from which on the matmul of the kept weight is no slower than the compressed-weight kernel."""
    return (gnm.nm_strides.get("kernel") == "sm100-expanded" and tokens >= ops.SP24_MIN_TOKENS
            and gnm.val.dtype != torch.float32 and x2d.stride(-1) == 1 and x2d.data_ptr() % 16 == 0 and x2d.stride(0) % 8 == 0
            and gnm.expanded() is not None)


def _native_weight(weight):
    """(GroupedNMTensor, its host-side handle) of a weight the matmul kernels can serve."""
    gnm = weight.wrapped_tensor
    h = gnm.native()
    if h is None:
        raise sten.DispatchError("grouped n:m matmul needs a 2-D weight with n:m blocks along dim 0 and groups along dim 1")
    return gnm, h


def sparse_dense_mul_dispatch(weight, dense2d, bias, layout):
    """One C-ABI call; replaces the compile-or-load + ctypes call of the reference (sten_impls.py:44-140)."""
    gnm, h = _native_weight(weight)
    if layout == nat.NMG_ACT_K_MAJOR and bias is None:
        return h.mm(gnm, dense2d)
    if layout != nat.NMG_ACT_TOKEN_MAJOR:
        s = gnm.nm_strides
        M, K = s["dense_shape"]
        return ops.spmm(gnm.val, gnm.idx, M, K, s["n"], s["m"], s["group_size"], dense2d, bias=bias, layout=layout)
    if gnm.nm_strides.get("kernel") == "sm100-expanded" and _wants_expanded(gnm, dense2d, dense2d.shape[0]):
        M, K = gnm.nm_strides["dense_shape"]
        return ops.spmm_expanded(gnm.expanded(), M, K, dense2d, bias=bias)
    return h.linear(gnm, dense2d, bias, nat.NMG_EPI_NONE, None)


def _linear_fwd(ctx, inputs, output_sparsifiers):
    if len(inputs) == 3:
        x, weight, bias = inputs
        ctx.save_for_backward(x, weight, bias)
    else:
        (x, weight), bias = inputs, None
        ctx.save_for_backward(x, weight)
    gnm, h = _native_weight(weight)
    if gnm.nm_strides.get("kernel") == "sm100-expanded":
        y = sparse_dense_mul_dispatch(weight, x.reshape(-1, x.shape[-1]), bias, nat.NMG_ACT_TOKEN_MAJOR)
        return y.reshape(*x.shape[:-1], y.shape[-1])
    return h.linear(gnm, x, bias, nat.NMG_EPI_NONE, None)


_linear_fwd.native_call = "linear"  # a repeated call without gradients is one call of the handle (see dispatch.use_native_repeat)
_LIN_OUT = [(sten.KeepAll, torch.Tensor)]
sparse_torch_nn_functional_linear = sten.register_fwd_op_impl(
    operator=torch.nn.functional.linear, inp=(torch.Tensor, GroupedNMTensor, torch.Tensor), out=_LIN_OUT)(_linear_fwd)
sten.register_fwd_op_impl(operator=torch.nn.functional.linear, inp=(torch.Tensor, GroupedNMTensor), out=_LIN_OUT)(_linear_fwd)


def _linear_grads(ctx, grad_outputs, in_layout):
    saved = ctx.saved_tensors
    needs = ctx.needs_input_grad
    gnm, h = _native_weight(saved[1])
    mask = (1 if needs[1] else 0) | (2 if needs[2] else 0) | (4 if len(saved) == 3 and needs[3] else 0)
    return len(saved), gnm, h.linear_grads(gnm, saved[0], grad_outputs[0], ops.SP24_MIN_TOKENS, mask, in_layout)


def _linear_bwd(ctx, grad_outputs, input_sparsifiers):
    count, _, grads = _linear_grads(ctx, grad_outputs, 0)
    return grads[:count]


def _linear_bwd_weight_layout(ctx, grad_outputs, input_sparsifiers):
    """Same products as ``_linear_bwd``; dW leaves as a GroupedNMTensor in the weight's layout.  dY^T X runs on the tensor
    cores at the dense rate into a transient buffer (a sampled product on the FP32 pipes would be an order of magnitude
    slower on this hardware) and one gather pass keeps the layout's positions."""
    count, gnm, (dx, dw, db) = _linear_grads(ctx, grad_outputs, 1)
    if dw is not None:
        dw = sten.SparseTensorWrapper([GroupedNMTensor(dw, gnm.idx, gnm.nm_strides)], False, sten._DEFAULT_GRAD_FMT(), shared_dummy=True)
        dw.made_as_gradient = True
    return (dx, dw, db)[:count]


_DENSE_GRAD = (sten.KeepAll, torch.Tensor)
_LAYOUT_GRAD = (WeightLayoutSparsifier, GroupedNMTensor)
for _inp in ((torch.Tensor, GroupedNMTensor, torch.Tensor), (torch.Tensor, GroupedNMTensor)):
    sten.register_bwd_op_impl(operator=torch.nn.functional.linear, grad_out=(torch.Tensor,),
                              grad_inp=tuple(_DENSE_GRAD for _ in _inp), inp=_inp)(_linear_bwd)
    sten.register_bwd_op_impl(operator=torch.nn.functional.linear, grad_out=(torch.Tensor,),
                              grad_inp=tuple(_LAYOUT_GRAD if f is GroupedNMTensor else _DENSE_GRAD for f in _inp),
                              inp=_inp)(_linear_bwd_weight_layout)


def _mm_fwd(ctx, inputs, output_sparsifiers):
    weight, b = inputs
    ctx.save_for_backward(weight, b)
    if b.dim() != 2:
        raise sten.DispatchError("grouped n:m matmul expects a 2-D right operand")
    gnm, h = _native_weight(weight)
    return h.mm(gnm, b)


_mm_fwd.native_call = "mm"


def _mm_bwd(ctx, grad_outputs, input_sparsifiers):
    weight, b = ctx.saved_tensors
    [dc] = grad_outputs  # [M, N]
    needs = tuple(ctx.needs_input_grad[1:]) + (False,) * 2
    gnm, h = _native_weight(weight)
    dw = db = None
    if needs[0]:
        dw = dc.mm(b.t())
    if needs[1]:
        # dB = W^T dC : the transposed kernel computes (dC^T W)[N, K]; hand back its transpose
        db = h.linear_t(gnm, dc.t().contiguous(), ops.SP24_MIN_TOKENS).t()
    return dw, db


for _op in (torch.mm, torch.matmul):
    sten.register_fwd_op_impl(operator=_op, inp=(GroupedNMTensor, torch.Tensor), out=_LIN_OUT)(_mm_fwd)
    sten.register_bwd_op_impl(operator=_op, grad_out=(torch.Tensor,), grad_inp=(_DENSE_GRAD, _DENSE_GRAD),
                              inp=(GroupedNMTensor, torch.Tensor))(_mm_bwd)
