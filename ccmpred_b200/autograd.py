"""``torch.autograd.Function`` over the C ABI: the pseudo-likelihood as a
differentiable function of the single fields V and the couplings W.

The backward is the library's own gradient kernel, in the ``partial``
convention (true partial derivatives of f with respect to every entry, the
couplings untied and the self-edge blocks included), so that autograd and
finite differences agree.  The reference's optimizer uses the ``tied``
convention instead (src/evaluate_cpu.c:131-163); for a symmetric W the two are
related by  tied(b,k,a,j) = partial(b,k,a,j) + partial(a,j,b,k)  for k != j.

Tensor layouts:
  V  (L, 20)           V[j, a]        = single field of state a in column j
  W  (L, L, 21, 21)    W[k, j, b, a]  = coupling of state b in column k with
                                        state a in column j  (reference W(b,k,a,j))
"""
from __future__ import annotations

import ctypes

import torch

from . import Evaluator, nsingle_padded, nvar_padded
from ._lib import check, lib

Q = 21
QPAD = 32


def pack(V: torch.Tensor, W: torch.Tensor) -> torch.Tensor:
    """(V, W) -> x in the reference's padded layout (differentiable)."""
    L = V.shape[0]
    nsp = nsingle_padded(L)
    head = torch.cat([V.transpose(0, 1).reshape(-1),
                      V.new_zeros(nsp - (Q - 1) * L)])
    x2 = W.permute(2, 0, 3, 1)                                     # [b, k, a, j]
    x2 = torch.cat([x2, W.new_zeros(Q, L, QPAD - Q, L)], dim=2)     # pad a to 32
    return torch.cat([head, x2.reshape(-1)])


def unpack(x: torch.Tensor, L: int):
    """x (padded layout) -> (V, W)."""
    nsp = nsingle_padded(L)
    V = x[: (Q - 1) * L].reshape(Q - 1, L).transpose(0, 1)
    W = x[nsp:].reshape(Q, L, QPAD, L)[:, :, :Q, :].permute(1, 3, 0, 2)
    return V, W


class PseudoLikelihoodFunction(torch.autograd.Function):
    """f(x) for a padded parameter vector x; backward = the CUDA gradient kernels."""

    @staticmethod
    def forward(ctx, x: torch.Tensor, evaluator: Evaluator):
        if evaluator.gradient != "partial":
            raise ValueError("autograd needs an Evaluator with gradient='partial'")
        xc = x.detach().contiguous()
        g = torch.empty_like(xc)
        f = evaluator.evaluate(xc, g)
        ctx.save_for_backward(g)
        return torch.tensor(f, dtype=x.dtype, device=x.device)

    @staticmethod
    def backward(ctx, grad_out):
        (g,) = ctx.saved_tensors
        return grad_out * g, None


def _strides(t: torch.Tensor):
    return (ctypes.c_longlong * t.dim())(*t.stride())


def _target(t, dims: int):
    """Pointer and strides of a gradient, or of none."""
    return (None, (ctypes.c_longlong * dims)()) if t is None else (t.data_ptr(), _strides(t))


def _plain(t: torch.Tensor) -> bool:
    """A dense CUDA tensor with memory of its own (not one of a function transform)."""
    if not t.is_cuda or t.layout != torch.strided or t.is_conj() or t.is_neg():
        return False
    try:
        return t.data_ptr() != 0
    except RuntimeError:  # batched, functional or fake: no storage
        return False


def _native(V: torch.Tensor, W: torch.Tensor, evaluator: Evaluator) -> bool:
    """Whether the packing kernels take V and W: the shapes and the type of the
    evaluator's path, on the current device.  Everything else goes through pack(), with
    its own errors and promotions."""
    L = evaluator.L
    dtype = torch.float64 if evaluator.path == "simt_f64" else torch.float32
    return (V.shape == (L, Q - 1) and W.shape == (L, L, Q, Q) and V.dtype == W.dtype == dtype
            and _plain(V) and _plain(W) and V.device == W.device
            and V.device.index == torch.cuda.current_device())


class PseudoLikelihoodVWFunction(torch.autograd.Function):
    """f(V, W): the parameters packed and the gradient unpacked by one kernel each."""

    @staticmethod
    def forward(ctx, V: torch.Tensor, W: torch.Tensor, evaluator: Evaluator):
        if evaluator.gradient != "partial":
            raise ValueError("autograd needs an Evaluator with gradient='partial'")
        x = torch.empty(evaluator.nvar, dtype=V.dtype, device=V.device)
        g = torch.empty_like(x)
        check(lib().ccm_pack_parameters(V.data_ptr(), _strides(V), W.data_ptr(), _strides(W),
                                        evaluator.L, x.element_size(), x.data_ptr(),
                                        torch.cuda.current_stream().cuda_stream))
        f = evaluator.evaluate(x, g)
        ctx.save_for_backward(g)
        ctx.L = evaluator.L
        if V.dtype == torch.float32:
            f = ctypes.c_float(f).value  # infinite past its range, where full() would raise
        return torch.full((), f, dtype=V.dtype, device=V.device)

    @staticmethod
    def backward(ctx, grad_out):
        (g,) = ctx.saved_tensors
        L = ctx.L
        need_v, need_w, _ = ctx.needs_input_grad
        # (g may have been through saved-tensor hooks)
        if (torch.is_grad_enabled() or not _plain(grad_out) or not _plain(g)
                or not g.is_contiguous() or g.shape != (nvar_padded(L),)
                or grad_out.dtype != g.dtype or g.device.index != torch.cuda.current_device()):
            dV, dW = unpack(grad_out * g, L)  # differentiable, and open to transforms
            return dV if need_v else None, dW if need_w else None, None
        dV = torch.empty((L, Q - 1), dtype=g.dtype, device=g.device) if need_v else None
        dW = torch.empty((L, L, Q, Q), dtype=g.dtype, device=g.device) if need_w else None
        check(lib().ccm_unpack_gradient(g.data_ptr(), grad_out.data_ptr(), L, g.element_size(),
                                        *_target(dV, 2), *_target(dW, 4),
                                        torch.cuda.current_stream().cuda_stream))
        return dV, dW, None


def pseudo_likelihood(V: torch.Tensor, W: torch.Tensor, evaluator: Evaluator) -> torch.Tensor:
    """Differentiable f(V, W) (float32 on the tensor-core paths, float64 on simt_f64)."""
    if _native(V, W, evaluator):
        return PseudoLikelihoodVWFunction.apply(V, W, evaluator)
    x = pack(V, W)
    assert x.numel() == nvar_padded(V.shape[0])
    return PseudoLikelihoodFunction.apply(x, evaluator)
