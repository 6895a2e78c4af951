"""The supervised loss: scaled errors of predicted energies, forces and virials.

The same scales and loss as src/nabladyn/training/_loss.py:26-46 and :105-125. On a GPU the
loss of plain tensors and its first derivatives take one kernel each (nd_loss_forward,
nd_loss_backward); anything else, such as a functorch transform, tensor weights, batched
gradients or a second derivative, is computed by torch operations.
"""

import ctypes
from collections.abc import Mapping

import torch
from torch import Tensor
from torch.autograd import forward_ad
from torch.overrides import _get_current_function_mode_stack
from torch.utils._device import DeviceContext

from .._native import LOSS_PARTIALS, LossArgs, call, dtype_code, on_device, ptr, stream_handle

CHANNELS = ("energy", "forces", "virial")


def scales(energy: Tensor | None = None, forces: Tensor | None = None,
           virial: Tensor | None = None) -> dict[str, float]:
    """Each given channel's scale from its labels: energy [F] and virial [F, 3, 3] by the RMS
    about the mean over frames, forces [F, N, 3] by the plain RMS; constant labels fall back to
    the plain RMS and all-zero labels to 1. Syncs with the host."""
    result = {}
    for name, labels, about_mean in (("energy", energy, True), ("forces", forces, False),
                                     ("virial", virial, True)):
        if labels is not None:
            rms = float(labels.square().mean().sqrt())
            spread = rms
            if about_mean:
                spread = float((labels - labels.mean(dim=0)).square().mean().sqrt())
            result[name] = spread or rms or 1.0
    return result


def loss(predicted: Mapping[str, Tensor], labels: Mapping[str, Tensor],
         weights: Mapping[str, float | Tensor], scales: Mapping[str, float | Tensor],
         coefficients: Tensor | None = None) -> tuple[Tensor, dict[str, Tensor]]:
    """The batch loss, the weighted sum of its channel terms, and the terms by name.

    A channel's term is each frame's mean of ((X - X*) / s_X)^2 over its components, times the
    frame's coefficient [B] (1/B when ``coefficients`` is None), summed over the frames.
    """
    if _one_kernel(predicted, labels, weights, scales, coefficients):
        names = tuple(predicted)
        total, *rest = _Loss.apply(
            tuple(float(weights[name]) for name in names),
            tuple(float(scales[name]) for name in names), coefficients,
            *(labels[name] for name in names), *(predicted[name] for name in names))
        return total, dict(zip(names, rest))
    return _defined(predicted, labels, weights, scales, coefficients)


def _defined(predicted, labels, weights, scales, coefficients):
    """The loss by torch operations."""
    terms = {}
    for name, value in predicted.items():
        squares = ((value - labels[name]) / scales[name]).square()
        per_frame = squares.reshape(squares.shape[0], -1).mean(dim=1)
        terms[name] = per_frame.mean() if coefficients is None else (coefficients * per_frame).sum()
    return sum(weights[name] * term for name, term in terms.items()), terms


def _plain_context() -> bool:
    """Whether nothing watches or transforms torch operations: no functorch transform,
    forward-mode level, trace, dispatch or function mode, which see the operations of a formula
    and would not see a kernel. (A default device is a function mode that watches nothing.)"""
    return not (torch._C._are_functorch_transforms_active() or forward_ad._current_level >= 0
                or torch.compiler.is_compiling() or torch.jit.is_tracing()
                or torch._C._len_torch_dispatch_stack()
                or (torch._C._len_torch_function_stack()
                    and any(not isinstance(mode, DeviceContext)
                            for mode in _get_current_function_mode_stack())))


def _one_kernel(predicted, labels, weights, scales, coefficients) -> bool:
    """Whether the loss is one of plain CUDA tensors with number weights and scales, and nothing
    watches its operations."""
    if not 1 <= len(predicted) <= 3 or not _plain_context():
        return False
    first = next(iter(predicted.values()))
    if (not isinstance(first, Tensor) or not first.is_cuda or first.ndim == 0
            or first.dtype not in (torch.float32, torch.float64) or first.shape[0] == 0):
        return False
    frames = first.shape[0]

    def plain(x, shape) -> bool:
        return (type(x) in (Tensor, torch.nn.Parameter) and x.layout is torch.strided
                and x.dtype == first.dtype and x.device == first.device and x.shape == shape)

    for name, value in predicted.items():
        label, weight, scale = labels[name], weights[name], scales[name]
        if (not isinstance(weight, (int, float)) or not isinstance(scale, (int, float))
                or not isinstance(label, Tensor) or label.requires_grad or not plain(value, label.shape)
                or not plain(label, value.shape) or value.ndim == 0 or value.shape[0] != frames
                or value.numel() == 0):
            return False
    return coefficients is None or (isinstance(coefficients, Tensor)
                                    and not coefficients.requires_grad
                                    and plain(coefficients, (frames,)))


class _Loss(torch.autograd.Function):
    """(L, t_c for every channel, their slopes dt_c/dX) of predictions, differentiable in the
    predictions to any order.

    The slopes are outputs, and all that is saved: the first derivative scales them and the second
    differentiates them through this node again (dt_c/dX is linear in X), so nothing of the
    predictions and labels is kept, a caller may overwrite them before the backward, and saved
    tensors are released and hooked like those of any other operation.
    """

    @staticmethod
    def forward(ctx, weights, scales, coefficients, *tensors):
        count = len(weights)
        labels, predicted = tensors[:count], tensors[count:]
        like = predicted[0]
        total, *terms = (torch.empty((), dtype=like.dtype, device=like.device)
                         for _ in range(1 + count))
        wanted = ctx.needs_input_grad[3 + count:]
        slopes = [torch.empty(value.shape, dtype=like.dtype, device=like.device) if want else None
                  for value, want in zip(predicted, wanted)]
        partials = torch.empty(LOSS_PARTIALS, dtype=torch.float64, device=like.device)
        kept = [value.contiguous() for value in (*predicted, *labels)]  # until the launch
        shares = None if coefficients is None else coefficients.contiguous()
        args = _loss_args(weights, kept[:count])
        args.coefficients, args.partials, args.total = ptr(shares), ptr(partials), ptr(total)
        for c, term in enumerate(terms):
            args.labels[c], args.scales[c] = ptr(kept[count + c]), scales[c]
            args.terms[c], args.gradients[c] = ptr(term), ptr(slopes[c])
        with on_device(like.device):
            call("nd_loss_forward", ctypes.byref(args), stream_handle(like.device))
        ctx.weights, ctx.scales = weights, scales
        ctx.set_materialize_grads(False)
        ctx.save_for_backward(coefficients, *slopes)
        return total, *terms, *slopes

    @staticmethod
    def backward(ctx, total_grad, *rest):
        count = len(ctx.weights)
        term_grads, slope_grads = rest[:count], rest[count:]
        coefficients, *slopes = ctx.saved_tensors
        given = [g for g in (total_grad, *term_grads) if g is not None]
        if (torch.is_grad_enabled() or any(g is not None for g in slope_grads)
                or not _plain_context() or not all(_addressable(g, slopes) for g in given)):
            gradients = [_gradient(ctx, c, slope, coefficients, total_grad, term_grads[c],
                                   slope_grads[c]) for c, slope in enumerate(slopes)]
        else:
            gradients = [None if slope is None else torch.empty_like(slope) for slope in slopes]
            like = next(slope for slope in slopes if slope is not None)
            args = _loss_args(ctx.weights, [like if s is None else s for s in slopes])
            args.total_grad = ptr(total_grad)
            for c, gradient in enumerate(gradients):
                args.term_grads[c], args.gradients[c] = ptr(term_grads[c]), ptr(gradient)
            with on_device(like.device):
                call("nd_loss_backward", ctypes.byref(args), stream_handle(like.device))
        return (None, None, None, *(None,) * count, *gradients)


def _addressable(gradient: Tensor, slopes) -> bool:
    """Whether an incoming gradient is one number of the slopes' dtype in memory (a batched one,
    of a vectorised Jacobian, has no storage)."""
    like = next((slope for slope in slopes if slope is not None), None)
    return (like is not None and type(gradient) is Tensor and torch._C._has_storage(gradient)
            and gradient.layout is torch.strided and gradient.ndim == 0
            and gradient.dtype == like.dtype and gradient.device == like.device)


def _gradient(ctx, c, slope, coefficients, total_grad, term_grad, slope_grad):
    """dL/dX of channel c by torch operations, differentiable themselves."""
    if slope is None:
        return None
    parts = []
    if total_grad is not None:
        parts.append(total_grad * ctx.weights[c] * slope)
    if term_grad is not None:
        parts.append(term_grad * slope)
    if slope_grad is not None:  # dt_c/dX = 2 k_f (X - Y) / (n s_c^2)
        frames = slope.shape[0]
        factor = 2.0 / (slope.numel() // frames * ctx.scales[c] ** 2)
        parts.append(slope_grad * (factor / frames) if coefficients is None else
                     slope_grad * (factor * coefficients.reshape(frames, *(1,) * (slope.ndim - 1))))
    return sum(parts) if parts else None


def _loss_args(weights, channels) -> LossArgs:
    """The arguments of one tensor [F, ...] per channel."""
    args = LossArgs(dtype=dtype_code(channels[0].dtype), channels=len(weights),
                    frames=channels[0].shape[0])
    for c, value in enumerate(channels):
        args.predicted[c], args.sizes[c] = ptr(value), value.numel() // value.shape[0]
        args.weights[c] = weights[c]
    return args


__all__ = ("CHANNELS", "scales", "loss")
