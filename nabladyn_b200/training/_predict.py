"""Batched Lennard-Jones predictions with a hand-written parameter backward.

``predict`` gives the energy, forces and virial of F frames in one kernel launch
(nd_lj_frames); its autograd backward is nd_lj_frames_parameter_backward, which turns the
loss's gradients with respect to E, F and W into dLoss/dsigma and dLoss/depsilon in one pass
over the pairs. The reference gets the same numbers by a torch.func double backward through
vmapped forces (src/nabladyn/training/_loss.py:71-102, _fit.py:245-271).
"""

from __future__ import annotations

from collections.abc import Mapping

import torch
from torch import Tensor

from .._native import LJBatchArgs, call, dtype_code, on_device, ptr, stream_handle
from ..potential._lennard_jones import LennardJones, evaluate_frames

CHANNELS = ("energy", "forces", "virial")


class _BatchLJ(torch.autograd.Function):
    """(sigma, epsilon) -> (E [F], F [F, N, 3], W [F, 3, 3]) of fixed frames."""

    @staticmethod
    def forward(ctx, sigma, epsilon, positions, cells, stacks, kernel_types, num_types, cutoff):
        dtype = positions.dtype
        sigma_c = sigma.detach().to(dtype).contiguous()
        epsilon_c = epsilon.detach().to(dtype).contiguous()
        energy, forces, virial, packed = evaluate_frames(
            positions, cells, stacks, kernel_types, num_types, sigma_c, epsilon_c, cutoff, True)
        ctx.save_for_backward(sigma_c, epsilon_c, packed, cells, stacks, kernel_types)
        ctx.num_types, ctx.cutoff, ctx.num_atoms = num_types, cutoff, positions.shape[1]
        ctx.parameter_dtype = sigma.dtype
        return energy, forces, virial

    @staticmethod
    def backward(ctx, grad_energy, grad_forces, grad_virial):
        sigma, epsilon, packed, cells, stacks, kernel_types = ctx.saved_tensors
        dtype, device = cells.dtype, cells.device
        frames, atoms = cells.shape[0], ctx.num_atoms

        def given(gradient, shape):
            if gradient is None:
                return torch.zeros(shape, dtype=dtype, device=device)
            return gradient.to(dtype).contiguous()

        ge = given(grad_energy, frames)
        gf = given(grad_forces, (frames, atoms, 3))
        gw = given(grad_virial, (frames, 3, 3))
        rows = sigma.numel()
        grads = torch.empty((2, rows), dtype=dtype, device=device)
        workspace = torch.empty_like(packed)
        args = LJBatchArgs(
            dtype=dtype_code(dtype), frames=frames, positions=ptr(packed), cells=ptr(cells),
            num_atoms=atoms, pairs=ptr(stacks), capacity=stacks.shape[2],
            atom_types=ptr(kernel_types) if ctx.num_types > 1 else None,
            num_types=ctx.num_types, sigma=ptr(sigma), epsilon=ptr(epsilon),
            cutoff=float(ctx.cutoff), energy_grad=ptr(ge), forces_grad=ptr(gf),
            virial_grad=ptr(gw), sigma_grad=grads.data_ptr(),
            epsilon_grad=grads.data_ptr() + rows * grads.element_size(),
        )
        with on_device(device):
            call("nd_lj_frames_parameter_backward", args, ptr(workspace), stream_handle(device))
        out_dtype = ctx.parameter_dtype
        return grads[0].to(out_dtype), grads[1].to(out_dtype), None, None, None, None, None, None


def predict(model: LennardJones, parameters: Mapping[str, Tensor], positions: Tensor,
            cells: Tensor, stacks: tuple[Tensor, ...], channels: tuple[str, ...]) -> dict[str, Tensor]:
    """The channels of F frames by name, differentiable in ``parameters``.

    Lennard-Jones runs the batched kernels and the hand-written backward; any other model the
    reference's torch.func algorithm (``_generic.predict``).

    positions [F, N, 3] (anywhere), cells [F, 3], ``stacks`` one [F, 2, C] pair stack per
    cutoff of the model (one for Lennard-Jones); ``parameters`` replaces the model's "sigma"
    and/or "epsilon". Gives energy [F], forces [F, N, 3], virial [F, 3, 3]. Gradients flow to
    the parameters only.
    """
    if not isinstance(model, LennardJones):
        from ._generic import predict as generic_predict

        return generic_predict(model, parameters, positions, cells, stacks, channels)
    unknown = set(channels) - set(CHANNELS)
    if not channels or unknown:
        raise ValueError(f"channels must be a nonempty subsequence of {CHANNELS}")
    if cells.shape != (positions.shape[0], 3) or cells.device != positions.device:
        raise ValueError(f"cells must be a [{positions.shape[0]}, 3] tensor on {positions.device}")
    dtype = torch.promote_types(positions.dtype, cells.dtype)
    positions, cells = positions.detach().to(dtype), cells.detach().to(dtype)
    sigma = parameters.get("sigma", model.sigma)
    epsilon = parameters.get("epsilon", model.epsilon)
    stack = stacks[-1]
    if stack.dtype != torch.int32:
        stack = stack.to(torch.int32)
    energy, forces, virial = _BatchLJ.apply(
        sigma, epsilon, positions.contiguous(), cells.contiguous(), stack.contiguous(),
        model._kernel_types, model.num_types, model.cutoff,
    )
    values = {"energy": energy, "forces": forces, "virial": virial}
    return {name: values[name] for name in channels}


__all__ = ("predict", "CHANNELS")
