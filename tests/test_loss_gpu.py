"""nd_loss_forward and nd_loss_backward (through training.loss) against the torch operations that
define the loss, in float64: block edges, one to three channels, coefficients, strided inputs,
partial gradients, second derivatives, and the calls that must keep the defining operations.

Tolerances: squares and slopes carry three roundings of the dtype, sums are float64: 2e-6
relative (float32), 1e-13 (float64).
"""

import pytest
import torch

from nabladyn_b200 import training
from nabladyn_b200.training import _loss

pytestmark = pytest.mark.gpu

SCALES = {"energy": 3.0, "forces": 0.7, "virial": 11.0}
WEIGHTS = {"energy": 1.0, "forces": 2.5, "virial": 0.25}


def batch(frames, atoms, dtype, device, names):
    generator = torch.Generator().manual_seed(frames * 1000 + atoms)
    shapes = {"energy": (frames,), "forces": (frames, atoms, 3), "virial": (frames, 3, 3)}
    draw = lambda name: torch.randn(shapes[name], generator=generator,  # noqa: E731
                                    dtype=torch.float64).to(dtype).to(device)
    return {n: draw(n) for n in names}, {n: draw(n) for n in names}


def reference(predicted, labels, coefficients):
    p = {n: x.detach().double().requires_grad_(True) for n, x in predicted.items()}
    y = {n: x.double() for n, x in labels.items()}
    k = None if coefficients is None else coefficients.double()
    total, terms = _loss._defined(p, y, WEIGHTS, SCALES, k)
    return total, terms, dict(zip(p, torch.autograd.grad(total, list(p.values()))))


@pytest.mark.parametrize("dtype, tolerance", ((torch.float32, 2e-6), (torch.float64, 1e-13)))
@pytest.mark.parametrize("frames, atoms, names, weighted", [
    (1, 1, ("energy",), False), (3, 5, ("forces",), True),
    (2, 683, ("energy", "forces", "virial"), False),  # 2,049 components per block of 2,048
    (7, 301, ("forces", "virial"), True), (64, 4096, ("energy", "forces", "virial"), False),
])
def test_loss_and_gradient_match_float64(cuda, dtype, tolerance, frames, atoms, names, weighted):
    predicted, labels = batch(frames, atoms, dtype, cuda, names)
    coefficients = torch.rand(frames, device=cuda).to(dtype) if weighted else None
    leaves = {n: x.clone().requires_grad_(True) for n, x in predicted.items()}
    total, terms = training.loss(leaves, labels, WEIGHTS, SCALES, coefficients)
    assert total.grad_fn is not None and "_Loss" in type(total.grad_fn).__name__
    exact, exact_terms, exact_gradient = reference(predicted, labels, coefficients)
    assert abs(float(total) - float(exact)) <= tolerance * abs(float(exact))
    for name in names:
        assert abs(float(terms[name]) - float(exact_terms[name])) <= tolerance * float(exact_terms[name])
    for name in names:  # what a caller may do to them before the backward
        labels[name].zero_()
    gradient = torch.autograd.grad(total, list(leaves.values()), retain_graph=True)
    again = torch.autograd.grad(3.0 * total + terms[names[0]], leaves[names[0]])[0]
    for name, got in zip(names, gradient):
        scale = float(exact_gradient[name].abs().max())
        assert float((got.double() - exact_gradient[name]).abs().max()) <= tolerance * scale
    want = exact_gradient[names[0]] * (3.0 + 1.0 / WEIGHTS[names[0]])
    assert float((again.double() - want).abs().max()) <= 4 * tolerance * float(want.abs().max())


def test_other_calls_keep_the_defining_operations(cuda):
    predicted, labels = batch(4, 50, torch.float64, cuda, ("energy", "forces"))
    leaf = predicted["forces"].clone().requires_grad_(True)
    mixed = {"energy": predicted["energy"], "forces": leaf}
    total, _ = training.loss(mixed, labels, WEIGHTS, SCALES)  # one channel without a gradient
    first, = torch.autograd.grad(total, leaf, create_graph=True)
    second, = torch.autograd.grad(first.sum(), leaf)
    constant = 2.0 * WEIGHTS["forces"] / (4 * 150 * SCALES["forces"] ** 2)
    torch.testing.assert_close(second, torch.full_like(second, constant), rtol=1e-12, atol=0.0)
    # strided predictions and labels
    wide = torch.stack([predicted["forces"], predicted["forces"]], dim=-1)[..., 0]
    assert not wide.is_contiguous()
    got, _ = training.loss({"forces": wide}, {"forces": labels["forces"]}, WEIGHTS, SCALES)
    want, _ = _loss._defined({"forces": wide}, labels, WEIGHTS, SCALES, None)
    torch.testing.assert_close(got, want, rtol=1e-13, atol=0.0)
    # a transform, a tensor weight, a mixed dtype and a host batch
    value = torch.func.grad(lambda x: training.loss({"forces": x}, labels, WEIGHTS, SCALES)[0])
    torch.testing.assert_close(value(predicted["forces"]), value(predicted["forces"]))
    for p, y, w in (
        ({"forces": leaf}, labels, {"forces": torch.tensor(2.5, device=cuda)}),
        ({"forces": leaf.float()}, labels, WEIGHTS),
        ({"forces": predicted["forces"].cpu()}, {"forces": labels["forces"].cpu()}, WEIGHTS),
    ):
        assert not _loss._one_kernel(p, y, w, SCALES, None)
        got, _ = training.loss(p, y, w, SCALES)
        assert float(got) == pytest.approx(float(want), rel=1e-5)
