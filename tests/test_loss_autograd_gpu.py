"""The one-kernel training loss under autograd's other uses: each gives what the loss by torch
operations gives, and refuses what it refuses.

Tolerance, float64: slopes and sums carry a few roundings, 1e-12 relative.
"""

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from nabladyn_b200 import training
from nabladyn_b200.training import _loss

pytestmark = pytest.mark.gpu

WEIGHTS, SCALES = {"energy": 1.5, "forces": 2.5}, {"energy": 3.0, "forces": 0.7}
CLOSE = {"rtol": 1e-12, "atol": 0.0}


@pytest.fixture(params=[False, True], ids=["even", "weighted"])
def case(cuda, request):
    generator = torch.Generator().manual_seed(5)
    draw = lambda *shape: torch.randn(shape, generator=generator,  # noqa: E731
                                      dtype=torch.float64).to(cuda)
    predicted = {"energy": draw(4).requires_grad_(True),
                 "forces": draw(4, 50, 3).requires_grad_(True)}
    labels = {"energy": draw(4), "forces": draw(4, 50, 3)}
    return predicted, labels, draw(4).abs() if request.param else None


def kernel(case):
    predicted, labels, coefficients = case
    total, terms = training.loss(predicted, labels, WEIGHTS, SCALES, coefficients)
    assert "_Loss" in type(total.grad_fn).__name__
    return total, terms


def defined(case):
    return _loss._defined(*case[:2], WEIGHTS, SCALES, case[2])


def leaves(case):
    return list(case[0].values())


def test_batched_gradients(case):
    """A vectorised Jacobian of outputs computed outside a transform."""
    def rows(pair):
        total, terms = pair
        return torch.autograd.grad([total, terms["forces"]], leaves(case),
                                   [torch.tensor([1.0, 0.0, 3.0], dtype=torch.float64).cuda(),
                                    torch.tensor([0.0, 2.0, 1.0], dtype=torch.float64).cuda()],
                                   is_grads_batched=True)

    for got, want in zip(rows(kernel(case)), rows(defined(case))):
        assert got.shape == want.shape
        torch.testing.assert_close(got, want, **CLOSE)


def test_a_freed_graph_is_refused(case):
    total, _ = kernel(case)
    total.backward()
    with pytest.raises(RuntimeError, match="second time"):
        total.backward()


def test_saved_tensor_hooks_see_what_is_kept(case):
    kept = []

    def pack(x):
        kept.append(x.shape)
        return x.cpu()

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda x: x.cuda()):
        total, _ = kernel(case)
    assert torch.Size([4, 50, 3]) in kept
    for got, want in zip(torch.autograd.grad(total, leaves(case)),
                         torch.autograd.grad(defined(case)[0], leaves(case))):
        torch.testing.assert_close(got, want, **CLOSE)


def test_second_derivatives(case):
    def second(pair):
        first = torch.autograd.grad(pair[0] + pair[1]["energy"], leaves(case), create_graph=True)
        return torch.autograd.grad(sum((g * g).sum() for g in first), leaves(case))

    for got, want in zip(second(kernel(case)), second(defined(case))):
        torch.testing.assert_close(got, want, **CLOSE)


def test_inputs_may_be_overwritten_before_the_backward(case):
    predicted, labels, coefficients = case
    want = torch.autograd.grad(defined(case)[0], leaves(case), create_graph=True)
    inner = {name: x * 1.0 for name, x in predicted.items()}
    total, _ = training.loss(inner, {k: x.clone() for k, x in labels.items()}, WEIGHTS, SCALES,
                             coefficients)
    with torch.no_grad():
        for x in inner.values():
            x.zero_()
    for create_graph in (False, True):
        got = torch.autograd.grad(total, leaves(case), retain_graph=True,
                                  create_graph=create_graph)
        for g, w in zip(got, want):
            torch.testing.assert_close(g, w.detach(), **CLOSE)


def test_forward_mode_in_the_backward(case):
    """A directional derivative of the gradient in the incoming gradient."""
    def tangent(pair):
        with torch.autograd.forward_ad.dual_level():
            one = torch.tensor(1.0, dtype=torch.float64, device="cuda")
            seed = torch.autograd.forward_ad.make_dual(one, 2.0 * one)
            got = torch.autograd.grad(pair[0], leaves(case), seed)
            return [torch.autograd.forward_ad.unpack_dual(g).tangent for g in got]

    for got, want in zip(tangent(kernel(case)), tangent(defined(case))):
        torch.testing.assert_close(got, want, **CLOSE)


def test_a_transform_gives_the_analytic_slope(case):
    predicted, labels, coefficients = case
    x = predicted["forces"].detach()
    got = torch.func.grad(lambda y: training.loss({"forces": y}, labels, WEIGHTS, SCALES,
                                                  coefficients)[0])(x)
    share = (torch.full((4,), 0.25, dtype=torch.float64, device=x.device)
             if coefficients is None else coefficients)
    want = (2.0 * WEIGHTS["forces"] / (150 * SCALES["forces"] ** 2)
            * share[:, None, None] * (x - labels["forces"]))
    torch.testing.assert_close(got, want, **CLOSE)


def test_a_dispatch_mode_sees_the_operations(case):
    class Names(TorchDispatchMode):
        seen = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.seen.append(str(func))
            return func(*args, **(kwargs or {}))

    predicted, labels, coefficients = case
    with Names():
        training.loss({k: v.detach() for k, v in predicted.items()}, labels, WEIGHTS, SCALES,
                      coefficients)
    assert any("sub" in name for name in Names.seen) and any("mean" in n for n in Names.seen)


def test_a_default_device_keeps_the_kernel(case):
    with torch.device("cuda"):
        total, _ = kernel(case)  # asserts the kernel's node
    torch.testing.assert_close(total, defined(case)[0], **CLOSE)
