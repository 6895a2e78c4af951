"""The Lennard-Jones entry points that take no workspace (nd_lj_batch_forward,
nd_lj_batch_parameter_backward, nd_lj_energy_force_virial without strain or parameter gradients),
called as a C program calls them, against plain torch float64 on the frames of the packed forms'
tests: capacities around a lane's and a warp's columns, columns in any order, padding and invalid
columns, one to eight types.

Tolerances as there: float64 sums keep 1e-12 of their scale (gradients 1e-11), float32 pair terms
1e-5 (gradients 1e-4).
"""

import pytest
import torch

from nabladyn_b200 import space
from nabladyn_b200._native import LJBatchArgs, LJPairsArgs, call, dtype_code, ptr, stream_handle
from test_lj_frames_gpu import CUTOFF, reference, system

pytestmark = pytest.mark.gpu

CASES = [(1, 2, 1, 1, True), (2, 9, 5, 2, False), (3, 40, 127, 1, True), (2, 65, 129, 2, True),
         (3, 130, 1023, 3, False), (1, 130, 1025, 1, True), (2, 500, 40003, 8, True)]


def arguments(x, cells, index, kinds, types, sigma, epsilon):
    return LJBatchArgs(
        dtype=dtype_code(x.dtype), frames=x.shape[0], positions=ptr(x), cells=ptr(cells),
        num_atoms=x.shape[1], pairs=ptr(index), capacity=index.shape[2], atom_types=ptr(kinds),
        num_types=types, sigma=ptr(sigma), epsilon=ptr(epsilon), cutoff=CUTOFF)


def prepared(case, dtype, device):
    frames, atoms, capacity, types, grouped = case
    x, cells, index, kinds, sigma, epsilon = system(frames, atoms, capacity, types, dtype, device,
                                                    grouped)
    return (space.wrapped_only(x, cells), cells, index, kinds.to(torch.int32), types, sigma,
            epsilon)


def outputs(frames, atoms, dtype, device):
    return (torch.full((frames,), 7.0, dtype=torch.float64, device=device),
            torch.full((frames, atoms, 3), 7.0, dtype=dtype, device=device),
            torch.full((frames, 3, 3), 7.0, dtype=torch.float64, device=device))


def check(got, want, tolerance):
    for value, exact in zip(got, want):
        scale = float(exact.abs().max()) + 1.0
        assert float((value.double() - exact).abs().max()) <= tolerance * scale


@pytest.mark.parametrize("dtype, tolerance", ((torch.float32, 1e-5), (torch.float64, 1e-12)))
@pytest.mark.parametrize("case", CASES)
def test_batch_forward(cuda, dtype, tolerance, case):
    given = prepared(case, dtype, cuda)
    got = outputs(case[0], case[1], dtype, cuda)
    args = arguments(*given)
    args.energy, args.forces, args.virial = (ptr(t) for t in got)
    call("nd_lj_batch_forward", args, stream_handle(cuda))
    check(got, reference(given[0], given[1], given[2], given[3].long(), *given[4:]), tolerance)


@pytest.mark.parametrize("dtype, tolerance", ((torch.float32, 1e-4), (torch.float64, 1e-11)))
@pytest.mark.parametrize("case", CASES)
def test_batch_parameter_backward(cuda, dtype, tolerance, case):
    x, cells, index, kinds, types, sigma, epsilon = prepared(case, dtype, cuda)
    generator = torch.Generator().manual_seed(case[2])
    adjoints = [torch.randn(shape, generator=generator, dtype=torch.float64).to(cuda)
                for shape in ((case[0],), (case[0], case[1], 3), (case[0], 3, 3))]
    adjoints[1] = adjoints[1].to(dtype)
    got = torch.full((2, sigma.numel()), 7.0, dtype=torch.float64, device=cuda)
    args = arguments(x, cells, index, kinds, types, sigma, epsilon)
    args.energy_grad, args.forces_grad, args.virial_grad = (ptr(t) for t in adjoints)
    args.sigma_grad, args.epsilon_grad = got[0].data_ptr(), got[1].data_ptr()
    call("nd_lj_batch_parameter_backward", args, stream_handle(cuda))
    parameters = [p.double().requires_grad_(True) for p in (sigma, epsilon)]
    exact = reference(x, cells, index, kinds.long(), types, *parameters)
    want = torch.autograd.grad(exact, parameters, [a.double() for a in adjoints])
    check(got, want, tolerance)


@pytest.mark.parametrize("dtype, tolerance", ((torch.float32, 1e-5), (torch.float64, 1e-12)))
@pytest.mark.parametrize("case", [case for case in CASES if case[0] == 1] + [(1, 500, 200003, 3, True)])
def test_one_frame(cuda, dtype, tolerance, case):
    x, cells, index, kinds, types, sigma, epsilon = given = prepared(case, dtype, cuda)
    got = outputs(1, case[1], dtype, cuda)
    args = LJPairsArgs(
        dtype=dtype_code(dtype), positions=ptr(x), cell=ptr(cells), num_atoms=case[1],
        pairs=ptr(index), capacity=index.shape[2], atom_types=ptr(kinds), num_types=types,
        sigma=ptr(sigma), epsilon=ptr(epsilon), cutoff=CUTOFF, energy=ptr(got[0]),
        forces=ptr(got[1]), virial=ptr(got[2]))
    call("nd_lj_energy_force_virial", args, stream_handle(cuda))
    check(got, reference(given[0], given[1], given[2], given[3].long(), *given[4:]), tolerance)
