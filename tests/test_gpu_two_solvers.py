"""Solvers of different sizes that are alive at the same time."""
import numpy as np
import pytest
import torch

from mydemcfd_b200 import _native as nat
from mydemcfd_b200 import workloads as W
from mydemcfd_b200.solver import B200PressureSolver, DeviceGrid, SMACStep

pytestmark = pytest.mark.gpu


def step_of(N, precision):
    case = W.vof_case(N[0], seed=5, ratio=100.0, N=N)
    g = DeviceGrid.from_case(case)
    step = SMACStep(g, case.dt)
    step.pressure_solver_ = B200PressureSolver(N, case.h, precision=precision, tol=1e-8)
    return step


def solution(step):
    st = step.solve_poisson()
    torch.cuda.synchronize()
    assert st["status"] == 0
    return step.grid_.p_delta_.cpu().numpy()


@pytest.mark.parametrize("precision", [nat.PRECISION_FP64, nat.PRECISION_MIXED])
@pytest.mark.parametrize("small", [(25, 25, 25), (38, 25, 19), (16, 16, 16)])
def test_a_smaller_solver_leaves_a_larger_one_as_it_is(small, precision):
    """The larger solver's kernels are captured at its first solve, and again once its options change: both after the
    smaller solver, whose cluster kernel needs less shared memory, was made."""
    alone = step_of((64, 64, 64), precision)
    want = solution(alone)
    alone.pressure_solver_.close()
    large = step_of((64, 64, 64), precision)
    other = step_of(small, precision)
    assert np.array_equal(solution(large), want)
    first = solution(other)
    large.pressure_solver_.set_options(nu1=1)
    large.pressure_solver_.set_options(nu1=2)
    again = step_of(small, precision)
    assert np.array_equal(solution(large), want)
    assert np.array_equal(solution(again), first)
    assert np.array_equal(solution(other), first)
