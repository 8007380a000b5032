"""How many iterations a solve may launch, and what it launches for nothing."""
import dataclasses

import pytest

from mydemcfd_b200 import _native as nat
from mydemcfd_b200 import workloads as W
from mydemcfd_b200.solver import B200PressureSolver, DeviceGrid

pytestmark = pytest.mark.gpu


def make(n, ratio, **options):
    case = dataclasses.replace(W.vof_case(n, seed=5, ratio=ratio), h=(1.0 / n,) * 3)
    g = DeviceGrid.from_case(case)
    s = B200PressureSolver(case.N, case.h, **options)
    s.set_coefficients(g)
    s.divergence(g, case.dt)
    return g, s


@pytest.mark.parametrize("n", [48, 64])
def test_a_restarted_solve_may_use_every_iteration_it_is_allowed(n):
    """A Jacobi solve of hundreds of iterations to 1e-14, whose recursive residual gets there before the true one, so
    that PCG starts again: iterations launched after the first stop, which do nothing, do not count against
    max_iter."""
    g, s = make(n, 1000.0, solver_type=nat.PURENEUMANN_STANDARD_PCG, tol=1e-14, max_iter=100000)
    its = s.solve_rhs(g.p_delta_)["iterations"]
    assert its > 200
    for extra in (0, 1, 2, 7):
        s.set_options(max_iter=its + extra)
        st = s.solve_rhs(g.p_delta_)
        assert st["status"] == 0 and st["iterations"] == its and st["rel_residual"] <= 1e-14, (extra, st)
    s.set_options(max_iter=its // 2)
    st = s.solve_rhs(g.p_delta_, raise_on_fail=False)
    assert st["status"] == nat.NOT_CONVERGED and st["iterations"] == its // 2, st
    assert 1e-14 < st["rel_residual"] < 1e-4


@pytest.mark.parametrize("precision", [nat.PRECISION_FP64, nat.PRECISION_MIXED])
def test_a_zero_right_hand_side_launches_no_more_than_two_iterations(precision):
    g, s = make(32, 100.0, precision=precision, tol=1e-8, max_iter=2)
    capped = s.solve_rhs(g.p_delta_, raise_on_fail=False)
    assert capped["iterations"] == 2
    s.set_options(max_iter=2000)
    g.rhs_.zero_()
    s.set_rhs(g.rhs_)
    st = s.solve_rhs(g.p_delta_)
    assert st["status"] == 0 and st["iterations"] == 0 and not g.p_delta_.any()
    assert st["kernel_launches"] <= capped["kernel_launches"]


@pytest.mark.parametrize("precision", [nat.PRECISION_FP64, nat.PRECISION_MIXED])
def test_a_long_solve_runs_in_batches(precision):
    """A Jacobi solve of hundreds of iterations: batches of an eighth of those done find the same end as a solve that
    may launch no more than it needs, and the mixed form takes about the iterations of FP64."""
    g, s = make(64, 1000.0, solver_type=nat.PURENEUMANN_STANDARD_PCG, precision=precision, tol=1e-10)
    st = s.solve_rhs(g.p_delta_)
    assert st["status"] == 0 and st["rel_residual"] <= 1e-10
    assert 500 < st["iterations"] < 600      # 547 in FP64, 572 mixed
    p = g.p_delta_.clone()
    s.set_options(max_iter=st["iterations"])
    s.divergence(g, 1.0)
    again = s.solve_rhs(g.p_delta_)
    assert again["iterations"] == st["iterations"] and (p == g.p_delta_).all()
    assert again["kernel_launches"] <= st["kernel_launches"]
