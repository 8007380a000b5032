"""Multigrid hierarchies of odd extents (n -> (n + 1) / 2, a last coarse cell with one child)."""
import dataclasses

import numpy as np
import pytest
import torch

from mydemcfd_b200 import _native as nat
from mydemcfd_b200 import workloads as W
from mydemcfd_b200.solver import B200PressureSolver, DeviceGrid, SMACStep, update_boundary_faces_device

pytestmark = pytest.mark.gpu

# odd at the first halving, at later ones, in one, two or all directions; the smallest that is halved; rows wider
# than the z-march's tile; planes that leave cluster ranks without work; 4097 cells, one more than a CTA's set
SIZES = [(25, 25, 25), (7, 9, 11), (50, 33, 18), (37, 24, 42), (75, 50, 38), (259, 9, 13), (16, 15, 95), (17, 241, 8),
         (22, 26, 31)]
# iterations measured with walls all around and with outlets, FP64 and mixed; where the mixed form takes more it has
# started again at a reliable update
ITERATIONS = {(25, 25, 25): (8, 8, 9, 9), (7, 9, 11): (8, 8, 7, 7), (50, 33, 18): (10, 10, 9, 9),
              (37, 24, 42): (10, 10, 9, 9), (75, 50, 38): (9, 9, 9, 9), (259, 9, 13): (30, 41, 8, 8),
              (16, 15, 95): (11, 12, 8, 8), (17, 241, 8): (27, 35, 9, 9), (22, 26, 31): (8, 8, 8, 8)}


def solved(N, precision, outlet, **options):
    case = dataclasses.replace(W.vof_case(N[0], seed=5, ratio=100.0, N=N), h=(1.0 / N[0],) * 3)
    g = DeviceGrid.from_case(case)
    if outlet:
        marks = tuple(torch.from_numpy(m).cuda() for m in W.outlet_marks(N, ("x+", "y+", "z+")))
        update_boundary_faces_device(N, case.h, marks, (g.f_bx_, g.f_by_, g.f_bz_))
    s = B200PressureSolver(N, case.h, precision=precision, solver_type=nat.GMG_PCG if outlet else
                           nat.PURENEUMANN_GMG_PCG, **options)
    step = SMACStep(g, case.dt)
    step.pressure_solver_ = s
    st = step.solve_poisson()
    torch.cuda.synchronize()
    return g, s, st


@pytest.mark.parametrize("outlet", [False, True])
@pytest.mark.parametrize("precision", [nat.PRECISION_FP64, nat.PRECISION_MIXED])
@pytest.mark.parametrize("N", SIZES)
def test_odd_extents_solve_in_few_iterations(N, precision, outlet):
    """The solve reaches the tolerance by the operator applied to its result, in at most two iterations more than it
    is known to take (a hierarchy cut at the first odd extent takes 30 to 60 on the compact grids), and every level
    halves."""
    tol = 1e-10
    g, s, st = solved(N, precision, outlet, tol=tol)
    assert st["status"] == 0
    known = ITERATIONS[N][2 * outlet + (precision == nat.PRECISION_MIXED)]
    assert st["iterations"] <= known + 2, st
    n = s.num_levels()
    assert all(m < 7 for m in s.level_shape(n - 1))
    y = torch.zeros_like(g.rhs_)
    s.apply_A(g.p_delta_, y)
    b, ax = W.interior(g.rhs_.cpu().numpy()), W.interior(y.cpu().numpy())
    if not outlet:
        b = b - b.mean()
    # the norm's rounding: 1e-15 of the terms, whose norm is at most |diag| |p| (h^-2, ratio 1)
    slack = 1e-15 * 12 * N[0] ** 2 * np.linalg.norm(W.interior(g.p_delta_.cpu().numpy()))
    assert np.linalg.norm(b - ax) <= tol * np.linalg.norm(b) + slack


@pytest.mark.parametrize("outlet", [False, True])
@pytest.mark.parametrize("precision", [nat.PRECISION_FP64, nat.PRECISION_MIXED])
@pytest.mark.parametrize("N", SIZES)
def test_odd_extents_every_kernel_gives_the_same_bits(N, precision, outlet):
    """Cluster set or single CTA, and each sweep kernel of the separately launched grids: the same p_delta."""
    ref = None
    for options in ({}, {"coarse_kernel": nat.COARSE_CTA}, {"sweep_kernel": nat.SWEEP_TMA},
                    {"sweep_kernel": nat.SWEEP_ZMARCH}, {"sweep_kernel": nat.SWEEP_SHARED}):
        g, s, st = solved(N, precision, outlet, tol=1e-9, **options)
        # (the last sweep's r.z is summed in another order by each kernel: the sweep itself is compared)
        if s.num_levels() >= 2:
            for mode in (0, 1, 2):
                assert s.selftest_sweep(precision, mode) == 0, (options, mode)
        p = g.p_delta_.cpu().numpy()
        if "sweep_kernel" not in options:
            ref = p if ref is None else ref
            assert np.array_equal(p, ref), options
        assert np.linalg.norm(p - ref) <= 1e-6 * np.linalg.norm(ref), options
        s.close()


@pytest.mark.parametrize("precision", [nat.PRECISION_FP64, nat.PRECISION_MIXED])
@pytest.mark.parametrize("N, min_coarse, levels", [
    ((1024, 2, 2), 4, 9),    # 4096 cells, the most that one CTA takes, halved eight times
    ((2, 801, 2), 4, 9),     # odd on the way down
    ((3, 2, 640), 2, 10),    # 640, 320, ..., 5, 3, 2
    ((257, 4, 3), 2, 9),
])
def test_one_cta_takes_as_many_grids_as_there_are(N, min_coarse, levels, precision):
    """Long thin grids: more than eight grids of at most 4096 cells, solved twice."""
    g, s, st = solved(N, precision, False, tol=1e-8, min_coarse=min_coarse)
    assert s.num_levels() == levels and s.level_shape(levels - 1)[int(np.argmax(N))] <= 4
    assert st["status"] == 0
    first = g.p_delta_.clone()
    s.divergence(g, 1.0)
    s.solve_rhs(g.p_delta_)
    assert torch.equal(first, g.p_delta_)
    y = torch.zeros_like(g.rhs_)
    s.apply_A(g.p_delta_, y)
    b, ax = W.interior(g.rhs_.cpu().numpy()), W.interior(y.cpu().numpy())
    b = b - b.mean()
    slack = 1e-15 * 12 * N[0] ** 2 * np.linalg.norm(W.interior(g.p_delta_.cpu().numpy()))
    assert np.linalg.norm(b - ax) <= 1e-8 * np.linalg.norm(b) + slack
