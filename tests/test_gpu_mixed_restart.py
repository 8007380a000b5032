"""Mixed precision where the FP32 increment's rounding lifts the true residual above the recursive one."""
import dataclasses

import numpy as np
import pytest
import torch

from mydemcfd_b200 import _native as nat
from mydemcfd_b200 import workloads as W
from mydemcfd_b200.solver import B200PressureSolver, DeviceGrid, SMACStep, update_boundary_faces_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [(64, 64, 64), (128, 128, 128), (128, 96, 64)])
def test_mixed_channel_takes_about_the_iterations_of_fp64(N):
    """A channel (inflow x-, outlet x+): the pressure is smooth and large, and the FP64 residual at a reliable update
    is not the recursive one.  PCG restarted there needs at most one more cycle of iterations per reliable update
    than FP64 (with the old direction kept: 42, no convergence within 2000, and 281)."""
    case = dataclasses.replace(W.vof_case(N[0], seed=2, ratio=100.0, N=N), h=(1.0 / N[0],) * 3)
    x = (np.arange(N[0] + 3) - 1.0) / N[0]
    vxs = np.where(case.fxt == W.F_INTERIOR, np.sin(6.0 * x)[None, None, :], 0.0)
    vxs[1:-1, 1:-1, 1] = 1.0
    case = dataclasses.replace(case, vxs=vxs, dt=0.1 / N[0])
    its = {}
    for precision in (nat.PRECISION_FP64, nat.PRECISION_MIXED):
        g = DeviceGrid.from_case(case)
        marks = tuple(torch.from_numpy(m).cuda() for m in W.outlet_marks(N, ("x+",)))
        update_boundary_faces_device(N, case.h, marks, (g.f_bx_, g.f_by_, g.f_bz_))
        s = B200PressureSolver(N, case.h, tol=1e-8, precision=precision, solver_type=nat.GMG_PCG)
        step = SMACStep(g, case.dt)
        step.pressure_solver_ = s
        st = step.solve_poisson()
        assert st["status"] == 0 and st["rel_residual"] <= 1e-8, st
        its[precision] = st["iterations"]
    assert its[nat.PRECISION_MIXED] <= 2 * its[nat.PRECISION_FP64] + 4, its
