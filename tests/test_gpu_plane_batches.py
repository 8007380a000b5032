"""Kernels that take several planes per thread or per block, at depths and rows that do not fill the last one."""
import numpy as np
import pytest
import torch

from _cases import ref_grid
from mydemcfd_b200 import workloads as W
from mydemcfd_b200.solver import B200PressureSolver, DeviceGrid, face_gradp_device, surface_tension_device
from oracle import oracle as O
from test_gpu_post import ST_KEYS, run_surface
from test_gpu_predictor_tiles import _device_us

pytestmark = pytest.mark.gpu

SIZES = [(33, 9, 7), (32, 8, 5), (31, 4, 3), (2, 3, 4), (65, 5, 17)]


def rnd(seed, shape, lo=-1.0, hi=1.0):
    return (lo + (hi - lo) * W.uniform01(seed, int(np.prod(shape)))).reshape(shape)


@pytest.mark.parametrize("with_eps, with_fs", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("N", SIZES)
def test_divergence_and_correction_bit_exact_over_depths(N, with_eps, with_fs):
    case = W.vof_case(N[0], seed=4, ratio=30.0, N=N)
    case.dt = 0.5
    sh = W.shapes(N)
    kw = {}
    if with_eps:
        kw.update(eps=rnd(1, sh["cell"], 0.5, 1.0), eps_old=rnd(2, sh["cell"], 0.5, 1.0))
    if with_fs:
        kw["fs"] = tuple(rnd(3 + i, sh[k]) for i, k in enumerate("xyz"))
    g = DeviceGrid.from_case(case)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    if with_eps:
        g.void_fraction_, g.void_fraction_old_ = dev(kw["eps"]), dev(kw["eps_old"])
    if with_fs:
        g.f_sx_, g.f_sy_, g.f_sz_ = map(dev, kw["fs"])
    s = B200PressureSolver(N, case.h)
    s.set_coefficients(g)
    s.divergence(g, case.dt)
    rg = ref_grid(case, **kw)
    assert np.array_equal(W.interior(g.rhs_.cpu().numpy()), W.interior(O.make_rhs(rg)))
    pd, p = rnd(9, sh["cell"]), rnd(10, sh["cell"])
    g.p_delta_.copy_(dev(pd))
    g.p_.copy_(dev(p))
    s.correct(g, case.dt, zero_p_delta=False)
    want = O.correct(rg, pd, p=p.copy())
    for got, v, t in zip((g.f_vx_, g.f_vy_, g.f_vz_), want, (case.fxt, case.fyt, case.fzt)):
        m = t == W.F_INTERIOR
        assert np.array_equal(got.cpu().numpy()[m], v[m])
        assert np.all(got.cpu().numpy()[~m] == 0.0)
    assert np.array_equal(g.p_.cpu().numpy(), want[3])


@pytest.mark.parametrize("N", SIZES)
def test_surface_tension_bit_exact_over_depths(N):
    for kind in ("random", "sphere"):
        n, h, alpha, ct, sigma = W.surface_case(N, seed=6, kind=kind, solid_fraction=0.1)
        work = [rnd(900 + k, W.shapes(n)["cell"]) for k in range(5)]
        for k, a, b in zip(ST_KEYS, run_surface(n, h, alpha, ct, sigma, work),
                           O.surface_tension(n, h, alpha, ct, sigma, *work)):
            assert np.array_equal(a, b), k


@pytest.mark.parametrize("N", [(33, 9, 1479), (33, 9, 1480), (33, 9, 1481),    # below eight waves of blocks, from them on
                               (65, 5, 1975), (2, 2, 65537)])                  # beyond a launch's planes
def test_surface_tension_bit_exact_with_two_planes(N):
    n, h, alpha, ct, sigma = W.surface_case(N, seed=6, kind="random", solid_fraction=0.1 if min(N) > 4 else 0.0)
    work = [rnd(900 + k, W.shapes(n)["cell"]) for k in range(5)]
    for k, a, b in zip(ST_KEYS, run_surface(n, h, alpha, ct, sigma, work),
                       O.surface_tension(n, h, alpha, ct, sigma, *work)):
        assert np.array_equal(a, b), k


@pytest.mark.parametrize("N", SIZES)
def test_imported_operator_with_solids(N):
    """The operator of masked coefficients (solids, faces that are not F_INTERIOR, Dirichlet walls) against numpy;
    each row sums seven products in another order: 8 roundings of at most the row's terms."""
    c = W.post_case(N, seed=3, h=(0.5, 0.25, 0.125), solid_fraction=0.2 if min(N) > 4 else 0.0, solid_margin=1)
    sh = W.shapes(N)
    fb = [rnd(20 + i, sh[k], 0.1, 1.0) for i, k in enumerate("xyz")]   # walls and masked faces hold values too
    x = rnd(30, sh["cell"])
    s = B200PressureSolver(N, c.h)
    g = DeviceGrid.from_case(W.plain_case(N=N))
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    g.f_bx_, g.f_by_, g.f_bz_ = map(dev, fb)
    g.celltype_ = dev(c.ct)
    g.f_xtype_, g.f_ytype_, g.f_ztype_ = map(dev, c.ft)
    s.set_coefficients(g)
    y = torch.zeros(sh["cell"], dtype=torch.float64, device="cuda")
    s.apply_A(dev(x), y)
    inside = W.interior(c.ct) == W.C_INTERIOR
    xi = W.interior(x)
    want, size = np.zeros_like(xi), np.zeros_like(xi)
    for f in range(3):
        ax, n = 2 - f, N[f]
        b = fb[f][1:-1, 1:-1, 1:-1]         # faces 1 .. n+1 of the interior rows
        t = c.ft[f][1:-1, 1:-1, 1:-1]
        b = np.moveaxis(b, ax, 0).copy()
        t, q, v = np.moveaxis(t, ax, 0), np.moveaxis(inside, ax, 0), np.moveaxis(xi, ax, 0)
        b[:-1][~q] = 0.0
        b[1:][~q] = 0.0
        b[1:-1][t[1:-1] != W.F_INTERIOR] = 0.0
        w = b * (1.0 / (c.h[f] * c.h[f]))
        pad = np.concatenate([np.zeros_like(v[:1]), v, np.zeros_like(v[:1])])
        y1 = w[:-1] * (v - pad[:-2]) + w[1:] * (v - pad[2:])
        want += np.moveaxis(y1, 0, ax)
        size += np.moveaxis(w[:-1] * (abs(v) + abs(pad[:-2])) + w[1:] * (abs(v) + abs(pad[2:])), 0, ax)
    assert np.all(np.abs(W.interior(y.cpu().numpy()) - want) <= 16 * np.finfo(float).eps * size + 1e-300)


def test_divergence_of_a_coupled_step_runs_near_the_plain_ones_bandwidth():
    """192^3, by the bytes each form must move per cell: u* in, rhs out twice, cell bits (41); void fractions (16) and
    surface tension with its f_b (48) besides. 1.09 of the plain form's rate; 0.85 with two planes per thread."""
    n = 192
    case = W.plain_case(n)
    g = DeviceGrid.from_case(case)
    stream = torch.cuda.Stream()
    s = B200PressureSolver(case.N, case.h, stream=stream)
    s.set_coefficients(g)
    us = {}
    for key, nbytes in (("plain", 41), ("coupled", 105)):
        if key == "coupled":
            g.void_fraction_, g.void_fraction_old_ = torch.rand_like(g.p_), torch.rand_like(g.p_)
            g.f_sx_, g.f_sy_, g.f_sz_ = (torch.rand_like(v) for v in (g.f_vx_, g.f_vy_, g.f_vz_))
            torch.cuda.synchronize()
        us[key] = _device_us(lambda: s.divergence(g, 1.0), stream) / nbytes
    print(f"divergence 192^3: {41 * us['plain']:.1f} us, with everything {105 * us['coupled']:.1f} us")
    assert us["coupled"] <= us["plain"] / 0.9


def test_surface_tension_of_a_small_grid_takes_one_plane_per_thread():
    """32^3, against the one-load kernel of the pressure gradient: 5 times its device time; 6.5 and more with two
    planes per thread, whose chains of loads run one after the other on a grid of one wave."""
    n, h, alpha, ct, sigma = W.surface_case((32, 32, 32), seed=6, kind="sphere")
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    a, c = dev(alpha), dev(ct)
    work = [torch.zeros_like(a) for _ in range(5)]
    faces = [torch.zeros(W.shapes(n)[k], dtype=torch.float64, device="cuda") for k in "xyz"]
    us = _device_us(lambda: surface_tension_device(n, h, a, c, sigma, work, faces))
    gradp = _device_us(lambda: face_gradp_device(n, h, a, faces))
    print(f"surface tension 32^3: {us:.1f} us, pressure gradient {gradp:.1f} us")
    assert us <= 6.1 * gradp
