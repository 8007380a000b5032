"""The predictor's two forms: one thread per face on small grids; on larger ones tiles of regular faces by side
differences and the others by the boundary rules."""
import numpy as np
import pytest
import torch

from mydemcfd_b200 import workloads as W
from mydemcfd_b200.solver import BoundaryConditions, face_gradp_device, predict_vstar_device
from oracle import oracle as O
from test_gpu_post import _cuda, _momentum_fields, run_predict

pytestmark = pytest.mark.gpu
# device time of the predictor over that of the pressure gradient's kernel: 7.4 at 20^3 and 6.6 at 32^3 (9.7 and
# 11.9 us); 14.7 and more where a march takes these grids
BOUND = 10.5


@pytest.mark.parametrize("two_way", [False, True])
@pytest.mark.parametrize("N, solid", [
    ((30, 7, 9), 0.0),       # faces 1..N+1 fill a tile of 31 x 8 and a chunk of 10 planes
    ((31, 8, 10), 0.0),      # one more in each direction
    ((61, 15, 19), 0.0),     # two of each, and one more
    ((62, 16, 20), 0.1),     # with solids
    ((93, 33, 31), 0.02),    # chunks whose types are all interior beside chunks with solids
    ((4, 4, 4), 0.0),        # the smallest grid the march takes; no face is regular
    ((5, 6, 40), 0.0),
    ((3, 70, 5), 0.0),       # below it
    ((2, 3, 33), 0.0),
])
def test_predictor_bit_exact_over_tile_edges(N, solid, two_way):
    m = W.momentum_case(N, seed=7 + N[0], sides=("x+", "y-", "z+"), solid_fraction=solid, two_way=two_way)
    for k, a, b in zip("xyz", run_predict(m), O.predict_vstar(m)):
        assert np.array_equal(a, b), k


@pytest.mark.parametrize("two_way", [False, True])
@pytest.mark.parametrize("N, solid", [
    ((30, 110, 123), 0.02),  # the last grid of one thread per face, by warps (148 SMs)
    ((30, 111, 123), 0.02),  # the first one that is marched
    ((30, 127, 119), 0.0),   # faces 1..N+1 fill tiles of 31 x 8 and chunks of 10 planes
    ((31, 160, 130), 0.0),   # one more in x and y
    ((61, 88, 79), 0.0),     # two tiles of 31
    ((62, 103, 90), 0.1),    # three, with solids
    ((93, 71, 79), 0.02),    # chunks whose types are all interior beside chunks with solids
    ((4, 115, 121), 0.0),    # the thinnest grids that are marched
    ((740, 4, 121), 0.0),
    ((240, 351, 4), 0.0),
    ((3, 115, 121), 0.0),    # thinner: one thread per face at any size,
    ((2, 3, 21842), 0.0),    # up to the planes that a launch holds,
    ((2, 3, 21844), 0.0),    # and from the queue beyond them
])
def test_marched_predictor_bit_exact_over_tile_edges(N, solid, two_way):
    m = W.momentum_case(N, seed=7 + N[0], sides=("x+", "y-", "z+"), solid_fraction=solid, two_way=two_way)
    for k, a, b in zip("xyz", run_predict(m), O.predict_vstar(m)):
        assert np.array_equal(a, b), k


def _device_us(fn, stream=None):
    """Device time of one call of 20 in a graph."""
    stream = stream or torch.cuda.Stream()
    with torch.cuda.stream(stream):
        fn()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            for _ in range(20):
                fn()
        best = float("inf")
        for _ in range(10):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            graph.replay()
            e1.record()
            e1.synchronize()
            best = min(best, e0.elapsed_time(e1) / 20 * 1e3)
    return best


@pytest.mark.parametrize("n", [20, 32])
def test_predictor_of_a_small_grid_takes_one_chain_of_loads(n):
    """A grid of at most two waves of faces costs about one face's chain of loads, BOUND times the one-load kernel
    of the pressure gradient; a march of it costs that per plane of a chunk and pass of a queue."""
    m = W.momentum_case((n, n, n), seed=3)
    vs, gp = [_cuda(a) for a in m.vs], [_cuda(np.zeros_like(a)) for a in m.vs]
    bc, fields, p = BoundaryConditions(m.bc_type, *m.bc_v), _momentum_fields(m), _cuda(m.p)
    predict = _device_us(lambda: predict_vstar_device(m.N, m.h, bc, fields, m.dt, m.g, vs))
    gradp = _device_us(lambda: face_gradp_device(m.N, m.h, p, gp))
    print(f"{n}^3: predictor {predict:.1f} us, pressure gradient {gradp:.1f} us")
    assert predict <= BOUND * gradp
