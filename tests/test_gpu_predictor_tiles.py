"""The predictor's tiles: regular faces by side differences, the others by the boundary rules."""
import numpy as np
import pytest

from mydemcfd_b200 import workloads as W
from oracle import oracle as O
from test_gpu_post import run_predict

pytestmark = pytest.mark.gpu


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
