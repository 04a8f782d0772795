"""The batch DVND sweep with two diagonals a thread against the oracle at the
edges of its tiles: sizes around multiples of their diagonals and rows, tours of
fewer rows than a tile, each of its tile shapes.  Whole numbers: exact equality."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SIZES = [5, 6, 7, 9, 15, 16, 17, 18, 19, 31, 33, 34, 35, 63, 64, 65, 66, 67, 80, 81, 127, 128, 129, 130, 131, 145, 200]


@pytest.mark.parametrize("shape", [10, 11, 12, 13])
def test_tile_edges(mlpgpu_mod, shape):
    b, want = mlpgpu_mod.Batch(), []
    b.set_tile_shape(shape)
    for q, n in enumerate(SIZES):
        x, y = (oracle.clustered_instance if q % 2 else oracle.uniform_instance)(n, q)
        t = oracle.random_perm_tour(n, q)
        b.add(mlpgpu_mod.Problem.from_coords(x, y), t)
        want.append(oracle.dvnd(t, oracle.dist(x, y, True)))
    b.run()
    for q, (tour, stats) in enumerate(want):
        t, st = b.result(q)
        assert np.array_equal(t, tour)
        assert all(st[k] == stats[k] for k in ("cost", "iterations", "moves", "evals"))
