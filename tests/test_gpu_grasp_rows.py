"""The constructor over ordered rows (k_grasp_sort, k_grasp) at its edges: sort
sizes around powers of two, rows around one group of 256 clients, and a batch of
instances of several sizes in one call.  Whole numbers: exact equality with the
oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 33, 64, 65, 255, 256, 257, 512, 513, 1024, 1025, 2048, 2049])
def test_rows(mlpgpu_mod, n):
    x, y = oracle.clustered_instance(n, n)  # many equal distances
    D = oracle.dist(x, y, True)
    p = mlpgpu_mod.Problem.from_coords(x, y)
    for alpha in (0.02, 1.0):
        tours = p.random_tours([n, 5], alpha)
        for q, sd in enumerate((n, 5)):
            assert np.array_equal(tours[q], oracle.random_tour_canonical(D, sd, alpha)), (sd, alpha)


def test_batch_of_sizes(mlpgpu_mod):
    b, want = mlpgpu_mod.Batch(), []
    for q, n in enumerate((40, 7, 300, 129, 64)):
        x, y = oracle.uniform_instance(n, q)
        D = oracle.dist(x, y, True)
        p = mlpgpu_mod.Problem.from_coords(x, y)
        for sd in (q, q + 100):
            b.add_random(p, sd, 0.4)
            want.append(oracle.dvnd(oracle.random_tour_canonical(D, sd, 0.4), D))
    b.run()
    for j, (t, st) in enumerate(want):
        bt, bst = b.result(j)
        assert np.array_equal(bt, t) and bst["cost"] == st["cost"]
