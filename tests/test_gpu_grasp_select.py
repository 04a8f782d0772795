"""The constructor's selection from unsorted rows (k_grasp_select), which serves
where no rows are ordered: at the edges of its 32-at-a-time draws, of its
shared-memory candidates (n = 2048 / 2049) and of alpha, beside starts of the
other kinds in one call.  Whole numbers: exact equality with the oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SEEDS = [0, 9, 4294967295]


@pytest.mark.parametrize("n", [5, 6, 32, 33, 34, 65, 625, 1000, 2048, 2049, 2500])
def test_selection(mlpgpu_mod, n):
    x, y = oracle.clustered_instance(n, n)  # many equal distances
    D = oracle.dist(x, y, True)
    p = mlpgpu_mod.Problem.from_coords(x, y)
    p.set_start_rows(2)
    for alpha in (0.0, 0.1, 0.5, 1.0):
        tours = p.random_tours(SEEDS, alpha)
        p.set_start_rows(1)
        assert np.array_equal(tours, p.random_tours(SEEDS, alpha)), alpha
        p.set_start_rows(2)
        if n <= 1000 or alpha in (0.1, 1.0):
            for q, sd in enumerate(SEEDS):
                assert np.array_equal(tours[q], oracle.random_tour_canonical(D, sd, alpha)), (sd, alpha)


def test_largest_distances(mlpgpu_mod):
    """Keys of 16-bit distances: all three digits of the radix selection, and ties."""
    for n, lo in ((40, 65530), (300, 0)):
        r = np.random.default_rng(n)
        D = np.triu(r.integers(lo, 65536, (n, n)), 1).astype(np.int32)
        D = D + D.T
        p = mlpgpu_mod.Problem.from_matrix(D)
        for mode in (1, 2):
            p.set_start_rows(mode)
            tours = p.random_tours(SEEDS, 0.6)
            for q, sd in enumerate(SEEDS):
                assert np.array_equal(tours[q], oracle.random_tour_canonical(D, sd, 0.6)), (n, mode, sd)


def test_kinds_in_one_call(mlpgpu_mod):
    b, want = mlpgpu_mod.Batch(), []
    for q, n in enumerate((70, 33, 120, 50, 9)):
        x, y = oracle.uniform_instance(n, q)
        D = oracle.dist(x, y, True)
        p = mlpgpu_mod.Problem.from_coords(x, y)
        p.set_start_rows(q % 3)
        for k, ties in enumerate((0, 1, 0)):
            b.add_random(p, 10 * q + k, 0.4, ties=ties)
            t = (oracle.random_tour if ties else oracle.random_tour_canonical)(D, 10 * q + k, 0.4)
            want.append(oracle.dvnd(t, D))
    b.run()
    for j, (t, st) in enumerate(want):
        bt, bst = b.result(j)
        assert np.array_equal(bt, t) and bst["cost"] == st["cost"], j


@pytest.mark.parametrize("matrices", [740, 800, 1250])
def test_many_matrices(mlpgpu_mod, matrices):
    """Either side of the rule between ordered rows and selection (one start a matrix)."""
    n, b, want = 24, mlpgpu_mod.Batch(), []
    for q in range(matrices):
        x, y = oracle.uniform_instance(n, q)
        b.add_random(mlpgpu_mod.Problem.from_coords(x, y), q, 0.5)
        if q % 97 == 0:
            D = oracle.dist(x, y, True)
            want.append((q, *oracle.dvnd(oracle.random_tour_canonical(D, q, 0.5), D)))
    b.run()
    for q, t, st in want:
        bt, bst = b.result(q)
        assert np.array_equal(bt, t) and bst["cost"] == st["cost"]
