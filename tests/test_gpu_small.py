"""The one-launch search of a small instance (mlp_small.cu) against the oracle:
sizes with fewer tiles than CTAs, at the edges of its 32-diagonal tiles, at the
change from resident distances to copied rows (n = 222 / 223), at its largest
size and just past it, in both widths, with and without a sweep limit.  Whole
numbers: exact equality."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _check(s, D, tour, wide, cap=1 << 20):
    s.set_tour(tour)
    st = s.dvnd(max_iters=cap)
    ot, ost = oracle.dvnd(tour, D, wide, max_iters=cap)
    assert np.array_equal(s.tour(), ot)
    assert all(st[k] == ost[k] for k in ("cost", "iterations", "moves", "evals"))
    # The arrays that later calls read are those of the final tour.
    assert np.array_equal(s.weights(), oracle.weights(ot, D))
    c, i, j = s.eval(3)
    oc, oi, oj, _ = oracle.eval_nb(3, ot, D, wide)
    assert np.array_equal(c, oc) and np.array_equal(i, oi) and np.array_equal(j, oj)


@pytest.mark.parametrize("n", [5, 6, 8, 33, 34, 35, 66, 129, 222, 223, 226, 383, 384, 385])
@pytest.mark.parametrize("wide", [False, True])
def test_small_search(mlpgpu_mod, n, wide):
    gen = oracle.clustered_instance if n % 2 else oracle.uniform_instance
    x, y = gen(n, n)
    D = oracle.dist(x, y, True)
    s = mlpgpu_mod.Solver(mlpgpu_mod.Problem.from_coords(x, y), wide=wide)
    _check(s, D, oracle.random_perm_tour(n, n), wide)
    _check(s, D, oracle.random_perm_tour(n, n + 1), wide, cap=1)
    _check(s, D, oracle.random_perm_tour(n, n + 2), wide, cap=3)


@pytest.mark.parametrize("n,top", [(60, 65535), (230, 65535), (100, 210000 // 100)])
@pytest.mark.parametrize("wide", [False, True])
def test_small_search_matrix(mlpgpu_mod, n, top, wide):
    """Symmetric matrices without a metric, up to the largest distances: 32-bit
    costs wrap as the reference's, and 64-bit ones that may leave 32 bits take
    the 64-bit kernels."""
    r = np.random.default_rng(n + top)
    D = np.triu(r.integers(0, top + 1, (n, n)), 1).astype(np.int32)
    D = D + D.T
    s = mlpgpu_mod.Solver(mlpgpu_mod.Problem.from_matrix(D), wide=wide)
    _check(s, D, oracle.random_perm_tour(n, 3), wide, cap=40)
