"""The merges on both sides of the rule that chooses among them: one search
around its largest tour (2,000 positions) and around the largest that the
one-CTA merge's memory would take, sets around their limit (1,094 positions)
and between it and the sizes of other tests, recorded moves, both widths.
Whole numbers: exact equality with the oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cap", [(1155, 12), (1919, 6), (1998, 8), (1999, 8), (2000, 8), (2001, 8), (2047, 6), (2113, 6),
                                   (2114, 6), (2115, 6)])
@pytest.mark.parametrize("wide", [False, True])
def test_one_search(mlpgpu_mod, n, cap, wide):
    x, y = (oracle.clustered_instance if n % 2 else oracle.uniform_instance)(n, n)
    D = oracle.dist(x, y, True)
    t = oracle.random_perm_tour(n, n)
    s = mlpgpu_mod.Solver(mlpgpu_mod.Problem.from_coords(x, y), wide=wide)
    s.set_tour(t)
    st = s.dvnd(max_iters=cap)
    ot, ost = oracle.dvnd(t, D, wide, max_iters=cap, threads=8)
    assert np.array_equal(s.tour(), ot)
    assert all(st[k] == ost[k] for k in ("cost", "iterations", "moves", "evals"))
    assert np.array_equal(s.weights(), oracle.weights(ot, D))
    for nb in (0, 1, 4):
        cost, moves = s.pass_(nb)
        ot, oc, om = oracle.pass_(nb, ot, D, wide)
        assert cost == oc and moves == om and np.array_equal(s.tour(), ot)


@pytest.mark.parametrize("top", [1092, 1093, 1094])
@pytest.mark.parametrize("jobs", [3, 18])
@pytest.mark.parametrize("wide", [False, True])
def test_set(mlpgpu_mod, top, jobs, wide):
    sizes = [top] + [730 + 19 * q for q in range(jobs - 1)]
    b, want = mlpgpu_mod.Batch(wide=wide), []
    for q, n in enumerate(sizes):
        x, y = (oracle.clustered_instance if q % 2 else oracle.uniform_instance)(n, q)
        t = oracle.random_perm_tour(n, q)
        b.add(mlpgpu_mod.Problem.from_coords(x, y), t)
        want.append(oracle.dvnd(t, oracle.dist(x, y, True), wide, max_iters=10, threads=8) if q < 6 else None)
    b.run(max_iters=10)
    for q, w in enumerate(want):
        if w is None:
            continue
        bt, bst = b.result(q)
        assert np.array_equal(bt, w[0]), sizes[q]
        assert all(bst[k] == w[1][k] for k in ("cost", "iterations", "moves", "evals"))
