"""The one-CTA merge (mlp_merge_one.cu) against the oracle: sizes with one, two
and three positions a thread, its largest tour and just past it, lists of every
length (first iterations: all blocks improve; last ones: a few), both widths,
recorded moves, and batches of few and many searches.  Whole numbers: exact
equality."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cap", [(385, 1 << 20), (600, 1 << 20), (1022, 40), (1025, 40), (1700, 24), (2030, 10),
                                   (2045, 10), (2060, 10), (2120, 6)])
@pytest.mark.parametrize("wide", [False, True])
def test_search(mlpgpu_mod, n, cap, wide):
    gen = oracle.clustered_instance if n % 2 else oracle.uniform_instance
    x, y = gen(n, n)
    D = oracle.dist(x, y, True)
    t = oracle.random_perm_tour(n, n)
    s = mlpgpu_mod.Solver(mlpgpu_mod.Problem.from_coords(x, y), wide=wide)
    s.set_tour(t)
    s.set_unroll(8)  # two kernels an iteration, checked by the host
    st = s.dvnd(max_iters=cap)
    ot, ost = oracle.dvnd(t, D, wide, max_iters=cap, threads=8)
    assert np.array_equal(s.tour(), ot)
    assert all(st[k] == ost[k] for k in ("cost", "iterations", "moves", "evals"))
    assert np.array_equal(s.weights(), oracle.weights(ot, D))
    cost, moves = s.pass_(2)  # one neighbourhood, with its moves recorded
    ot, oc, om = oracle.pass_(2, ot, D, wide)
    assert cost == oc and moves == om and np.array_equal(s.tour(), ot)


@pytest.mark.parametrize("sizes", [(7, 400, 90), tuple(range(5, 45)) + (513, 700)])
@pytest.mark.parametrize("wide", [False, True])
def test_batch(mlpgpu_mod, sizes, wide):
    b, want = mlpgpu_mod.Batch(wide=wide), []
    for q, n in enumerate(sizes):
        x, y = oracle.clustered_instance(n, q)
        t = oracle.random_perm_tour(n, q)
        b.add(mlpgpu_mod.Problem.from_coords(x, y), t)
        want.append(oracle.dvnd(t, oracle.dist(x, y, True), wide))
    b.run()
    for q, (t, st) in enumerate(want):
        bt, bst = b.result(q)
        assert np.array_equal(bt, t)
        assert all(bst[k] == st[k] for k in ("cost", "iterations", "moves", "evals"))
