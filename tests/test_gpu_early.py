"""Searches limited to their first iterations, which merge in a cluster above 600
positions, on both sides of that rule: sizes, limits, both widths and loop modes,
alternating with unlimited runs of the same solver; and limited batches.  Whole
numbers: exact equality with the oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _same(got_tour, got, want_tour, want):
    assert np.array_equal(got_tour, want_tour)
    assert all(got[k] == want[k] for k in ("cost", "iterations", "moves", "evals"))


@pytest.mark.parametrize("n", [400, 599, 600, 601, 1200])
@pytest.mark.parametrize("wide", [False, True])
def test_limits(mlpgpu_mod, n, wide):
    x, y = (oracle.clustered_instance if n % 2 else oracle.uniform_instance)(n, n)
    D = oracle.dist(x, y, True)
    t = oracle.random_perm_tour(n, n)
    s = mlpgpu_mod.Solver(mlpgpu_mod.Problem.from_coords(x, y), wide=wide)
    at = (n + 1) // 12
    want = {cap: oracle.dvnd(t, D, wide, max_iters=cap, threads=8) for cap in (3, at, at + 1)}
    for unroll in (0, 4):
        s.set_unroll(unroll)
        for cap in (at, at + 1, 3, at, at + 1):
            s.set_tour(t)
            st = s.dvnd(max_iters=cap)
            _same(s.tour(), st, *want[cap])
    s.set_unroll(0)
    for cap in (at, at + 1):  # begun, then enqueued in two parts
        s.set_tour(t)
        s.begin(31, cap)
        s.enqueue(5)
        s.enqueue(cap)
        _same(s.tour(), s.stats(), *want[cap])
        s.set_tour(t)
        s.dvnd_async(31, cap)
        _same(s.tour(), s.stats(), *want[cap])


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("sizes", [(700, 90, 300), (1300, 1200), (5, 6, 130, 64)])
def test_batches(mlpgpu_mod, sizes, wide):
    b, inst = mlpgpu_mod.Batch(wide=wide), []
    for q, n in enumerate(sizes):
        x, y = oracle.uniform_instance(n, q)
        t = oracle.random_perm_tour(n, q)
        b.add(mlpgpu_mod.Problem.from_coords(x, y), t)
        inst.append((t, oracle.dist(x, y, True)))
    at = sum(n + 1 for n in sizes) // (12 * len(sizes))
    want = {cap: [oracle.dvnd(t, D, wide, max_iters=cap, threads=8) for t, D in inst] for cap in (at, at + 1, 2)}
    for shape in (-1, 10, 11, 12, 13):
        if shape >= 0:
            b.set_tile_shape(shape)
        for cap in (at, at + 1, 2):
            b.reset()
            b.run(max_iters=cap)
            for q, w in enumerate(want[cap]):
                _same(*b.result(q), *w)
