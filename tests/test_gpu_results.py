"""Results read by one kernel into pinned memory (batch results, recorded
passes) and searches of a few iterations launched without the device-side loop,
against the oracle at the edges of their copies and of the rule."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,seed", [(5, 1), (511, 2), (513, 3)])
@pytest.mark.parametrize("wide", [False, True])
def test_recorded_pass_by_capacity(mlpgpu_mod, n, seed, wide):
    """The first min(moves, capacity) moves, none of a later one's left over."""
    x, y = oracle.clustered_instance(n, seed)
    t, D = oracle.random_perm_tour(n, seed), oracle.dist(x, y, True)
    s = mlpgpu_mod.Solver(mlpgpu_mod.Problem.from_coords(x, y), wide=wide)
    for nb in range(5):
        want_tour, want_cost, want = oracle.pass_(nb, t, D, wide)
        for cap in (1 << 15, 1, 3, 0):
            s.set_tour(t)
            cost, moves = s.pass_(nb, max_moves=cap)
            assert cost == want_cost and moves == want[:cap]
            assert np.array_equal(s.tour(), want_tour)


@pytest.mark.parametrize("n", [7, 255, 257, 700])
@pytest.mark.parametrize("wide", [False, True])
def test_candidates_leave_clean_keys(mlpgpu_mod, n, wide):
    """Evaluations in any order, each from reset keys; Or-opt-k passes by capacity."""
    x, y = oracle.clustered_instance(n, n)
    t, D = oracle.random_perm_tour(n, n), oracle.dist(x, y, True)
    s = mlpgpu_mod.Solver(mlpgpu_mod.Problem.from_coords(x, y), wide=wide)
    s.set_tour(t)
    for nb in (4, 0, 1, 0, 3, 2, 4):
        c, i, j = s.eval(nb)
        wc, wi, wj, _ = oracle.eval_nb(nb, t, D, wide)
        assert np.array_equal(c, wc) and np.array_equal(i, wi) and np.array_equal(j, wj)
    want_cost, want = s.pass_oropt(2)
    want_tour = s.tour()
    for cap in (0, 1, 1 << 15):
        s.set_tour(t)
        s.eval_oropt(2)
        cost, moves = s.pass_oropt(2, max_moves=cap)
        assert cost == want_cost == oracle.cost(want_tour, D, wide) and moves == want[:cap]
        assert np.array_equal(s.tour(), want_tour)
    want_tour, want = oracle.dvnd(want_tour, D, wide)
    s.dvnd()
    assert np.array_equal(s.tour(), want_tour)


@pytest.mark.parametrize("n", [5, 100, 420])
@pytest.mark.parametrize("iters", [1, 7, 8, 9])
def test_few_iterations(mlpgpu_mod, n, iters):
    """Either side of the limit below which the iterations are launched as such."""
    x, y = oracle.uniform_instance(n, n)
    t = oracle.random_perm_tour(n, n)
    s = mlpgpu_mod.Solver(mlpgpu_mod.Problem.from_coords(x, y))
    s.set_tour(t)
    st = s.dvnd(max_iters=iters)
    want_tour, want = oracle.dvnd(t, oracle.dist(x, y, True), False, max_iters=iters)
    assert np.array_equal(s.tour(), want_tour)
    assert all(st[k] == want[k] for k in ("cost", "iterations", "moves", "evals"))


def test_batch_results_in_any_order(mlpgpu_mod):
    sizes = [5, 6, 511, 512, 40]
    b, want = mlpgpu_mod.Batch(), []
    for q, n in enumerate(sizes):
        x, y = oracle.clustered_instance(n, q)
        t = oracle.random_perm_tour(n, q)
        b.add(mlpgpu_mod.Problem.from_coords(x, y), t)
        want.append(oracle.dvnd(t, oracle.dist(x, y, True)))
    b.run()
    for q in (2, 0, 4, 3, 1, 2):
        t, st = b.result(q)
        assert np.array_equal(t, want[q][0]) and st["cost"] == want[q][1]["cost"]


def test_batch_results_from_threads(mlpgpu_mod):
    from concurrent.futures import ThreadPoolExecutor

    b = mlpgpu_mod.Batch()
    for q in range(24):
        x, y = oracle.uniform_instance(30 + 17 * q, q)
        b.add(mlpgpu_mod.Problem.from_coords(x, y), oracle.random_perm_tour(30 + 17 * q, q))
    b.run()
    want = [b.result(q) for q in range(24)]
    with ThreadPoolExecutor(8) as pool:
        got = list(pool.map(lambda q: b.result(q % 24), range(960)))
    for q, (t, st) in enumerate(got):
        assert np.array_equal(t, want[q % 24][0]) and st == want[q % 24][1]


@pytest.mark.parametrize("n", [52, 420])
@pytest.mark.parametrize("wide", [False, True])
def test_under_stream_capture(mlpgpu_mod, n, wide):
    """A capturing stream takes the reset and the sweep, and refuses a search, a
    pass and a change of the mask, after which the solver works as before."""
    torch = pytest.importorskip("torch")
    x, y = oracle.uniform_instance(n, n)
    t = oracle.random_perm_tour(n, n)
    s = mlpgpu_mod.Solver(mlpgpu_mod.Problem.from_coords(x, y), wide=wide)
    s.set_tour(t)
    stream = torch.cuda.Stream()
    assert mlpgpu_mod.lib().mlp_solver_set_stream(s._h, stream.cuda_stream) == 0
    calls = [(lambda: s.begin(31, 5), True), (lambda: s.sweep(31, 1), True), (lambda: s.dvnd_async(31, 20), False),
             (lambda: s.dvnd_async(31, 2), False), (lambda: s.pass_(1), False), (lambda: s.begin(1, 5), False)]
    for call, taken in calls:
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(stream):
            graph.capture_begin(capture_error_mode="thread_local")
            try:
                if taken:
                    call()
                else:
                    with pytest.raises(Exception):
                        call()
            finally:
                graph.capture_end()
        s.set_tour(t)
        want_tour, _ = oracle.dvnd(t, oracle.dist(x, y, True), wide)
        s.dvnd()
        assert np.array_equal(s.tour(), want_tour)
        s.set_tour(t)
