"""The one-launch search's forms against the oracle: clusters of 16 and 8 CTAs
and the iterated kernels in its place, around the size where the distances leave
shared memory (n = 223 / 224) and the largest sizes of both clusters (n = 384, and
366 with 8 CTAs); and a wait that runs out."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 6, 34, 68, 222, 223, 224, 225, 300, 366, 367, 384, 385])
@pytest.mark.parametrize("wide", [False, True])
def test_forms(mlpgpu_mod, n, wide):
    x, y = (oracle.clustered_instance if n % 2 else oracle.uniform_instance)(n, n)
    D = oracle.dist(x, y, True)
    t = oracle.random_perm_tour(n, n)
    p = mlpgpu_mod.Problem.from_coords(x, y)
    for cap in (1 << 20, 2):
        ot, ost = oracle.dvnd(t, D, wide, max_iters=cap)
        for ctas in (0, 16, 8, -1):
            s = mlpgpu_mod.Solver(p, wide=wide)
            s.set_small_search(ctas)
            s.set_tour(t)
            st = s.dvnd(max_iters=cap)
            assert np.array_equal(s.tour(), ot), ctas
            assert all(st[k] == ost[k] for k in ("cost", "iterations", "moves", "evals")), ctas
            assert np.array_equal(s.weights(), oracle.weights(ot, D)), ctas


@pytest.mark.parametrize("n", [224, 300, 384])
@pytest.mark.parametrize("ctas", [0, 8])
def test_wait_that_runs_out(mlpgpu_mod, n, ctas):
    """No poll at all: the search reports the rows as missing and ends at once;
    its copies land while it still holds the memory, and the device goes on."""
    x, y = oracle.uniform_instance(n, n)
    t = oracle.random_perm_tour(n, n)
    p = mlpgpu_mod.Problem.from_coords(x, y)
    s = mlpgpu_mod.Solver(p)
    s.set_small_search(ctas, 0)
    s.set_tour(t)
    if ctas == 8 and n > 366:  # the iterated kernels, which wait for no copies
        s.dvnd()
    else:
        with pytest.raises(mlpgpu_mod.MLPError, match="did not arrive"):
            s.dvnd()
        assert sorted(s.tour()[1:-1]) == list(range(1, n))
    s = mlpgpu_mod.Solver(p)
    s.set_small_search(ctas)
    s.set_tour(t)
    st = s.dvnd()
    ot, ost = oracle.dvnd(t, oracle.dist(x, y, True))
    assert np.array_equal(s.tour(), ot) and st["cost"] == ost["cost"]


def test_resident_search_waits_for_nothing(mlpgpu_mod):
    x, y = oracle.uniform_instance(223, 1)
    t = oracle.random_perm_tour(223, 1)
    s = mlpgpu_mod.Solver(mlpgpu_mod.Problem.from_coords(x, y))
    s.set_small_search(0, 0)
    s.set_tour(t)
    s.dvnd()
    assert np.array_equal(s.tour(), oracle.dvnd(t, oracle.dist(x, y, True))[0])
    for bad in ((1, -1), (32, -1), (0, -2)):
        with pytest.raises(mlpgpu_mod.MLPError):
            s.set_small_search(*bad)
