"""The 64-bit DVND sweep (mlp_sweep_wide.cu) against the oracle: symmetric
matrices up to the largest distance, whose costs leave 32 bits, at sizes around
its tiles and in every tile shape; a 64-bit batch; and the bound at which one
search's costs still fit 32 bits.  Whole numbers: exact equality."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _matrix(n, top, seed=0):
    r = np.random.default_rng(1000 * n + seed)
    D = np.triu(r.integers(0, top + 1, (n, n)), 1).astype(np.int32)
    return D + D.T


def _same(s, D, t, cap):
    s.set_tour(t)
    st = s.dvnd(max_iters=cap)
    ot, ost = oracle.dvnd(t, D, True, max_iters=cap)
    assert np.array_equal(s.tour(), ot)
    assert all(st[k] == ost[k] for k in ("cost", "iterations", "moves", "evals"))


@pytest.mark.parametrize("n,shape", [(5, 3), (6, 7), (7, 0), (9, 4), (19, 7), (34, 1), (66, 3), (67, 7), (68, 6),
                                     (130, 7), (131, 4), (147, 12), (260, 2), (401, -1), (700, -1)])
def test_search(mlpgpu_mod, n, shape):
    D = _matrix(n, 65535)
    s = mlpgpu_mod.Solver(mlpgpu_mod.Problem.from_matrix(D), wide=True)
    s.set_merge_mode(1)  # two kernels an iteration at every size
    if shape >= 0:
        s.set_tile_shape(shape)
    _same(s, D, oracle.random_perm_tour(n, 1), 30)
    # An evaluation between searches uses the other tile list.
    t = s.tour()
    c, i, j = s.eval(2)
    oc, oi, oj, _ = oracle.eval_nb(2, t, D, True)
    assert np.array_equal(c, oc) and np.array_equal(i, oi) and np.array_equal(j, oj)
    _same(s, D, oracle.random_perm_tour(n, 2), 30)


@pytest.mark.parametrize("top", [1000, 65535])
def test_batch(mlpgpu_mod, top):
    b, want = mlpgpu_mod.Batch(wide=True), []
    for q, n in enumerate((8, 40, 77, 129, 300)):
        D = _matrix(n, top, q)
        t = oracle.random_perm_tour(n, q)
        b.add(mlpgpu_mod.Problem.from_matrix(D), t)
        want.append(oracle.dvnd(t, D, True))
    b.run()
    for q, (t, st) in enumerate(want):
        bt, bst = b.result(q)
        assert np.array_equal(bt, t) and bst["cost"] == st["cost"] and bst["moves"] == st["moves"]


@pytest.mark.parametrize("n", [300, 450])
@pytest.mark.parametrize("over", [0, 1])
def test_width_bound(mlpgpu_mod, n, over):
    """dmax * size^2 just within 2^31 - 1 (deltas taken in 32 bits) and just over."""
    top = (2**31 - 1) // (n + 1) ** 2 + over
    D = _matrix(n, top)
    D[0, 1] = D[1, 0] = top
    s = mlpgpu_mod.Solver(mlpgpu_mod.Problem.from_matrix(D), wide=True)
    _same(s, D, oracle.random_perm_tour(n, 3), 1 << 20)
