"""A server step that needs two merge launches a sweep (one search too large for
the shared-memory merge beside small ones), where one group ends inside the
step: every search gives what it gives alone, on few and on many searches and
in both widths.  Whole numbers: exact equality."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _instance(n, seed):
    x, y = (oracle.clustered_instance if seed % 2 else oracle.uniform_instance)(n, seed)
    return x, y, oracle.random_perm_tour(n, seed)


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("smalls", [3, 20])
@pytest.mark.parametrize("large_limit,small_limit", [(24, 1), (24, 3), (2, 1 << 20), (11, 5)])
def test_one_group_ends_inside_a_step(mlpgpu_mod, wide, smalls, large_limit, small_limit):
    reqs = [(2200, large_limit), (1900, large_limit + 1)] + [(40 + 13 * q, small_limit) for q in range(smalls)]
    srv = mlpgpu_mod.Server(1 << 32, wide=wide, max_active=64)
    ids = []
    for q, (n, limit) in enumerate(reqs):
        x, y, t = _instance(n, q)
        ids.append(srv.submit(x, y, t, max_iters=limit))
    left, got = set(ids), {}
    for _ in range(1000):
        srv.step(8)
        for rid in srv.finished():
            got[rid] = srv.result(rid, reqs[ids.index(rid)][0])
            left.discard(rid)
        if not left:
            break
    assert not left
    for q, (n, limit) in enumerate(reqs):
        x, y, t = _instance(n, q)
        tour, st, info = got[ids[q]]
        if n < 1000:
            want, ws = oracle.dvnd(t, oracle.dist(x, y, True), wide, max_iters=limit)
        else:
            s = mlpgpu_mod.Solver(mlpgpu_mod.Problem.from_coords(x, y), wide=wide)
            s.set_tour(t)
            ws = s.dvnd(max_iters=limit)
            want = s.tour()
        assert info["status"] == 0 and np.array_equal(tour, want), (n, limit)
        assert all(st[k] == ws[k] for k in ("cost", "iterations", "moves", "evals")), (n, limit)
