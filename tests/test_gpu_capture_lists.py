"""Sweeps on a capturing stream after (and during) switches of the sweep kernel
and the candidate mode, on a 64-bit solver whose costs leave 32 bits: the
captured graphs replay, and searches afterwards equal the oracle's."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,shape", [(60, 0), (420, -1), (420, 5)])
@pytest.mark.parametrize("before,inside", [((), None), ((0,), None), ((), 0), ((0,), 1), ((0, 1), None)])
@pytest.mark.parametrize("total", [False, True])
def test_sweep_kernels_under_capture(mlpgpu_mod, n, shape, before, inside, total):
    torch = pytest.importorskip("torch")
    r = np.random.default_rng(n)
    D = np.triu(r.integers(0, 65536, (n, n)), 1).astype(np.int32)
    D = D + D.T
    t = oracle.random_perm_tour(n, n)
    s = mlpgpu_mod.Solver(mlpgpu_mod.Problem.from_matrix(D), wide=True)
    if shape >= 0:
        s.set_tile_shape(shape)
    s.set_tour(t)
    stream = torch.cuda.Stream()
    assert mlpgpu_mod.lib().mlp_solver_set_stream(s._h, stream.cuda_stream) == 0
    if total:
        s.set_total(True)
    for variant in before:
        s.set_sweep_kernel(variant)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="thread_local")
        try:
            if inside is not None:  # no search ran yet: there is no graph to drop during the capture
                s.set_sweep_kernel(inside)
            s.sweep(31, 2)
        finally:
            graph.capture_end()
        graph.replay()
    torch.cuda.synchronize()
    if total:
        s.set_total(False)
    want_tour, want = oracle.dvnd(t, D, True, max_iters=12)
    s.set_tour(t)
    st = s.dvnd(max_iters=12)
    assert np.array_equal(s.tour(), want_tour)
    assert all(st[k] == want[k] for k in ("cost", "iterations", "moves", "evals"))
