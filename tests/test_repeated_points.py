"""Inputs with many repeated points: the solver that runs, the size class and the
buffers follow the distinct points (get_KXY drops the others before anything
else, FXY.hpp:252-267), in single calls and in a batch of one."""
import numpy as np
import pytest

import f2m_b200
from f2m_b200 import synth

pytestmark = pytest.mark.gpu


def _repeated(n, k, seed):
    """n points over k distinct ones; every distinct one occurs."""
    x, y = synth.uniform_int_points(k, seed, box=100_000)
    i = (synth.uniform(seed, 7, n) * k).astype(int)
    i[synth.splitmix64(np.arange(k) + seed).argsort()] = np.arange(k)
    return x[i], y[i]


@pytest.mark.parametrize("n,k", [(5000, 50), (2501, 2500), (5000, 2600), (20000, 200), (20000, 9000), (30000, 12000)])
def test_solve_of_repeated_points(ctx, oracle, n, k):
    x, y = _repeated(n, k, 60 + k)
    labels = (np.arange(n) * 2 + 5).astype(np.int32)
    o = oracle.solve_points(x, y, 8, K=labels, threads=8)
    r = ctx.solve_points(x, y, 8, labels=labels)
    assert r.status == o.status == 0
    assert np.array_equal(r.F, o.F) and np.array_equal(r.Do, o.Do)
    assert np.array_equal(r.lab1, o.lab1) and np.array_equal(r.lab2, o.lab2)
    if k <= 10000:
        lp, st = ctx.solve_batch(np.array([0, n]), x, y, 8)
        assert st[0] == 0 and abs(lp[0] - o.lp) <= 1e-9 * o.lp  # (Ax=b where a comb is irregular)


def test_buffers_follow_the_distinct_points():
    """200,000 inputs over 5,000 points: a stage of under 100 bytes an input, then
    the call of 5,000 points, where a call of 200,000 takes over 500 MB."""
    import torch
    n, k = 200_000, 5000
    x, y = _repeated(n, k, 11)
    torch.cuda.synchronize()
    c = f2m_b200.Context(0)
    try:
        small = c.solve_points(x[:300], y[:300], 12)  # the module and its pools
        free0 = torch.cuda.mem_get_info()[0]
        r = c.solve_points(x, y, 12)
        used = free0 - torch.cuda.mem_get_info()[0]
    finally:
        c.close()
    assert small.status == 0 and r.status == 0 and r.n_nodes == k
    assert used < 150e6
