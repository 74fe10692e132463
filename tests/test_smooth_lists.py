"""The smoothed bound's union lists, sorted by a warp each: in registers up to 64
entries, in place above, hubs of hundreds of entries (coincident points) among
them.  Edges, their order and their costs equal the oracle's graph exactly."""
import numpy as np
import pytest

import f2m_b200
from f2m_b200 import synth

pytestmark = pytest.mark.gpu


def _clustered(n, seed):
    k = n // 40
    a = (synth.uniform(seed, 3, n) * k).astype(int)
    x = synth.uniform(seed, 1, k)[a] * 10 + 0.1 * synth.normal(seed, 4, n)
    y = synth.uniform(seed, 2, k)[a] * 10 + 0.1 * synth.normal(seed, 5, n)
    return x.astype(np.float32), y.astype(np.float32)


def _coincident(n, seed):
    x, y = synth.config4(seed, n)
    x[: n // 2], y[: n // 2] = x[0], y[0]
    return x, y


@pytest.mark.parametrize("make,n,N", [
    (_clustered, 400, 12), (_clustered, 400, 31), (_clustered, 400, 32), (_clustered, 500, 33),
    (_clustered, 700, 48), (_clustered, 700, 63), (_clustered, 700, 64), (synth.jittered_lattice, 300, 32),
    (_coincident, 300, 20), (_coincident, 600, 64), (synth.jittered_lattice, 40, 64)])
def test_lists_equal_the_oracles(ctx, oracle, make, n, N):
    x, y = make(n, 90 + N)
    row, nbr, c = oracle.smooth_graph(x, y, N)
    v = np.repeat(np.arange(n), np.diff(row))
    up = nbr > v
    offs = np.array([0, n], np.int64)
    for solver in (1, 2):
        p = f2m_b200.default_smooth_params(iters=2, solver=solver)
        ea, eb, ec, _ = ctx.smoothed_bound_edges(offs, x, y, N, params=p)[3]
        assert np.array_equal(ea, v[up]) and np.array_equal(eb, nbr[up])
        assert np.array_equal(ec, c[up])
