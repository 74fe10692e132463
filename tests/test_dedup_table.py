"""De-duplication of the rounded points on the device (get_KXY, FXY.hpp:252-267):
the first of equal points is kept, in input order, at sizes around a chunk of 256
points and on large inputs, with heavy repetition, signed zeros and labels."""
import numpy as np
import pytest

import f2m_b200
from f2m_b200 import synth

pytestmark = pytest.mark.gpu


def _first_occurrences(x, y):
    rx, ry = np.round(x * 1000) / 1000 + 0.0, np.round(y * 1000) / 1000 + 0.0
    _, first = np.unique(np.stack([rx, ry]), axis=1, return_index=True)
    return np.sort(first)


@pytest.mark.parametrize("n,repeat", [(255, 0.3), (257, 0.9), (5000, 0.5), (20000, 0.2), (20000, 0.99)])
def test_first_of_equal_points_is_kept(ctx, oracle, n, repeat):
    x, y = synth.uniform_int_points(n, 900 + n, box=3000)
    k = int(n * repeat)  # the tail repeats points of the head, within the rounding
    src = (synth.uniform(n, 5, k) * (n - k)).astype(np.int64)
    x[n - k:], y[n - k:] = x[src] + 0.0004, y[src]
    x[0], y[0] = -0.0, 7.0
    x[n - 1], y[n - 1] = 0.0, 7.0
    labels = (np.arange(n) * 3 + 10).astype(np.int32)
    keep = _first_occurrences(x, y)
    r = ctx.knn(x, y, 6, labels=labels)
    assert r.n_nodes == len(keep)
    assert np.array_equal(r.label, labels[keep])
    o = oracle.build_graph(x[keep], y[keep], 6)
    assert np.array_equal(r.Do, o.Do)
    assert np.array_equal(r.v1, o.v1) and np.array_equal(r.v2, o.v2)


@pytest.mark.parametrize("n", [100, 2501, 5000, 20000])
def test_all_points_equal_is_an_input_error(ctx, n):
    """On one SM and on the whole GPU, which must leave an instance without a
    graph alone."""
    with pytest.raises(f2m_b200.F2MError) as e:
        ctx.solve_points(np.full(n, 3.0), np.full(n, 4.0), 8)
    assert e.value.status == f2m_b200.ERR_INPUT
