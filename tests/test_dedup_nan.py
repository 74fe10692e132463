"""A point with a NaN coordinate equals no point (get_KXY's comparison, FXY.hpp:
252-267): it is never dropped as a repeat, however many share its bits, and the
instance is then refused, as no neighbour lies within any radius of it."""
import numpy as np
import pytest

import f2m_b200
from f2m_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nans", [(300, 6), (300, 297), (3000, 1500), (20000, 10000)])
def test_nan_points_are_never_repeats(ctx, n, nans):
    x, y = synth.uniform_int_points(n, 40 + n)
    x[10:10 + nans // 2] = np.nan
    y[10 + nans // 3:10 + nans] = np.nan  # a third with one of each, a sixth with both
    x[5], y[5] = x[3], y[3]  # one repeat
    bad = np.isnan(x) | np.isnan(y)
    distinct = len(np.unique(np.stack([x[~bad], y[~bad]]), axis=1).T) + int(bad.sum())
    r = ctx.knn(x, y, 6)
    assert r.n_nodes == distinct and r.n_edges == 0
    with pytest.raises(f2m_b200.F2MError) as e:
        ctx.solve_points(x, y, 6)
    assert e.value.status == f2m_b200.ERR_CAPACITY


def test_nan_instance_of_a_batch_leaves_the_others_alone(ctx):
    parts = [synth.uniform_int_points(n, n) for n in (200, 300, 250)]
    offs = np.array([0, 200, 500, 750])
    x, y = (np.concatenate(p) for p in zip(*parts))
    lp, st = ctx.solve_batch(offs, x, y, 8)
    x[200:350] = np.nan
    lp2, st2 = ctx.solve_batch(offs, x, y, 8)
    assert list(st2) == [0, f2m_b200.ERR_CAPACITY, 0] and list(st) == [0, 0, 0]
    assert lp2[0] == lp[0] and lp2[2] == lp[2]
