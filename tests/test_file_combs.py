"""Files whose combs need Ax=b (comb_thread.cpp:272-304) or the repair loop
(graph_cuda.cu:69-126): the host comb stage takes over from a solve on one SM,
where the device's own Ax=b does not run, as from one on the whole GPU."""
import numpy as np
import pytest

import f2m_b200
from f2m_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", [0, 1, 2])
@pytest.mark.parametrize("n,seed", [(700, 5), (1500, 3), (1500, 4)])
def test_file_with_irregular_combs(ctx, oracle, tmp_path, n, seed, solver):
    x, y = synth.lattice_points(n, seed, keep=0.3)
    path = str(tmp_path / "a.tsp")
    synth.write_tsplib(path, x, y)
    o = oracle.solve_file(path, 10)
    r = ctx.solve_file(path, 10, params=f2m_b200.default_params(solver=solver))
    assert r.stats["irr_a"] > 0
    assert r.status == o.status == 0
    assert np.array_equal(r.F, o.F)
    # Ax=b rows follow the host stage's order, as in the oracle: the LP values
    # differ by the rounding of their sums
    assert abs(r.lp - o.lp) <= 1e-9 * o.lp
