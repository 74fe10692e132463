"""Sizes that run on the whole GPU for speed alone (2,501 to 10,000 points) solve
on one SM when a grid barrier wait runs out, as they did before they moved; a
call that asks for the whole GPU still fails.  A limit of one poll lets the first
CTA to arrive give up, and every CTA leaves the solve: no fault, no trap."""
import numpy as np
import pytest

import f2m_b200
from f2m_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", ["uniform", "lattice"])
def test_automatic_choice_falls_back_to_one_sm(ctx, tmp_path, shape):
    n = 3000
    x, y = synth.uniform_int_points(n, 31) if shape == "uniform" else synth.lattice_points(n, 31, keep=0.3)
    short = f2m_b200.default_params(grid_spin_limit=1)
    one = f2m_b200.default_params(solver=1)
    r, t = ctx.solve_points(x, y, 10, params=short), ctx.solve_points(x, y, 10, params=one)
    assert r.status == t.status == 0 and r.lp == t.lp
    assert np.array_equal(r.F, t.F) and np.array_equal(r.x, t.x)
    offs = np.array([0, n])
    a, b = (ctx.solve_batch(offs, x, y, 10, params=p) for p in (short, one))
    assert a[1][0] == 0 and a[0][0] == b[0][0]
    import torch
    dev = [torch.from_numpy(q).cuda() for q in (offs.astype(np.int64), x, y)]
    lp = torch.zeros(1, dtype=torch.float64, device="cuda")
    st = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    ctx.solve_batch_device(offs, *(q.data_ptr() for q in dev), 10, lp.data_ptr(), st.data_ptr(), short)
    ctx.sync()
    assert int(st) == 0 and float(lp) == b[0][0]
    path = str(tmp_path / "a.tsp")
    synth.write_tsplib(path, x, y)
    r, t = ctx.solve_file(path, 10, params=short), ctx.solve_file(path, 10, params=one)
    assert r.status == t.status == 0 and np.array_equal(r.F, t.F)


def test_whole_gpu_by_request_still_fails(ctx):
    x, y = synth.uniform_int_points(3000, 31)
    with pytest.raises(f2m_b200.F2MError) as e:
        ctx.solve_points(x, y, 10, params=f2m_b200.default_params(solver=2, grid_spin_limit=1))
    assert e.value.status == f2m_b200.ERR_CUDA
