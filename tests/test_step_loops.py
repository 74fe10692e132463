"""The step loops of the team solver hold a warp's slices in registers where
they fit and read the rest from the SELL arrays; which loop runs follows from
the instance's size, the team's width and the list lengths.  The potentials
must equal the oracle's bit for bit in every one of them."""
import numpy as np
import pytest

import f2m_b200
from f2m_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 32, 33, 129, 1025, 2049, 4097, 8161, 8200])
def test_potentials_at_slice_edges(ctx, oracle, n):
    """Around whole slices, one slice a warp, four slices a warp, and the last
    size whose offsets fit 16 bits (8,160)."""
    x, y = synth.uniform_int_points(n, 500 + n)
    o = oracle.solve_points(x, y, 12, threads=8)
    r = ctx.solve_points(x, y, 12)
    assert r.status == o.status
    assert np.array_equal(r.F, o.F)


@pytest.mark.parametrize("bounds", [[4, 5, 6], [4, 5, 3000], [4, 2500, 4000], [700, 2000, 5000]])
def test_potentials_do_not_depend_on_the_team(ctx, oracle, bounds):
    """One to eight slices a warp, with four- to eight-entry and
    longer first slices (the lattice's lists)."""
    start = f2m_b200.get_class_bounds()
    try:
        f2m_b200.set_class_bounds(bounds)
        for (x, y), N in [(synth.uniform_int_points(2000, 9), 16), (synth.lattice_points(700, 5, keep=0.3), 10)]:
            o = oracle.solve_points(x, y, N)
            r = ctx.solve_points(x, y, N)
            assert r.status == o.status
            assert np.array_equal(r.F, o.F)
    finally:
        f2m_b200.set_class_bounds(start)


@pytest.mark.parametrize("scale", [2.0 ** -600, 2.0 ** -400, 1.0])
def test_costs_outside_the_short_forms_range(ctx, oracle, scale):
    """Costs below 1e-150 take the reference's chain step by step."""
    x, y = synth.uniform_int_points(300, 17)
    g = oracle.build_graph(x, y, 10)
    o = oracle.solve_graph(g.n_nodes, g.v1, g.v2, g.D * scale, g.Do, label=g.label)
    r = ctx.solve_graph(g.n_nodes, g.v1, g.v2, g.D * scale, g.Do, labels=g.label)
    assert r.status == o.status
    assert np.array_equal(r.F, o.F)


@pytest.mark.parametrize("solver", [0, 1])
@pytest.mark.parametrize("n", [2500, 2501, 4097, 8161, 8200, 9999])
def test_potentials_on_one_sm_and_on_all(ctx, oracle, n, solver):
    """A single instance moves to the whole GPU above 2,500 points; solver = 1
    keeps it on one SM."""
    x, y = synth.uniform_int_points(n, 700 + n)
    o = oracle.solve_points(x, y, 10, threads=8)
    r = ctx.solve_points(x, y, 10, params=f2m_b200.default_params(solver=solver))
    assert r.status == o.status
    assert np.array_equal(r.F, o.F)
    lp, st = ctx.solve_batch(np.array([0, n]), x, y, 10, params=f2m_b200.default_params(solver=solver))
    assert st[0] == o.status and abs(lp[0] - o.lp) <= 1e-12 * o.lp


def test_largest_instance_of_a_class(ctx, oracle):
    """The largest instance a 128-thread team's share of shared memory holds: its
    last slice is cut short, so its potentials stay in node order."""
    start = f2m_b200.get_class_bounds()
    lo, hi = 4, 8000
    try:
        while lo < hi:
            mid = (lo + hi + 1) // 2
            try:
                f2m_b200.set_class_bounds([mid, mid + 1, mid + 2])
                lo = mid
            except f2m_b200.F2MError:
                hi = mid - 1
        f2m_b200.set_class_bounds([lo, lo + 1, lo + 2])
        x, y = synth.uniform_int_points(lo, 77)
        o = oracle.solve_points(x, y, 6)
        # enough instances that the call keeps the narrow teams; the others are small
        sizes = np.array([lo] * 4 + [8] * 700, np.int64)
        offs = np.concatenate([[0], np.cumsum(sizes)])
        sx, sy = synth.uniform_int_points(8, 78)
        X = np.concatenate([np.tile(x, 4), np.tile(sx, 700)])
        Y = np.concatenate([np.tile(y, 4), np.tile(sy, 700)])
        out = ctx.solve_batch(offs, X, Y, 6, details=True)
        assert np.all(out["status"] == 0)
        assert np.all(np.abs(out["lp"][:4] - o.lp) <= 1e-12 * o.lp)
    finally:
        f2m_b200.set_class_bounds(start)
