"""The smoothed bound's automatic choice between one CTA an instance and a launch
a step follows the list entries within reach of a root, counted by the graph
build: warm temperatures, clusters far below the spacing of the bounding box, a
collinear largest instance and an outlier.  Every path that calls of many points
take (four or eight lanes a node, ragged instances) against the FP64 oracle."""
import numpy as np
import pytest

import f2m_b200
from f2m_b200 import synth

pytestmark = pytest.mark.gpu


def _clusters(n, seed, spread=0.1):
    k = max(2, n // 40)
    a = (synth.uniform(seed, 3, n) * k).astype(int)
    x = synth.uniform(seed, 1, k)[a] * 30 + spread * synth.normal(seed, 4, n)
    y = synth.uniform(seed, 2, k)[a] * 30 + spread * synth.normal(seed, 5, n)
    return x.astype(np.float32), y.astype(np.float32)


def _batch(make, sizes, seed):
    parts = [make(int(m), seed + b) for b, m in enumerate(sizes)]
    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    return offs, np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts])


def _check(ctx, oracle, offs, x, y, N, tau, iters, solver, sample):
    p = f2m_b200.default_smooth_params(tau=tau, iters=iters, checkpoint=7, solver=solver)
    L, gx, gy = ctx.smoothed_bound(offs, x, y, N, params=p, grad=True)
    for b in sample:
        s = slice(offs[b], offs[b + 1])
        Lo, dx, dy, _ = oracle.smooth_bound(x[s], y[s], N, tau=tau, iters=iters, grad=True)
        assert abs(L[b] - Lo) <= 1e-9 * abs(Lo)
        # at the coldest temperature here whole lists are saturated and the adjoint is
        # inf * 0 for entries that the sums over what is within reach leave out:
        # compared where the oracle has a value
        fx, fy = np.isfinite(dx), np.isfinite(dy)
        scale = max(np.abs(dx[fx]).max(), np.abs(dy[fy]).max())
        assert np.abs(gx[s][fx] - dx[fx]).max() <= 1e-5 * scale
        assert np.abs(gy[s][fy] - dy[fy]).max() <= 1e-5 * scale


def _many():
    import torch
    return 2 * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("make,tau,persistent", [
    (synth.jittered_lattice, 1e-3, True), (synth.jittered_lattice, 5e-2, False),
    (_clusters, 1e-5, True), (_clusters, 1e-2, False)])
def test_automatic_choice_follows_the_lists(ctx, oracle, make, tau, persistent):
    sizes = 40 + np.arange(_many()) % 53
    offs, x, y = _batch(make, sizes, 500)
    _check(ctx, oracle, offs, x, y, 12, tau, 20, 0, (0, 52, len(sizes) - 1))
    assert (ctx.smooth_work()[0] >= 0) == persistent


@pytest.mark.parametrize("odd", ["collinear", "outlier"])
def test_one_odd_instance_does_not_move_the_batch(ctx, oracle, odd):
    """Cold lattices, the largest instance collinear; warm ones, one point of the
    largest instance far away."""
    sizes = 40 + np.arange(_many()) % 20
    sizes[3] = 80
    offs, x, y = _batch(synth.jittered_lattice, sizes, 900)
    if odd == "collinear":
        y[offs[3]:offs[4]] = 1.0
    else:
        x[offs[3]] = 1e5
    _check(ctx, oracle, offs, x, y, 12, 1e-3 if odd == "collinear" else 5e-2, 10, 0, (0, 4, len(sizes) - 1))
    assert (ctx.smooth_work()[0] >= 0) == (odd == "collinear")


@pytest.mark.parametrize("make,N,tau", [(synth.jittered_lattice, 24, 1e-3), (synth.jittered_lattice, 12, 5e-2),
                                        (_clusters, 32, 1e-2), (_clusters, 24, 1e-4)])
def test_steps_over_many_points(ctx, oracle, make, N, tau):
    """More than 14,000 points in the call: four lanes a node, eight where lists
    within reach are long."""
    sizes = np.array([4, 5, 31, 32, 33, 7, 900, 1500, 2011, 64, 65] + [1100] * 10)
    offs, x, y = _batch(make, sizes, 700)
    assert offs[-1] > 14000
    _check(ctx, oracle, offs, x, y, N, tau, 20, 2, (0, 1, 2, 3, 4, 5, 6, 8, 10, len(sizes) - 1))
    _check(ctx, oracle, offs, x, y, N, tau, 20, 1, (0, 4, 7, len(sizes) - 1))


def test_terms_taken_are_those_within_reach(ctx):
    """Cold lattices have three or four of some 36 entries within reach; at a warm
    temperature whole lists are, and the reverse steps' second passes come on top."""
    offs, x, y = _batch(synth.jittered_lattice, [400, 500, 600], 40)
    taken = {}
    for tau in (1e-3, 0.5):
        p = f2m_b200.default_smooth_params(tau=tau, iters=10, solver=1)
        for grad in (False, True):
            ctx.smoothed_bound(offs, x, y, 24, params=p, grad=grad)
            taken[tau, grad] = ctx.smooth_taken() / ctx.smooth_work()[0]
    # (the bound itself takes every edge once, less than a tenth of what ten steps cover)
    assert 3 / 48 < taken[1e-3, False] < 0.25 and 3 / 48 < taken[1e-3, True] < 0.25
    assert taken[0.5, False] == 1.0 and taken[0.5, True] > 1.0
    ctx.smoothed_bound(offs, x, y, 24, params=f2m_b200.default_smooth_params(solver=2))
    assert ctx.smooth_taken() == -1
