"""The smoothed bound's node roots use only the list entries within reach of the
root, read from lists sorted by cost; the candidate search collects the first N
neighbours with one sort.  Every branch of that against the FP64 oracle, which
sums whole lists: hubs (lists past the sorted slices and the local sorts), ties
past the collection buffer, N above 32, temperatures at which whole lists are
within reach, the smallest instances, and one near the largest size, where
little scratch is left."""
import numpy as np
import pytest

from f2m_b200 import synth

pytestmark = pytest.mark.gpu


def _hub():
    """A centre that every point of six tight clusters of 24 has as its 24th neighbour."""
    a = np.repeat(np.arange(6), 24) * (np.pi / 3)
    r = 1e-3 * synth.uniform(1, 1, 144)
    t = 2 * np.pi * synth.uniform(1, 2, 144)
    x = np.concatenate([[0.0], np.cos(a) + r * np.cos(t)])
    y = np.concatenate([[0.0], np.sin(a) + r * np.sin(t)])
    return x.astype(np.float32), y.astype(np.float32)


def _repeats():
    """80 copies of one point among 120 others."""
    x, y = synth.config4(3, 200)
    x[:80], y[:80] = x[0], y[0]
    return x, y


CASES = {
    "hub": (_hub, 24, 1e-2, 30),
    "repeats": (_repeats, 12, 1e-2, 20),
    "n40": (lambda: synth.config4(5, 400), 40, 1e-3, 20),
    "warm": (lambda: synth.jittered_lattice(300, 6), 24, 5e-2, 30),
    "hot": (lambda: synth.config4(7, 300), 30, 0.5, 20),
    "four": (lambda: synth.config4(8, 4), 3, 1e-2, 10),
    "five": (lambda: synth.config4(9, 5), 8, 1e-3, 10),
    "n33": (lambda: synth.config4(10, 33), 32, 1e-3, 20),
    "n257": (lambda: synth.jittered_lattice(257, 11), 8, 1e-3, 20),
    "large": (lambda: synth.config4(12, 13500), 8, 1e-3, 3),
}


@pytest.mark.parametrize("solver", [1, 2])
@pytest.mark.parametrize("name", sorted(CASES))
def test_bound_and_gradient_match_oracle(ctx, oracle, name, solver):
    import f2m_b200
    make, N, tau, iters = CASES[name]
    x, y = make()
    p = f2m_b200.default_smooth_params(tau=tau, iters=iters, checkpoint=7, solver=solver)
    offs = np.array([0, len(x)], np.int64)
    L, gx, gy = ctx.smoothed_bound(offs, x, y, N, params=p, grad=True)
    Lo, dx, dy, _ = oracle.smooth_bound(x, y, N, tau=tau, iters=iters, grad=True)
    assert abs(L[0] - Lo) <= 1e-9 * abs(Lo)
    scale = max(np.abs(dx).max(), np.abs(dy).max())
    assert np.abs(gx - dx).max() <= 1e-5 * scale
    assert np.abs(gy - dy).max() <= 1e-5 * scale
    again = ctx.smoothed_bound(offs, x, y, N, params=p, grad=True)
    assert again[0][0] == L[0] and np.array_equal(again[1], gx) and np.array_equal(again[2], gy)
