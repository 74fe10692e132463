"""Every team width of the batched solver against the oracle, bit for bit: how many
instances share a call and the class bounds decide which team an instance runs
on, how many slices its warps hold and which step loop runs."""
import numpy as np
import pytest

import f2m_b200
from f2m_b200 import synth

pytestmark = pytest.mark.gpu
N = 12


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.fixture(scope="module")
def instances(oracle):
    """Uniform and lattice instances around whole slices, up to eight-entry and longer
    first slices (the lattice's lists), with their oracle solutions."""
    pts = [synth.uniform_int_points(n, 300 + n) for n in (4, 31, 32, 33, 300, 448, 449, 1000, 1793, 2500)]
    pts += [synth.lattice_points(n, n, keep=0.3) for n in (150, 700, 1500)]
    return pts, [oracle.solve_points(x, y, N, threads=8) for x, y in pts]


def _call(instances, count):
    """The instances, and tiny ones up to `count`."""
    tiny = synth.uniform_int_points(8, 78)
    parts = instances[0] + [tiny] * (count - len(instances[0]))
    offs = np.concatenate([[0], np.cumsum([len(p[0]) for p in parts])]).astype(np.int64)
    return offs, np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts])


@pytest.mark.parametrize("per_sm,narrowest", [(0.5, 1024), (1.5, 512), (3, 256), (5, 128), (9, 128)])
@pytest.mark.parametrize("bounds", [None, [4, 5, 6], [4, 5, 2500], [4, 2500, 3000], [700, 2000, 3000]])
def test_potentials_equal_the_oracles_on_every_team(ctx, instances, per_sm, narrowest, bounds):
    start = f2m_b200.get_class_bounds()
    try:
        if bounds:
            f2m_b200.set_class_bounds(bounds)
        b = list(f2m_b200.get_class_bounds())
        count = int(per_sm * _sms())
        for x, _ in instances[0]:
            wanted = [w for m, w in zip(b, (128, 256, 512)) if len(x) <= m] + [1024]
            assert f2m_b200.team_width(len(x), count) == max(wanted[0], narrowest)
        offs, x, y = _call(instances, count)
        out = ctx.solve_batch(offs, x, y, N, details=True)
        F = ctx.batch_potentials(len(x))
    finally:
        f2m_b200.set_class_bounds(start)
    for i, o in enumerate(instances[1]):
        assert out["status"][i] == o.status
        # (an instance whose irregular combs went through the repair loop holds the
        # potentials of its last step, as the oracle's)
        assert np.array_equal(F[offs[i]:offs[i] + o.n_nodes], o.F), len(instances[0][i][0])


def test_lp_bits_do_not_depend_on_the_call(ctx, instances):
    """The LP value sums in the order of the team that the size asks for."""
    lps = []
    for per_sm in (0.5, 1.5, 3, 5, 9):
        offs, x, y = _call(instances, int(per_sm * _sms()))
        lps.append(ctx.solve_batch(offs, x, y, N)[0][:len(instances[0])])
    for lp in lps[1:]:
        assert np.array_equal(lp, lps[0], equal_nan=True)
    for i, (x, y) in enumerate(instances[0]):
        assert ctx.solve_batch(np.array([0, len(x)]), x, y, N)[0][0] == lps[0][i]
