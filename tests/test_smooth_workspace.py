"""The smoothed bound's workspace a point stays within what whole lists took (80 N +
16 checkpoints + 8 per stored iterate + about 400 bytes with the gradient, 48 N + 240
without), whichever path runs and however many steps a segment holds."""
import numpy as np
import pytest

import f2m_b200
from f2m_b200 import synth

pytestmark = pytest.mark.gpu


def _batch(sizes):
    parts = [synth.jittered_lattice(int(m), 40 + b % 7) for b, m in enumerate(sizes)]
    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    return offs, np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts])


@pytest.mark.parametrize("solver", [0, 1, 2])
@pytest.mark.parametrize("size,count,N,ckpt,grad", [
    (900, 160, 24, 16, True), (900, 160, 64, 100, True), (33, 4000, 24, 16, True), (5, 20000, 4, 16, True),
    (900, 160, 24, 16, False), (33, 4000, 8, 16, False)])
def test_workspace_a_point(solver, size, count, N, ckpt, grad):
    import torch
    sizes = np.full(count, size)
    offs, x, y = _batch(sizes)
    iters = 100 if ckpt == 100 else 20
    p = f2m_b200.default_smooth_params(iters=iters, checkpoint=ckpt, solver=solver)
    c = f2m_b200.Context(0)
    try:
        c.smoothed_bound(offs[:9], x[:offs[8]], y[:offs[8]], N, params=p, grad=grad)  # the module and its pools
        torch.cuda.synchronize()
        free0 = torch.cuda.mem_get_info()[0]
        c.smoothed_bound(offs, x, y, N, params=p, grad=grad)
        used = free0 - torch.cuda.mem_get_info()[0]
    finally:
        c.close()
    n = int(offs[-1])
    a_point = 80 * N + 16 * ckpt + 8 * -(-iters // ckpt) + 400 if grad else 48 * N + 240
    a_point += 8 * (3 * iters + 4) / size + 64 / size  # per-instance values, a point
    # an eighth more is taken than asked for; allocations round up to 2 MB
    assert used <= 1.125 * a_point * n + (4 << 20)


def test_segment_length_does_not_change_results(ctx):
    x, y = synth.jittered_lattice(700, 3)
    offs = np.array([0, 300, 700], np.int64)
    for solver in (1, 2):
        out = [ctx.smoothed_bound(offs, x, y, 12, grad=True, params=f2m_b200.default_smooth_params(
            iters=90, checkpoint=k, solver=solver)) for k in (1, 7, 16, 60, 90, 1000)]
        for o in out[1:]:
            assert all(np.array_equal(a, b) for a, b in zip(out[0], o))
