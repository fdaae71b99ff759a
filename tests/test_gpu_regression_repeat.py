"""Cross-regression of frames with operands outside the fast quotients' range,
where the windows that reach them start again: what that may cost, and that
the sparsity's fixed and general row layouts agree with the oracle there."""
import numpy as np
import pytest
import torch

from gpu_util import N, T, frames
from helpers import assert_close
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def images(cd, H, W, seed):
    _, f = frames(cd, H, W, seed=seed)
    return [np.log1p(f["color"]), np.log1p(f["color2"]), f["albedo"], f["normal"]]


def elapsed(fn, n=10):
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    for _ in range(n):
        fn()
    b.record()
    torch.cuda.synchronize()
    return a.elapsed_time(b) / n


def test_non_finite_frame_costs_less_than_a_second_pass(cd, cuda):
    """Nearly every CTA starts again.  Two whole sweeps of a window in place
    of one, at the finite sweep's rate, would be 1.75 of the call (the sweep
    is two thirds of it, the second with selects); divisions on their slow
    path in the second were 2.46."""
    x = [T(a) for a in images(cd, 1080, 1920, seed=3)]
    bad = [t.clone() for t in x]
    i = torch.randperm(1080 * 1920, generator=torch.Generator().manual_seed(1))[:30000]
    bad[0].view(-1, 3)[i.to(bad[0].device)] = float("nan")
    run = lambda v: cd.ops.cross_regression(*v, win_size=17, sparsity=4)
    for v in (x, bad):
        run(v)
    torch.cuda.synchronize()
    clean, odd = [min(elapsed(lambda: run(v)) for _ in range(3)) for v in (x, bad)]
    assert odd < 2.0 * clean, (odd, clean)


@pytest.mark.parametrize("H,W,win,sp", [(44, 132, 17, 4), (46, 130, 9, 2), (48, 66, 9, 3), (40, 32, 1, 1)])
@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("y", [0, 21, -1])
def test_bad_pixel_in_any_row(cd, cuda, H, W, win, sp, value, y):
    """First, middle or last image row: the window starts again early, late, or
    with the bad row mirrored into it."""
    x = images(cd, H, W, seed=H)
    x[0][0, y, W // 3, 1] = value
    o = cd.ops.cross_regression(*[T(a) for a in x], win_size=win, sparsity=sp)
    torch.cuda.synchronize()
    for a, r, nm in zip(o, orc.cross_regression(*x, win, sp, 1), ("outa", "outb", "vara", "varb")):
        assert_close(N(a), r, nm, atol=1e-5)   # the op's floor, as in test_gpu_regression.py
