"""The forms of the cross-regression kernels against the oracle: the fixed row
layouts of sparsities 2 and 4 and the general one, one and two output rows
per reconstruction thread with a last odd row, and operands outside the fast
quotients' range (the repeated window)."""
import numpy as np
import pytest
import torch

from gpu_util import N, T, frames
from helpers import assert_close
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
ATOL = 1e-5   # the op's floor, as in test_gpu_regression.py


def compare(cd, x, win, sp, rs):
    o = cd.ops.cross_regression(*[T(a) for a in x], win_size=win, sparsity=sp, recon_scale=rs)
    torch.cuda.synchronize()
    for a, r, nm in zip(o, orc.cross_regression(*x, win, sp, rs), ("outa", "outb", "vara", "varb")):
        assert_close(N(a), r, nm, atol=ATOL)


def images(cd, H, W, seed):
    _, f = frames(cd, H, W, seed=seed)
    return [np.log1p(f["color"]), np.log1p(f["color2"]), f["albedo"], f["normal"]]


@pytest.mark.parametrize("H,W,win,sp,rs", [
    (44, 132, 19, 4, 1), (60, 64, 21, 4, 1),      # sparsity 4: the fixed layout's widest window, the general one
    (46, 130, 19, 2, 1), (50, 66, 21, 2, 2),      # sparsity 2, likewise
    (39, 33, 9, 3, 1), (45, 63, 5, 1, 1),         # odd row counts, one and two records per row
    (36, 60, 19, 4, 4), (60, 60, 13, 1, 1),       # nine output rows; one row per thread
])
def test_forms(cd, cuda, H, W, win, sp, rs):
    compare(cd, images(cd, H, W, seed=H + win), win, sp, rs)


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("image", [0, 1])
def test_out_of_range_pixel(cd, cuda, value, image):
    x = images(cd, 64, 96, seed=7)
    x[image][0, 30, 41, 1] = value
    compare(cd, x, 9, 4, 1)


@pytest.mark.parametrize("H,W,win,sp", [(48, 160, 9, 4), (32, 96, 9, 2), (30, 96, 7, 3)])
@pytest.mark.parametrize("value", [np.inf, np.nan, 1e25])
def test_fast_quotients_equal_divisions(cd, cuda, H, W, win, sp, value):
    """A pixel near the left edge makes its CTAs repeat their windows with
    IEEE divisions: every output it does not reach stays the same bit for bit."""
    x = images(cd, H, W, seed=9)
    run = lambda: [N(t) for t in cd.ops.cross_regression(*[T(a) for a in x], win_size=win, sparsity=sp)]
    clean = run()
    x[0][0, H // 2, 1, 0] = value
    far = 2 + 2 * (win // 2) + sp   # past the variance, the windows and the reconstruction
    for a, b in zip(run(), clean):
        np.testing.assert_array_equal(a[:, :, far + 1:], b[:, :, far + 1:])
