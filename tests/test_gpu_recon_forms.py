"""The three forms of the reconstruction kernel: two output rows per thread
(grids of two CTAs per SM and more, here a batch), and one, lean or unrolled
(few CTAs, few or many centres).  Every form gives the same bits, so a batch
equals its images run alone, and one of them the oracle."""
import numpy as np
import pytest
import torch

from gpu_util import N, T, frames
from helpers import assert_close
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,win,sp,rs", [
    (64, 96, 17, 4, 1), (44, 132, 9, 4, 1), (63, 66, 9, 3, 1),   # two rows: full tiles, partial ones, a last odd row
    (60, 132, 19, 4, 2), (30, 130, 5, 2, 1),
    (44, 132, 7, 4, 1), (46, 34, 1, 2, 1),                        # at most two centres a row: lean in both
    (40, 66, 5, 1, 1), (36, 96, 3, 1, 1), (40, 72, 9, 4, 4),      # many centres: unrolled alone, two rows where they fit
])
def test_batch_equals_single_images(cd, cuda, H, W, win, sp, rs):
    rows, cols = -(-(H // rs) // 8), -(-(W // rs) // 32)
    B = -(-2 * 2 * 148 // (rows * cols))   # twice the CTAs from which the two-row form is taken
    _, f = frames(cd, H, W, seed=H + W)
    x = [np.log1p(f["color"]), np.log1p(f["color2"]), f["albedo"], f["normal"]]
    gain = np.linspace(0.5, 1.5, B, dtype=np.float32)[:, None, None, None]
    big = [T(a * gain) if i < 2 else T(np.repeat(a, B, 0)) for i, a in enumerate(x)]
    run = lambda v: cd.ops.cross_regression(*v, win_size=win, sparsity=sp, recon_scale=rs)
    whole = run(big)
    for k in (0, B // 2, B - 1):
        for a, b in zip(whole, run([t[k:k + 1].contiguous() for t in big])):
            assert torch.equal(a[k:k + 1], b)
    one = [N(t[:1]) for t in big]
    for a, r, nm in zip(whole, orc.cross_regression(*one, win, sp, rs), ("outa", "outb", "vara", "varb")):
        assert_close(N(a[:1]), r, nm, atol=1e-5)   # the op's floor, as in test_gpu_regression.py
