"""Band gradient of the spatial filter on both sides of the radius at which its
launch bound changes (three CTAs per SM below radius 3, in grids of more than 2 or 8 CTAs
per SM), against the oracle."""
import numpy as np
import pytest
import torch

from gpu_util import N, T, frames
from helpers import assert_close
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("win", [3, 5, 7])
@pytest.mark.parametrize("H,W,B", [(8, 32, 1), (41, 67, 2), (9, 33, 3), (41, 67, 25), (41, 67, 67)])
def test_gradient(cd, cuda, H, W, B, win):
    fs = [frames(cd, H, W, seed=win + b)[1] for b in range(min(B, 3))]
    cat = lambda k: np.concatenate([fs[b % len(fs)][k] for b in range(B)])
    band = cd.synth.random_band((B, H, W), torch.Generator().manual_seed(win)).numpy()
    x = [np.log1p(cat("color")), np.log1p(cat("color2")), cat("albedo"), cat("normal"), band]
    rng = np.random.default_rng(win)
    gs = [rng.normal(size=(B, H, W, c)).astype(np.float32) for c in (3, 3, 1, 1)]
    gb = cd.ops.spatial_filter_grad(*[T(a) for a in gs], *[T(a) for a in x], win_size=win)
    torch.cuda.synchronize()
    r = orc.spatial_filter(*x, win, partials=True)
    rg = orc.spatial_filter_grad_from_partials(*gs, r[4], r[5])
    assert_close(N(gb), rg, "grad_band", atol=1e-6 * np.abs(rg).max())   # as in test_gpu_spatial_filter.py
