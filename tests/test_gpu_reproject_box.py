"""Reproject's normal test near and away from its threshold
|n - n'| / (fwidthN + 1e-2) > 4, which squares decide outside a margin of
1e-4, and its 3x3 box under a previous opacity full of holes: success masks
equal to the oracle's (which takes the root and divides), outputs within 1e-4."""
import numpy as np
import pytest

from helpers import assert_close, assert_equal
from oracle import oracle as orc
from test_gpu_reproject import KEYS, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fwN", [0.0, 0.37, -0.005, -0.0095, 3e5, 1e7, 1e25, np.inf, np.nan])
def test_normal_ratio(cd, cuda, fwN):
    rng = np.random.default_rng(5)
    B, H, W = 1, 40, 64
    S = float(np.float32(fwN)) + 1e-2
    S = S if np.isfinite(S) else 1.0
    rel = rng.choice([-0.5, -2e-4, -1.01e-4, -0.99e-4, -1e-6, -1e-7, 0.0, 1e-7, 1e-6, 0.99e-4, 1.01e-4, 2e-4, 0.5],
                     (B, H, W))
    n = np.zeros((B, H, W, 3), np.float32)
    n[..., 2] = 4.0 * S * (1.0 + rel)
    n[0, 0, :3, 2] = np.inf, np.nan, -np.inf
    pn = np.zeros((B, H, W, 3), np.float32)
    pnf = np.zeros((B, H, W, 3), np.float32)
    pnf[..., 1] = fwN
    z = np.zeros((B, H, W, 3), np.float32)
    d = dict(mvec=np.zeros((B, H, W, 3), np.float32), linear_z=z, prev_linear_z=z, normal=n, prev_normal=pn,
             pn_fwidth=pnf, opacity=np.ones((B, H, W, 1), np.float32), prev_opacity=np.ones((B, H, W, 1), np.float32))
    lists = [rng.uniform(0, 1, (B, H, W, 3)).astype(np.float32) for _ in range(3)]
    s, _ = run(cd, d, lists)
    rs, _ = orc.reproject(d["mvec"], lists, *[d[k] for k in KEYS[1:]])
    assert_equal(s, rs, f"success, fwidthN {fwN}")


@pytest.mark.parametrize("H,W,B", [(1, 1, 1), (5, 33, 2), (37, 53, 2)])
@pytest.mark.parametrize("n_list", [1, 3])
def test_box_with_holes(cd, cuda, H, W, B, n_list):
    rng = np.random.default_rng(H + W + n_list)
    u = lambda *c: rng.uniform(0, 1, (B, H, W) + c).astype(np.float32)  # noqa: E731
    mv = (rng.uniform(-2, 2, (B, H, W, 3)) / np.array([W, H, 1])).astype(np.float32)
    nrm = lambda: (np.array([0, 0, 1]) + 0.03 * rng.standard_normal((B, H, W, 3))).astype(np.float32)  # noqa: E731
    d = dict(mvec=mv, linear_z=u(3), prev_linear_z=u(3) * 3, normal=nrm(), prev_normal=nrm(), pn_fwidth=0.01 * u(3),
             opacity=(u(1) > 0.1).astype(np.float32), prev_opacity=(u(1) > 0.8).astype(np.float32))
    d["linear_z"][..., 1] *= 0.1
    lists = [u(3) for _ in range(n_list)]
    s, outs = run(cd, d, lists)
    rs, routs = orc.reproject(d["mvec"], lists, *[d[k] for k in KEYS[1:]])
    assert_equal(s, rs, "success")
    for i in range(n_list):
        assert_close(outs[i], routs[i], f"out{i}")
