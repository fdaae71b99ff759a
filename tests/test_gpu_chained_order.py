"""Operators queued one behind the other, each reading what the one before has
just written: the chained launches give the same bits as the same calls with
the device idle in between."""
import pytest
import torch

from gpu_util import T, frames

pytestmark = pytest.mark.gpu


def chain(cd, x, band, mask, settle):
    o = cd.ops
    out = []
    a, b, alb, nrm = x
    for _ in range(3):
        y1, y2 = o.prepare_input(a.abs() + 0.1, b.abs() + 0.1)
        settle()
        r1, r2, va, vb = o.cross_regression(y1, y2, alb, nrm, win_size=9, sparsity=4)
        settle()
        s1, s2, w1, w2 = o.spatial_filter(r1, r2, alb, nrm, band, win_size=7)
        settle()
        g = o.spatial_filter_grad(s1, s2, w1, w2, r1, r2, alb, nrm, band, win_size=7)
        settle()
        ero = o.erode3x3(mask)
        settle()
        p0, p1, p2, ok = o.temporal_screening(r1, r2, s1, s1, s2, ero, 5, 3)
        settle()
        q0, q1, q2, ok2, ero2 = o.erode_temporal_screening(p1, p2, r1, r1, r2, mask, 7, 1)
        settle()
        a, b = q1, q2
        out += [y1, y2, r1, r2, va, vb, s1, s2, w1, w2, g, ero, p0, p1, p2, ok, q0, q1, q2, ok2, ero2]
    return out


@pytest.mark.parametrize("H,W", [(64, 96), (256, 256), (180, 332)])
def test_queued_equals_settled(cd, cuda, H, W):
    _, f = frames(cd, H, W, seed=H)
    x = [T(f[k]) for k in ("color", "color2", "albedo", "normal")]
    g = torch.Generator().manual_seed(W)
    band = cd.synth.random_band((1, H, W), g).cuda()
    mask = (torch.rand((1, H, W, 1), generator=g) < 0.97).cuda()
    settled = chain(cd, x, band, mask, torch.cuda.synchronize)
    for _ in range(5):
        queued = chain(cd, x, band, mask, lambda: None)
        for i, (a, b) in enumerate(zip(queued, settled)):
            assert torch.equal(a, b), i


@pytest.mark.parametrize("H,W", [(64, 96), (256, 256)])
def test_training_pass(cd, cuda, H, W):
    """Forward, backward and update, queued: the same parameters as settled."""
    _, f = frames(cd, H, W, seed=2)
    ins = [T(f[k]) for k in ("color", "color2", "color", "albedo", "normal")]
    gb, ga = torch.full((1, H, W, 5), 1e-4, device="cuda"), torch.full((1, H, W, 1), 1e-3, device="cuda")
    nets = []
    for settle in (torch.cuda.synchronize, lambda: None):
        u = cd.unet.UNet(seed=5)
        for _ in range(4):
            u.forward(*ins)
            settle()
            u.backward(gb, ga)
            settle()
            u.apply_gradients()
            settle()
        torch.cuda.synchronize()
        nets.append(u)
    assert torch.equal(nets[0].params, nets[1].params) and torch.equal(nets[0].grads, nets[1].grads)
