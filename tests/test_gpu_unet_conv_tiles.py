"""The persistent convolution's tall tiles (8 and 6 output rows instead of 4,
taken in the forward pass once every resident CTA has two such tiles): the
same K steps into every output in the same order as the per-tile kernel, so
the same bits, at partial tiles in x and y, across images of a batch and with
infinities and NaN in the input; and the fused pooling and the whole network
through them."""
import pytest
import torch

from oracle import unet_torch as ut
from test_gpu_unet import DEV, bf16, close_to_max, frame_inputs, rand_act, weights, well_conditioned_net

pytestmark = pytest.mark.gpu


def on_off(cd, f):
    out = []
    L = cd._lib.lib()
    try:
        for on in (1, 0):
            L.cd_set_persistent_kernels(on)
            out.append(f())
            torch.cuda.synchronize()
    finally:
        L.cd_set_persistent_kernels(1)
    return out


@pytest.mark.parametrize("B,H,W", [(40, 61, 130), (300, 13, 128), (1, 2371, 300)])
@pytest.mark.parametrize("cin,cout", [(8, 8), (15, 8), (24, 8), (8, 16), (16, 16)])
def test_layer(cd, cuda, B, H, W, cin, cout):
    g = torch.Generator().manual_seed(H + W + cin + 3 * cout)
    x = bf16(rand_act(B, H, W, cin, g))
    w, b = weights(cin, cout, g)
    xd, wd, bd = x.to(DEV, torch.bfloat16), w.to(DEV), b.to(DEV)
    xs = xd.clone()
    xs[0, H // 2, 5, 1], xs[0, H - 1, W - 1, 0], xs[-1, 0, W // 2, 2] = float("inf"), float("nan"), -float("inf")
    for inp in (xd, xs):
        def f():
            y, ws = cd.unet.conv3x3(wd, bd, inp, cin, cout)
            torch.cuda.synchronize()
            assert ws[:4].view(torch.int32).item() == 0
            return y[..., :cout].clone()
        y, y0 = on_off(cd, f)
        assert torch.equal(y.view(torch.int16), y0.view(torch.int16)), "tall tiles differ from the per-tile kernel"
        if inp is xd:
            k = B - 1
            ref = ut.conv3x3(x[k:, ..., :cin].permute(0, 3, 1, 2), bf16(w), b).permute(0, 2, 3, 1)
            close_to_max(y[k:].float().cpu(), ref, 1e-2, f"conv {cin}->{cout}")


def test_network(cd, cuda):
    B, H, W = 20, 76, 260
    ins = [t.to(DEV) for t in frame_inputs(B, H, W, 11)]
    net = well_conditioned_net(cd, 3)
    g = torch.Generator().manual_seed(5)
    gb, ga = torch.randn((B, H, W, 5), generator=g).to(DEV), torch.randn((B, H, W, 1), generator=g).to(DEV)

    def f():
        band, alpha = net(*ins)
        out = [band.clone(), alpha.clone(), net.backward(gb, ga).clone()]
        torch.cuda.synchronize()
        assert net.error_flag() == 0
        return out
    for a, b in zip(*on_off(cd, f)):
        assert torch.equal(a, b)
