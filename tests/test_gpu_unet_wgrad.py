"""The weight gradients of the U-Net's 3x3 layers at the edges of their
tiles (single-pixel images, 128-pixel column edges, partial row bands), with
two producers sharing a tile's copies, and the whole backward, whose layers'
partial sums are reduced in one launch, at small and ragged frames, with a
gradient through alpha only (the band's 1 / (p^2 + 1e-4) has a derivative of
up to 1e6 near p = 0, where bf16 activations alone move the gradient by 10 %).
Tolerances of test_gpu_unet.py: 2e-3 of max for a layer's fp32 sums, 3e-2 of
max per tensor for the whole network."""
import numpy as np
import pytest
import torch

from oracle import unet_torch as ut
from test_gpu_unet import DEV, bf16, close_to_max, frame_inputs, rand_act, reference, well_conditioned_net

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(1, 1, 1), (1, 2, 129), (3, 17, 128), (1, 200, 257), (2, 96, 1300)])
@pytest.mark.parametrize("cin,cout", [(8, 8), (15, 8), (24, 8), (8, 16), (16, 16), (48, 16), (16, 32), (32, 32),
                                      (48, 32), (32, 8)])
def test_layer(cd, cuda, B, H, W, cin, cout):
    g = torch.Generator().manual_seed(H * W + cin + 5 * cout)
    x = bf16(rand_act(B, H, W, cin, g))
    dz = bf16(torch.randn((B, H, W, cout), generator=g))
    dW, db, ws = cd.unet.conv3x3_wgrad(x.to(DEV, torch.bfloat16), dz.to(DEV, torch.bfloat16), cin, cout)
    torch.cuda.synchronize()
    assert ws[:4].view(torch.int32).item() == 0
    K = torch.zeros((3, 3, cin, cout), requires_grad=True)
    b = torch.zeros((cout,), requires_grad=True)
    out = ut.conv3x3(x[..., :cin].permute(0, 3, 1, 2).double(), K.double(), b.double(), relu=False)
    out.backward(dz.permute(0, 3, 1, 2).double())
    close_to_max(dW.cpu(), K.grad.float(), 2e-3, f"wgrad {cin}->{cout}")
    close_to_max(db.cpu(), b.grad.float(), 2e-3, f"bgrad {cin}->{cout}")


@pytest.mark.parametrize("B,H,W", [(1, 4, 4), (1, 20, 132), (2, 8, 516)])
def test_network(cd, cuda, B, H, W):
    ins = frame_inputs(B, H, W, 3 * H + W)
    net = well_conditioned_net(cd, 6)
    g = torch.Generator().manual_seed(H)
    gb, ga = torch.zeros((B, H, W, 5)), torch.randn((B, H, W, 1), generator=g)
    net(*[t.to(DEV) for t in ins])
    grads = net.backward(gb.to(DEV), ga.to(DEV)).cpu().clone().double()
    torch.cuda.synchronize()
    assert net.error_flag() == 0
    ref = reference(net.params, ins, True, gb, ga)
    o = 0
    for i, shape in enumerate(cd.unet.param_shapes()):
        n = int(np.prod(shape))
        close_to_max(grads[o:o + n], ref[o:o + n], 3e-2, f"param tensor {i} {shape}")
        o += n


@pytest.mark.parametrize("B,H,W", [(1, 4, 4), (1, 8, 12), (3, 4, 260), (1, 132, 520)])
def test_unaligned_gradients(cd, cuda, B, H, W):
    """Output gradients 4 bytes past a 16-byte boundary take the head
    backward's 4-byte copies: the same parameter gradients bit for bit, also
    where the last 32 pixels are not all there."""
    ins = [t.to(DEV) for t in frame_inputs(B, H, W, H + 7 * W)]
    g = torch.Generator().manual_seed(W)
    gb, ga = torch.randn((B, H, W, 5), generator=g).to(DEV), torch.randn((B, H, W, 1), generator=g).to(DEV)

    def shifted(t):
        v = torch.empty(t.numel() + 1, device=DEV)[1:].view(t.shape)
        return v.copy_(t)

    net = well_conditioned_net(cd, 3)
    net(*ins)
    want = net.backward(gb, ga).clone()
    got = net.backward(shifted(gb), shifted(ga)).clone()
    torch.cuda.synchronize()
    assert net.error_flag() == 0
    assert torch.equal(got, want)
