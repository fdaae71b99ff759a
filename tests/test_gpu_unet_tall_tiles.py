"""The persistent convolution's 8- and 6-row tiles at batches that the device's
SM count puts well inside their range (twice the tiles from which they are
taken, two per resident CTA), as layers, as a network with pooling, and
replayed from a captured graph: the bits of the per-tile kernel."""
import pytest
import torch

from test_gpu_unet import DEV, bf16, frame_inputs, rand_act, weights, well_conditioned_net
from test_gpu_unet_conv_tiles import on_off

pytestmark = pytest.mark.gpu


def batch(H, W, rows):
    """Images of H x W that make twice 4 tiles of `rows` x 128 pixels per SM."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles = -(-H // rows) * -(-W // 128)
    return -(-2 * 4 * sms // tiles)


@pytest.mark.parametrize("H,W", [(61, 130), (13, 128), (23, 257)])
@pytest.mark.parametrize("cin,cout,rows", [(8, 8, 8), (15, 8, 8), (16, 16, 8), (24, 8, 6)])
def test_layer(cd, cuda, H, W, cin, cout, rows):
    B = batch(H, W, rows)
    g = torch.Generator().manual_seed(H + W + cin + 3 * cout)
    x = bf16(rand_act(B, H, W, cin, g)).to(DEV, torch.bfloat16)
    w, b = [t.to(DEV) for t in weights(cin, cout, g)]

    def f():
        y, ws = cd.unet.conv3x3(w, b, x, cin, cout)
        torch.cuda.synchronize()
        assert ws[:4].view(torch.int32).item() == 0
        return y[..., :cout].clone()
    y, y0 = on_off(cd, f)
    assert torch.equal(y.view(torch.int16), y0.view(torch.int16))


def test_network_and_graph(cd, cuda):
    """Pooling at full and half resolution, both in tall tiles."""
    H, W = 44, 260
    B = batch(H // 2, W // 2, 8)
    ins = [t.to(DEV) for t in frame_inputs(B, H, W, 11)]
    net = well_conditioned_net(cd, 3)

    def f():
        out = [t.clone() for t in net(*ins)]
        torch.cuda.synchronize()
        assert net.error_flag() == 0
        return out
    tall, tile = on_off(cd, f)
    for a, b in zip(tall, tile):
        assert torch.equal(a, b)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        out = net(*ins)
    for t in out:
        t.zero_()
    graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(out, tall):
        assert torch.equal(a, b)
    assert net.error_flag() == 0
