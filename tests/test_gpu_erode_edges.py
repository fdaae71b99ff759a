"""The erosion at image edges and in images of one to three rows or columns,
against a minimum over the window's pixels inside the image."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(1, 1, 1), (2, 1, 5), (1, 7, 1), (1, 2, 2), (3, 3, 33), (1, 8, 32), (2, 9, 65), (1, 40, 130)])
@pytest.mark.parametrize("density", [0.5, 0.95, 1.0])
def test_window_minimum(cd, cuda, B, H, W, density):
    g = torch.Generator().manual_seed(H * 1000 + W)
    m = torch.rand((B, H, W, 1), generator=g) < density
    padded = torch.ones((B, H + 2, W + 2, 1), dtype=torch.bool)
    padded[:, 1:-1, 1:-1] = m
    want = torch.ones_like(m)
    for dy in range(3):
        for dx in range(3):
            want &= padded[:, dy:dy + H, dx:dx + W]
    assert torch.equal(cd.ops.erode3x3(m.cuda()).cpu(), want.float())
