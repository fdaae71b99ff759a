"""Every layer shape that the weight-gradient entry point accepts runs on the
persistent kernel: one partial row per CTA, 148 at most, however large the
image (the workspace query, no GPU)."""
import pytest


@pytest.mark.parametrize("cin", [8, 15, 16, 24, 32, 48])
@pytest.mark.parametrize("cout", [8, 16, 32])
def test_rows(cd, cin, cout):
    size = cd._lib.lib().cd_unet_conv3x3_wgrad_workspace_size
    row = 4 * (9 * cin * cout + cout)
    pad = lambda n: (n + 255) // 256 * 256
    assert size(cin, cout, 4, 4096, 4096) == 256 + pad(148 * row)
    assert size(cin, cout, 1, 1, 1) == 256 + pad(row)


def test_other_shapes_are_refused(cd):
    size = cd._lib.lib().cd_unet_conv3x3_wgrad_workspace_size
    for cin, cout in ((64, 8), (8, 24), (8, 48), (7, 8)):
        assert size(cin, cout, 1, 64, 64) == 0
