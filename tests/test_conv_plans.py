"""How a convolution runs (operand by TMA or gathered, tile width, K slices): asked of the native plan, on the host."""
import pytest

from ronn_b200 import _native

WORKSPACE = 1 << 22                                        # fp32 values that the provider hands over


def plan(N, H, W, C, Cout, R, S, stride, pad, dil=1, out=None, workspace=WORKSPACE):
    Ho, Wo = out or ((H + 2 * pad - dil * (R - 1) - 1) // stride + 1, (W + 2 * pad - dil * (S - 1) - 1) // stride + 1)
    p = _native.cuda().ronn_conv2d_plan(N, H, W, C, Cout, R, S, stride, pad, dil, Ho, Wo, workspace)
    return bool(p >> 20), p & 0xfff, p >> 12 & 0xff


def test_sixteen_channels_count_the_ctas_that_run():
    """100 tiles of 128 columns, one CTA per SM: two K slices would take two waves."""
    assert plan(2, 80, 80, 16, 128, 10, 10, 1, 4, out=(80, 80)) == (True, 128, 1)
    assert plan(1, 80, 80, 16, 128, 10, 10, 1, 4, out=(80, 80)) == (True, 128, 2)      # 50 tiles: one wave of slices
    assert plan(1, 112, 112, 16, 64, 10, 10, 1, 4, out=(112, 112)) == (True, 64, 3)    # 98 tiles of 64 columns, two CTAs per SM: 294 slots of 296


# what a ResNet-18 asks for, and what its descriptor or its channel count keeps from the TMA form
@pytest.mark.parametrize("layer,want", [
    ((1, 56, 56, 64, 64, 3, 3, 1, 1), (True, 64)), ((32, 56, 56, 64, 64, 3, 3, 1, 1), (True, 64)), ((117, 28, 28, 128, 128, 3, 3, 1, 1), (True, 128)),
    ((117, 14, 14, 256, 256, 3, 3, 1, 1), (True, 256)), ((8, 224, 224, 24, 64, 3, 3, 1, 1), (False, 64)), ((8, 56, 56, 64, 40, 3, 3, 1, 1), (False, 32)),
    ((1, 40, 40, 64, 64, 3, 3, 9, 1), (False, 64)), ((1, 300, 300, 64, 64, 3, 3, 1, 140), (False, 64)), ((2, 16, 16, 16, 64, 3, 3, 1, 1), (False, 64))])
def test_layers(layer, want):
    assert plan(*layer)[:2] == want


def test_slices_fit_the_workspace():
    assert plan(1, 7, 7, 512, 512, 3, 3, 1, 1)[2] > 1
    assert plan(1, 7, 7, 512, 512, 3, 3, 1, 1, workspace=0)[2] == 1
    for n in (1, 2, 4, 8, 32):
        for c in (64, 128, 256, 512):
            tma, bn, slices = plan(n, 14, 14, c, c, 3, 3, 1, 1)
            assert slices == 1 or slices * n * 196 * c <= WORKSPACE
