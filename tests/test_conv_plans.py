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


# the image network's first convolution: sizes that the one-call form never takes ask it for nothing and allocate nothing for it
@pytest.mark.parametrize("cout,one_call", [(64, True), (72, True), (40, False), (68, False)])
def test_stem_allocates_for_the_form_that_runs(cout, one_call, monkeypatch):
    from types import SimpleNamespace

    import torch

    from ronn_b200.providers import gpu_conv as G
    calls, sizes, empty = [], [], torch.empty
    lib = SimpleNamespace(ronn_stem_conv=lambda *a: calls.append("stem") or 0, ronn_nchw_to_s2d16=lambda *a: calls.append("s2d") or 0)
    monkeypatch.setattr(G._native, "cuda", lambda: lib)
    monkeypatch.setattr(G.K, "status_word", lambda device: torch.zeros(4, dtype=torch.int32))
    monkeypatch.setattr(G.torch.cuda, "current_stream", lambda: SimpleNamespace(cuda_stream=0))
    monkeypatch.setattr(G.torch, "empty", lambda shape, **kw: sizes.append(shape) or empty(shape, **kw))
    monkeypatch.setattr(G, "conv2d_nhwc", lambda *a, **kw: calls.append("conv"))
    G.stem_conv_s2d(torch.zeros(1, 3, 8, 12, dtype=torch.float16), torch.zeros(cout, 4, 4, 16, dtype=torch.float16), None, True)
    assert calls == (["stem"] if one_call else ["s2d", "conv"])
    assert sizes == ([(1, 4, 6, cout), 4 * 9 * 16] if one_call else [(1, 4, 6, 16)])
