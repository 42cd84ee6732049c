"""Convolutions whose operand arrives by TMA im2col loads, against a 64-bit convolution of the same rounded operands.

fp32 accumulation of K <= 9 * 256 products and one rounding of the result: relative error of the whole result below half a
unit in the last place of the 16-bit type plus K^0.5 * 2^-23."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _ref(x, w, b, res, stride, pad, dil, relu, out_hw=None):
    y = F.conv2d(F.pad(x.double().permute(0, 3, 1, 2), (pad, pad + 8, pad, pad + 8)), w.double().permute(0, 3, 1, 2), None, stride, 0, dil)
    N, H, W, _ = x.shape
    ho = out_hw[0] if out_hw else (H + 2 * pad - dil * (w.shape[1] - 1) - 1) // stride + 1
    wo = out_hw[1] if out_hw else (W + 2 * pad - dil * (w.shape[2] - 1) - 1) // stride + 1
    y = y[:, :, :ho, :wo].permute(0, 2, 3, 1) + b.double()
    y = y if res is None else y + res.double()
    return F.relu(y) if relu else y


# N, H, W, C, Cout, R, S, stride, pad, dil: non-square images and filters, the last tile past the last image, one and several
# channel blocks per tap, column tiles of 64 / 128 / 256 and a ragged one, K slices, four taps per K block
@pytest.mark.parametrize("shape", [(2, 13, 9, 64, 64, 3, 3, 1, 1, 1), (1, 7, 7, 512, 512, 3, 3, 1, 1, 1), (3, 30, 17, 128, 136, 3, 3, 2, 1, 1),
                                   (2, 20, 22, 64, 128, 1, 1, 2, 0, 1), (1, 25, 19, 192, 72, 3, 5, 1, 2, 2), (37, 28, 29, 128, 256, 3, 3, 1, 1, 1),
                                   (2, 18, 31, 16, 64, 4, 4, 1, 2, 1), (1, 9, 40, 16, 128, 2, 2, 1, 0, 1), (5, 40, 33, 64, 64, 5, 3, 3, 0, 1),
                                   (2, 12, 12, 24, 64, 3, 3, 1, 1, 1), (1, 8, 8, 64, 40, 3, 3, 1, 1, 1)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_conv_against_64_bits(shape, dtype):
    from ronn_b200.ops import kernels as K
    from ronn_b200.providers.gpu_conv import conv2d_nhwc
    N, H, W, C, Cout, R, S, stride, pad, dil = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    x = torch.randn(N, H, W, C, generator=g, device="cuda").to(dtype)
    w = (torch.randn(Cout, R, S, C, generator=g, device="cuda") / (R * S * C) ** 0.5).to(dtype)
    b = torch.randn(Cout, generator=g, device="cuda").to(dtype)
    hw = (H, W) if (R, C) == (4, 16) else None               # the stem form: one output position per input position
    ref = _ref(x, w, b, None, stride, pad, dil, False, hw)
    y = conv2d_nhwc(x, w, b, None, stride, pad, dil, False, out_hw=hw)
    K.check_status()
    tol = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -11
    assert y.shape == ref.shape and ((y.double() - ref).norm() / ref.norm()).item() < tol
    res = torch.randn(y.shape, generator=g, device="cuda").to(dtype)
    ref = _ref(x, w, b, res, stride, pad, dil, True, hw)
    y = conv2d_nhwc(x, w, b, res, stride, pad, dil, True, out_hw=hw)
    K.check_status()
    assert ((y.double() - ref).norm() / ref.norm()).item() < tol


# 7x7 / stride 2 / pad 3 from NCHW: narrow and wide images, every channel count the rearranged form holds, one and two column
# tiles, and (40 channels out) the two-call form
@pytest.mark.parametrize("shape", [(1, 3, 224, 224, 64), (2, 4, 18, 30, 64), (3, 1, 2, 2, 72), (5, 3, 160, 256, 136), (2, 3, 20, 22, 40)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_stem_against_64_bits(shape, dtype):
    from ronn_b200.ops import kernels as K
    from ronn_b200.providers.gpu_conv import stem_conv_s2d, stem_weights_s2d
    N, C, H, W, Cout = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    x = torch.randn(N, C, H, W, generator=g, device="cuda").to(dtype)
    w = (torch.randn(Cout, C, 7, 7, generator=g, device="cuda") / (49 * C) ** 0.5).to(dtype)
    b = torch.randn(Cout, generator=g, device="cuda").to(dtype)
    y = stem_conv_s2d(x, stem_weights_s2d(w.permute(0, 2, 3, 1).contiguous()), b, True)
    K.check_status()
    ref = F.relu(F.conv2d(x.double(), w.double(), b.double(), 2, 3)).permute(0, 2, 3, 1)
    assert y.shape == ref.shape and ((y.double() - ref).norm() / ref.norm()).item() < (2 ** -8 if dtype == torch.bfloat16 else 2 ** -11)


# every form that a plan may take on a chip of 148 SMs; every value within its own bound, so that a lost or misplaced piece shows:
# the rounding of the result (2^-11 for fp16) and K products summed in fp32 (K x 2^-23 of the sum of their magnitudes)
@pytest.mark.parametrize("shape,want", [
    ((40, 30, 29, 128, 256, 3, 3, 1, 1), (True, 256, 1)), ((40, 30, 29, 128, 128, 3, 3, 1, 1), (True, 128, 1)), ((33, 57, 55, 64, 72, 3, 3, 1, 1), (True, 64, 1)),
    ((2, 20, 21, 64, 64, 1, 1, 1, 0), (True, 64, 1)), ((1, 7, 7, 512, 512, 3, 3, 1, 1), (True, None, None)), ((2, 57, 56, 16, 64, 4, 4, 1, 1), (True, 64, 1)),
    ((2, 57, 56, 16, 136, 2, 2, 2, 0), (True, 128, 1)), ((1, 84, 84, 16, 128, 10, 10, 1, 2), (True, 128, 3)), ((2, 30, 31, 24, 136, 3, 3, 1, 1), (False, 128, None))])
def test_every_plan_value_by_value(shape, want):
    from ronn_b200 import _native
    from ronn_b200.ops import kernels as K
    from ronn_b200.providers.gpu_conv import conv2d_nhwc
    N, H, W, C, Cout, R, S, stride, pad = shape
    Ho, Wo = (H + 2 * pad - R) // stride + 1, (W + 2 * pad - S) // stride + 1
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        p = _native.cuda().ronn_conv2d_plan(N, H, W, C, Cout, R, S, stride, pad, 1, Ho, Wo, 1 << 22)
        got = (bool(p >> 20), p & 0xfff, p >> 12 & 0xff)
        assert all(w is None or w == v for w, v in zip(want, got)), got
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    x = torch.randn(N, H, W, C, generator=g, device="cuda").half()
    w = (torch.randn(Cout, R, S, C, generator=g, device="cuda") / (R * S * C) ** 0.5).half()
    b = torch.randn(Cout, generator=g, device="cuda").half()
    y = conv2d_nhwc(x, w, b, None, stride, pad, 1, False)
    K.check_status()
    ref = _ref(x, w, b, None, stride, pad, 1, False)
    bound = 2 ** -11 * ref.abs() + (R * S * C) * 2 ** -23 * _ref(x.abs(), w.abs(), b.abs(), None, stride, pad, 1, False) + 2 ** -24
    assert y.shape == ref.shape and bool(((y.double() - ref).abs() <= bound).all())
