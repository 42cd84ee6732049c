"""Tile shapes and store paths of the tcgen05 GEMM against a 64-bit product of the same rounded operands: one rounding of the
result to 16 bits (half a unit in the last place, so below 2^-8 for bf16 and 2^-11 for fp16 as a relative error of the
whole)."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
TOL = {torch.bfloat16: 2 ** -8, torch.float16: 2 ** -11}


def _operands(M, N, Kd, dtype):
    g = torch.Generator(device="cuda").manual_seed(M * 131 + N + Kd)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dtype)
    return r(M, Kd), (r(N, Kd).float() / Kd ** 0.5).to(dtype), r(N), r(M, N)


# output rows that do not start on 16-byte boundaries: rows past the end of the last tile, column tiles cut short, every
# tile width the automatic choice takes there
@pytest.mark.parametrize("M,N,Kd", [(129, 1001, 64), (300, 131, 72), (1030, 4099, 128), (2600, 8009, 64), (513, 7, 8)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_rows_off_the_16_byte_grid(M, N, Kd, dtype):
    from ronn_b200.ops import kernels as K
    x, w, bias, res = _operands(M, N, Kd, dtype)
    out = torch.full((M + 1, N), 7.0, dtype=dtype, device="cuda")
    K.gemm(x, w, bias, res, "relu", out=out[:M])
    K.check_status()
    ref = F.relu(x.double() @ w.double().t() + bias.double()) + res.double()
    assert ((out[:M].double() - ref).norm() / ref.norm()).item() < TOL[dtype] and bool((out[M] == 7).all())


# bias on and off the 16-byte grid, columns cut short, residual rows with and without whole pieces
@pytest.mark.parametrize("M,N,Kd", [(200, 264, 64), (1100, 1000, 128), (1100, 260, 64)])
@pytest.mark.parametrize("off", [0, 1, 8])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_bias_and_residual_alignment(M, N, Kd, off, dtype):
    from ronn_b200.ops import kernels as K
    x, w, _, res = _operands(M, N, Kd, dtype)
    bias = torch.randn(N + off, device="cuda").to(dtype)[off:]
    y = K.gemm(x, w, bias, res, "gelu")
    K.check_status()
    ref = F.gelu(x.double() @ w.double().t() + bias.double(), approximate="tanh") + res.double()
    assert ((y.double() - ref).norm() / ref.norm()).item() < TOL[dtype]


# CTA pairs: rows past the second half of a tile, columns cut inside a box and inside a tile, one and several K blocks, results
# on and off the 16-byte grid, more tiles than pairs
@pytest.mark.parametrize("M,N,Kd", [(256, 256, 64), (129, 200, 72), (300, 1000, 128), (1, 264, 8), (1000, 515, 320), (5200, 2304, 64)])
@pytest.mark.parametrize("act", ["", "relu", "gelu"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_cta_pairs(M, N, Kd, act, dtype):
    from ronn_b200.ops import kernels as K
    x, w, bias, res = _operands(M, N, Kd, dtype)
    lin = x.double() @ w.double().t() + bias.double()
    ref = {"": lin, "relu": F.relu(lin), "gelu": F.gelu(lin, approximate="tanh")}[act]
    for r in (None, res):
        out = torch.full((M + 1, N), 7.0, dtype=dtype, device="cuda")
        K.gemm(x, w, bias, r, act, out=out[:M], bn=0x4000 | 256)
        K.check_status()
        want = ref if r is None else ref + r.double()
        assert ((out[:M].double() - want).norm() / want.norm()).item() < TOL[dtype] and bool((out[M] == 7).all())
    y32 = K.gemm(x, w, None, None, "", out_fp32=True, bn=0x4000 | 256)
    assert ((y32.double() - x.double() @ w.double().t()).norm() / y32.double().norm()).item() < 1e-5


# the automatic choice over sizes that end in each of its forms
@pytest.mark.parametrize("M,N,Kd", [(1024, 768, 768), (2048, 768, 3072), (4662, 1024, 1024), (8192, 3072, 768), (1024, 96, 64)])
def test_automatic_forms_agree(M, N, Kd):
    from ronn_b200.ops import kernels as K
    x, w, bias, res = _operands(M, N, Kd, torch.bfloat16)
    want = F.gelu(x.double() @ w.double().t() + bias.double(), approximate="tanh") + res.double()
    y = K.gemm(x, w, bias, res, "gelu")
    K.check_status()
    assert ((y.double() - want).norm() / want.norm()).item() < TOL[torch.bfloat16]


# the automatic choice on a chip of 148 SMs, one size and more for every form that it has; every value within its own bound, so
# that a single lost or misplaced piece of a row shows: the rounding of the result (half a unit in the last place: 2^-8 for
# the 8-bit significand of bf16) and K products summed in fp32 (K x 2^-23 of the sum of their magnitudes, times 1.13 for the slope of GELU)
@pytest.mark.parametrize("M,N,Kd,act,resid,fp32,width,ring", [
    (1024, 16, 64, "", False, False, 32, 0x2000), (1024, 10, 64, "", True, False, 32, 0x1000), (1100, 64, 1000, "", False, True, 32, 0x1000),
    (8192, 520, 64, "relu", True, False, 64, 0x2000), (1030, 768, 768, "gelu", True, False, 64, 0x1000),
    (1500, 1000, 2048, "", True, False, 128, 0x1000), (8192, 203, 1024, "gelu", False, False, 128, 0x1000),
    (1536, 8192, 64, "", False, True, 128, 0x2000), (2048, 2304, 4096, "", False, True, 256, 0),
    (8190, 776, 768, "gelu", True, False, 256, 0x4000), (4662, 4099, 128, "", False, False, 256, 0x4000)])
def test_every_form_of_the_automatic_choice(M, N, Kd, act, resid, fp32, width, ring):
    from ronn_b200 import _native
    from ronn_b200.ops import kernels as K
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        ldc = N if N % 8 else -(-N // 8) * 8
        assert _native.cuda().ronn_gemm_form(M, N, Kd, K._ACT[act], int(resid), int(fp32), ldc, 0) == width | ring
    x, w, bias, res = _operands(M, N, Kd, torch.bfloat16)
    lin = x.double() @ w.double().t() + bias.double()
    want = F.relu(lin) if act == "relu" else F.gelu(lin, approximate="tanh") if act == "gelu" else lin
    want = want + res.double() if resid else want
    out = torch.full((M + 1, N), 7.0, dtype=torch.float32 if fp32 else torch.bfloat16, device="cuda")
    K.gemm(x, w, bias, res if resid else None, act, out=out[:M])
    K.check_status()
    bound = (2 ** -24 if fp32 else 2 ** -8) * want.abs() + 1.13 * Kd * 2 ** -23 * (x.double().abs() @ w.double().abs().t() + bias.double().abs()) + 2 ** -23 * res.double().abs() + 1e-5
    assert bool(((out[:M].double() - want).abs() <= bound).all()) and bool((out[M] == 7).all())
