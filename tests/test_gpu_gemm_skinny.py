"""The few-rows projection kernel: against a 64-bit product of the same rounded operands.

fp32 results: sums of K products in fp32, relative error of the whole result below K^0.5 * 2^-23 plus the fast-math GELU
(about 1e-6): 1e-5.  With a fused norm the normalised rows are rounded to 16 bits and values that sit on a rounding boundary
may fall the other way (one unit in the last place in a small share of the values): 2^-8 / 8 for bf16, 2^-11 / 8 for fp16."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from ronn_b200.ops import kernels
    return kernels


def _operands(M, N, Kd, dtype):
    g = torch.Generator(device="cuda").manual_seed(M * 131 + N + Kd)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dtype)
    return r(M, Kd), (r(N, Kd).float() / Kd ** 0.5).to(dtype), r(N), r(M, N)


def _err(y, ref):
    return ((y.double() - ref).norm() / ref.norm()).item()


# rows at the edges of the 8- and 16-row halves and of a second slice; columns off the tile; K at one value group, at and
# past the register-resident limit (1024), off the 32-value piece
@pytest.mark.parametrize("M,N,Kd", [(1, 10, 128), (8, 50, 784), (9, 1000, 512), (16, 7, 8), (17, 768, 1024), (40, 136, 1032),
                                    (33, 131, 2568), (48, 768, 3072), (3, 50257, 64), (12, 50257, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("act", ["", "relu", "gelu"])
def test_few_rows_gemm(K, M, N, Kd, dtype, act):
    x, w, bias, res = _operands(M, N, Kd, dtype)
    ref = x.double() @ w.double().t() + bias.double()
    ref = F.relu(ref) if act == "relu" else F.gelu(ref, approximate="tanh") if act == "gelu" else ref
    y32 = K.gemm(x, w, bias, None, act, out_fp32=True)
    assert _err(y32, ref) < 1e-5
    y = K.gemm(x, w, bias, res, act)
    assert y.dtype == dtype and _err(y, ref + res.double()) < (2 ** -8 if dtype == torch.bfloat16 else 2 ** -11)


@pytest.mark.parametrize("M,N,Kd", [(1, 3072, 1024), (2, 20, 8), (7, 2304, 768), (8, 50257, 264)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("norm", ["layernorm", "rmsnorm"])
def test_norm_joins_the_projection(K, M, N, Kd, dtype, norm):
    x, w, bias, _ = _operands(M, N, Kd, dtype)
    x = x * 3 + 1
    gamma, beta = (torch.rand(Kd, device="cuda") + 0.5).to(dtype), torch.randn(Kd, device="cuda").to(dtype)
    if norm == "layernorm":
        h = F.layer_norm(x.double(), (Kd,), gamma.double(), beta.double(), 1e-5)
    else:
        beta = None
        h = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-5) * gamma.double()
    ref = h.to(dtype).double() @ w.double().t() + bias.double()
    y = K.norm_gemm(x, gamma, beta, 1e-5, norm, w, bias, out=torch.empty(M, N, device="cuda", dtype=torch.float32))
    assert _err(y, ref) < (2 ** -11 if dtype == torch.bfloat16 else 2 ** -14)


def test_strided_operands_and_refusals(K):
    x, w, bias, _ = _operands(5, 40, 64, torch.bfloat16)
    wide = torch.zeros(5, 128, dtype=torch.bfloat16, device="cuda")
    wide[:, 64:] = x
    out = torch.full((5, 48), 7.0, dtype=torch.bfloat16, device="cuda")
    K.gemm(wide[:, 64:], w, bias, out=out[:, :40])
    assert torch.equal(out[:, :40], K.gemm(x, w, bias)) and bool((out[:, 40:] == 7).all())
    flat = torch.zeros(5 * 64 + 1, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(K.KernelError):                       # operand off the 16-byte grid
        K.gemm(flat[1:].view(5, 64), w)
    with pytest.raises(K.KernelError):                       # K not a multiple of 8
        K.gemm(x[:, :60].contiguous(), w[:, :60].contiguous())
    big = torch.zeros(9, 64, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(K.KernelError):                       # more rows than a fused norm takes
        K.norm_gemm(big, bias[:1].expand(64).contiguous(), None, 1e-5, "rmsnorm", w)
    nan = x.clone()
    nan[2, 3] = float("nan")
    y = K.gemm(nan, w)
    assert bool(y[2].isnan().all()) and torch.equal(y[[0, 1, 3, 4]], K.gemm(x, w)[[0, 1, 3, 4]])


# four, five and six slices of 16 rows, whatever the automatic choice takes: K in registers and streamed, K off the 32-value piece,
# two row groups per tile (N past 4736 on 148 SMs), the last slice with one row and whole.  Every value within its own bound:
# the rounding of the result (2^-24 for fp32, 2^-8 and 2^-11 for bf16 and fp16), K products summed in fp32 (K x 2^-23 of the
# sum of their magnitudes, times 1.13 for the slope of GELU) and 2^-18 of a GELU's value for its fast exponential
@pytest.mark.parametrize("M,N,Kd", [(49, 136, 1032), (64, 768, 3072), (65, 131, 2568), (80, 4800, 72), (81, 1000, 512), (96, 7, 8), (96, 768, 3072), (96, 5000, 1024)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("act", ["", "gelu"])
def test_up_to_six_slices(K, M, N, Kd, dtype, act):
    from ronn_b200 import _native
    x, w, bias, res = _operands(M, N, Kd, dtype)
    lin = x.double() @ w.double().t() + bias.double()
    ref = F.gelu(lin, approximate="tanh") if act == "gelu" else lin
    sums = 1.13 * Kd * 2 ** -23 * (x.double().abs() @ w.double().abs().t() + bias.double().abs()) + 2 ** -18 * ref.abs() + 1e-6
    for out_dtype, r in ((torch.float32, None), (dtype, res)):
        out = torch.full((M + 1, N), 7.0, dtype=out_dtype, device="cuda")
        rc = _native.cuda().ronn_gemm_skinny(x.data_ptr(), w.data_ptr(), out.data_ptr(), bias.data_ptr(), K._ptr(r), None, None, 0.0, 0,
                                             M, N, Kd, Kd, Kd, N, K._DT[dtype], K._ACT[act], int(out_dtype == torch.float32), K._stream())
        want = ref if r is None else ref + r.double()
        u = {torch.float32: 2 ** -24, torch.bfloat16: 2 ** -8, torch.float16: 2 ** -11}[out_dtype]
        assert rc == 0 and bool(((out[:M].double() - want).abs() <= u * want.abs() + sums + 2 ** -23 * res.double().abs()).all())
        assert bool((out[M] == 7).all())


# both sides of the line between the few-rows kernel and the tiles, up to its last row
@pytest.mark.parametrize("M,N,Kd,skinny", [(48, 2304, 768, True), (64, 2304, 768, False), (96, 768, 3072, True), (97, 768, 3072, False),
                                           (64, 1024, 4096, True), (64, 8192, 64, False), (16, 8192, 64, True), (32, 768, 768, True)])
def test_both_sides_of_the_line(K, M, N, Kd, skinny):
    from ronn_b200 import _native
    assert (_native.cuda().ronn_gemm_form(M, N, Kd, 0, 1, 0, N, 0) == 0x8000) == skinny
    x, w, bias, res = _operands(M, N, Kd, torch.bfloat16)
    ref = x.double() @ w.double().t() + bias.double() + res.double()
    y = K.gemm(x, w, bias, res)
    K.check_status()
    bound = 2 ** -8 * ref.abs() + Kd * 2 ** -23 * (x.double().abs() @ w.double().abs().t()) + 2 ** -22 * (bias.double().abs() + res.double().abs()) + 1e-6
    assert bool(((y.double() - ref).abs() <= bound).all())
