"""BitLinear calls with many rows (weights expanded once, dense int8 GEMM) against an integer product in 64 bits: the sums
are exact, so the result is one rounding of sum * (x_scale * w_scale) [+ bias]."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,Kd", [(1024, 256, 64), (1025, 264, 192), (1500, 1000, 2560), (2049, 40, 320), (1023, 264, 192), (1100, 136, 48)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_many_rows(M, N, Kd, dtype):
    from ronn_b200.ops import bitnet as B
    from ronn_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(M + N + Kd)
    q = torch.randint(-127, 128, (M, Kd), generator=g, device="cuda", dtype=torch.int8)
    w = torch.randint(-1, 2, (N, Kd), generator=g, device="cuda", dtype=torch.int8)
    s = torch.rand(M, generator=g, device="cuda") * 0.01 + 0.001
    acc = q.double() @ w.double().t()
    y = B.bitlinear_q(q, s, B.ternary_pack(w), 0.043, None, N, Kd, dtype)
    K.check_status()
    want = acc.float() * (s * torch.tensor(0.043, device="cuda"))[:, None]
    assert torch.equal(y, want.to(dtype))
    bias = torch.randn(N, generator=g, device="cuda").to(dtype)
    y = B.bitlinear_q(q, s, B.ternary_pack(w), 0.043, bias, N, Kd, dtype)
    ref = acc * (s.double() * 0.043)[:, None] + bias.double()
    assert ((y.double() - ref).norm() / ref.norm()).item() < (2 ** -8 if dtype == torch.bfloat16 else 2 ** -11)
