"""Key lengths of additive padding masks, and LayerNorm(x + skip) with a broadcast skip, against plain PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S", [(1, 1), (3, 31), (2, 256), (5, 300), (64, 128)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_key_lengths(B, S, dtype):
    from ronn_b200.ops import kernels as K
    lens = torch.randint(0, S + 1, (B, 1), generator=torch.Generator().manual_seed(S))
    one = torch.tensor(1.0, dtype=dtype)
    mask = ((one - (torch.arange(S)[None] < lens).to(dtype)) * torch.tensor(-10000.0, dtype=dtype)).cuda()
    want = lens.clamp(min=1).squeeze(1).to(torch.int32)
    assert torch.equal(K.key_lengths(mask).cpu(), want)
    wide = torch.zeros(B, 2 * S + 1, dtype=dtype, device="cuda")
    wide[:, 1:S + 1] = mask
    assert torch.equal(K.key_lengths(wide[:, 1:S + 1]).cpu(), want)
    mask[0, 0] = float("nan")                                # compares false, as in (mask > -1e4)
    assert torch.equal(K.key_lengths(mask), (mask > -1e4).sum(-1).clamp_(min=1).to(torch.int32))


@pytest.mark.parametrize("skip_shape", [(7, 64), (1, 7, 64), (64,), (4, 1, 64), (4, 7, 64)])
def test_skip_layernorm_broadcast(skip_shape):
    from ronn_b200 import Model, SessionOptions
    from ronn_b200.core.types import DataType
    from ronn_b200.graph.ir import ModelGraph, TensorInfo
    g = ModelGraph()
    g.inputs = [TensorInfo("x", [0, 0, 64], DataType.F16, [None] * 3), TensorInfo("s", list(skip_shape), DataType.F16, [None] * len(skip_shape))]
    g.outputs = [TensorInfo("y", [0, 0, 64], DataType.F16, [None] * 3)]
    gen = torch.Generator().manual_seed(0)
    g.initializers["w"] = torch.rand(64, generator=gen).half()
    g.initializers["b"] = torch.randn(64, generator=gen).half()
    g.add_node("Add", ["x", "s"], ["sum"], name="add")
    g.add_node("LayerNormalization", ["sum", "w", "b"], ["y"], {"axis": -1, "epsilon": 1e-5}, name="ln")
    x, s = torch.randn(4, 7, 64, generator=gen).half().cuda(), torch.randn(*skip_shape, generator=gen).half().cuda()
    y = Model.from_graph(g).create_session(SessionOptions().with_provider("gpu").with_optimization_level("O3")).run({"x": x, "s": s})["y"]
    ref = torch.nn.functional.layer_norm(x.double() + s.double(), (64,), g.initializers["w"].cuda().double(), g.initializers["b"].cuda().double(), 1e-5)
    assert y.shape == ref.shape and ((y.double() - ref).norm() / ref.norm()).item() < 2 ** -11 + 2 ** -11      # sum and result rounded once each
