"""Norm nodes of the GPU provider whose operands the kernel does not read as they are: the library operator's result, or
its error, and never a launch on an address of another type, device or length."""
from types import SimpleNamespace

import pytest
import torch
import torch.nn.functional as F

from ronn_b200.graph.ir import ModelGraph
from ronn_b200.ops import kernels as K
from ronn_b200.providers.gpu_ops import GpuOpTable

H = 64


def _node(op):
    """The provider's closure for one node, outside a session: (operands) -> outputs."""
    g = ModelGraph()
    names = {"SkipLayerNorm": ["x", "s", "w", "b"], "LayerNormalization": ["x", "w", "b"], "RMSNorm": ["x", "w"]}[op]
    node = g.add_node(op, names, ["y", "sum"] if op == "SkipLayerNorm" else ["y"], {"epsilon": 1e-5}, name="n")
    device = torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")
    table = GpuOpTable(SimpleNamespace(device=device, config=SimpleNamespace(enable_custom_kernels=True)), g, None)
    run = table.resolve(g.nodes[0] if node is None else node, g)
    return lambda *operands: run(list(operands), {"epsilon": 1e-5}, None)


def _operands(op, skip_shape, dtype=torch.float16, param_dtype=torch.float16, device="cpu"):
    gen = torch.Generator().manual_seed(3)
    x = torch.randn(4, 7, H, generator=gen).to(dtype)
    s = torch.randn(*skip_shape, generator=gen).to(dtype)
    w, b = (torch.rand(H, generator=gen) + 0.5).to(param_dtype), torch.randn(H, generator=gen).to(param_dtype)
    ops = {"SkipLayerNorm": [x, s, w, b], "LayerNormalization": [x, w, b], "RMSNorm": [x, w]}[op]
    return [t.to(device) for t in ops]


def _reference(op, ops):
    ops = [t.cpu().double() for t in ops]
    if op == "RMSNorm":
        return ops[0] * torch.rsqrt(ops[0].pow(2).mean(-1, keepdim=True) + 1e-5) * ops[1]
    x = (ops[0] + ops[1]).half().double() if op == "SkipLayerNorm" else ops[0]          # the sum is held in 16 bits
    return F.layer_norm(x, (H,), ops[-2], ops[-1], 1e-5)


KINDS = [("SkipLayerNorm", (4, 7, H)), ("SkipLayerNorm", (7, H)), ("LayerNormalization", (7, H)), ("RMSNorm", (7, H))]


# results are one rounding to 16 bits: half a unit in the last place, 2^-11 relative
@pytest.mark.parametrize("op,skip", KINDS)
def test_host_operands(op, skip):
    ops = _operands(op, skip)
    y = _node(op)(*ops)[0]
    assert y.dtype == torch.float16 and ((y.double() - _reference(op, ops)).norm() / _reference(op, ops).norm()).item() < 2 ** -11


@pytest.mark.parametrize("op,skip", KINDS)
@pytest.mark.parametrize("n", [H // 2, 2 * H])
def test_parameters_of_another_length_are_refused(op, skip, n):
    """On the host: a launch with them would read past the end of the parameters."""
    ops = _operands(op, skip)
    ops[-1] = torch.ones(n, dtype=torch.float16)
    with pytest.raises(RuntimeError):
        _node(op)(*ops)


def _fake(shape, dtype=torch.float16, device=0, contiguous=True, address=256):
    """A tensor as the check sees it; device -1 is the host."""
    n = 1
    for d in shape:
        n *= d
    return SimpleNamespace(shape=shape, dtype=dtype, get_device=lambda: device, numel=lambda: n,
                           is_contiguous=lambda: contiguous, data_ptr=lambda: address)


@pytest.mark.parametrize("bad", [dict(dtype=torch.float32), dict(dtype=torch.bfloat16), dict(device=-1), dict(device=1),
                                 dict(shape=(H // 2,)), dict(shape=(2 * H,)), dict(contiguous=False), dict(address=264)])
def test_the_kernel_refuses_other_parameters(bad):
    x = _fake((3, H))
    good = _fake((H,))
    K._check_norm_operands(x, _fake((3, H)), good, None, _fake((1, H)))
    with pytest.raises(K.OperandError):
        K._check_norm_operands(x, None, good, _fake(**{"shape": (H,), **bad}))


@pytest.mark.parametrize("x", [dict(dtype=torch.float32), dict(device=-1), dict(shape=(3, 60)), dict(shape=(2, 32776)), dict(shape=(3, 0))])
def test_the_kernel_refuses_other_rows(x):
    with pytest.raises(K.OperandError):
        K._check_norm_operands(_fake(**{"shape": (3, H), **x}), None)
    with pytest.raises(K.OperandError):
        K._check_norm_operands(_fake((3, H)), _fake(**{"shape": (3, H), "dtype": torch.bfloat16}))


@pytest.mark.gpu
@pytest.mark.parametrize("op,skip", KINDS)
@pytest.mark.parametrize("params", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("host", [None, 0, 1, -1])
def test_types_and_places_on_the_device(op, skip, params, host):
    """Parameters of every type, and each operand in turn on the host, as shape arithmetic leaves it."""
    ops = _operands(op, skip, param_dtype=params, device="cuda")
    if host is not None:
        ops[host] = ops[host].cpu()
    y = _node(op)(*ops)[0]
    ref = _reference(op, ops)
    assert y.is_cuda and y.dtype == torch.float16 and ((y.cpu().double() - ref).norm() / ref.norm()).item() < 2 ** -11 + 2 ** -11


@pytest.mark.gpu
def test_a_session_that_keeps_the_models_types():
    from ronn_b200 import Model, SessionOptions
    from ronn_b200.core.types import DataType
    from ronn_b200.graph.ir import TensorInfo
    g = ModelGraph()
    g.inputs = [TensorInfo("x", [0, 0, H], DataType.F16, [None] * 3), TensorInfo("s", [7, H], DataType.F16, [None] * 2)]
    g.outputs = [TensorInfo("y", [0, 0, H], DataType.F16, [None] * 3)]
    x, s, w, b = _operands("SkipLayerNorm", (7, H), param_dtype=torch.float32)
    g.initializers["w"], g.initializers["b"] = w, b
    g.add_node("Add", ["x", "s"], ["sum"], name="add")
    g.add_node("LayerNormalization", ["sum", "w", "b"], ["y"], {"axis": -1, "epsilon": 1e-5}, name="ln")
    session = Model.from_graph(g).create_session(SessionOptions().with_provider("gpu").with_optimization_level("O3"))
    y = session.run({"x": x.cuda(), "s": s.cuda()})["y"]
    ref = _reference("SkipLayerNorm", [x, s, w, b])
    assert ((y.cpu().double() - ref).norm() / ref.norm()).item() < 2 ** -11 + 2 ** -11
