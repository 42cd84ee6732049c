"""Scratch memory and launch plan of BitLinear calls: asked of the native rules on the host, and the slot form on the device."""
import pytest
import torch

from ronn_b200 import _native


def _bytes(M, N, K, slot=False):
    lib = _native.cuda()
    return (lib.ronn_bitlinear_slot_workspace_bytes if slot else lib.ronn_bitlinear_workspace_bytes)(M, N, K)


def _expands(M, N, K):
    return _bytes(M, N, K) == N * K > _bytes(M, N, K, slot=True)


# one byte per weight where the weights are expanded; never less than the slices that the same call falls back to
@pytest.mark.parametrize("M,N,K", [(1024, 2560, 6912), (8192, 7680, 2560), (1024, 2568, 192), (3000, 1000, 192), (1024, 256, 2560)])
def test_scratch_of_many_rows(M, N, K):
    assert _bytes(M, N, K) in (max(N * K, _bytes(M, N, K, slot=True)), _bytes(M, N, K, slot=True))


# microseconds of the kernel that expands in every row tile, and of one expansion with a dense product (one B200, bf16)
@pytest.mark.parametrize("M,N,K,tiles,once", [
    (1024, 64, 6912, 7.9, 24.4), (1100, 256, 64, 3.5, 9.0), (1024, 512, 2560, 10.2, 14.9), (1024, 1024, 2560, 11.6, 15.7),
    (2048, 512, 6912, 21.3, 26.4), (8192, 8, 128, 3.6, 8.5), (1024, 2560, 64, 9.5, 9.2), (1024, 2560, 2560, 26.4, 18.3),
    (1024, 2560, 6912, 57.2, 31.5), (8192, 512, 2560, 27.0, 17.2), (2048, 1024, 6912, 30.6, 29.0), (8192, 7680, 2560, 346.0, 121.0),
    (8192, 13824, 64, 216.0, 79.2)])
def test_many_rows_take_the_faster_way(M, N, K, tiles, once):
    assert (once if _expands(M, N, K) else tiles) <= 1.06 * min(tiles, once)


@pytest.mark.parametrize("M,N,K", [(128, 2560, 6912), (1023, 256, 2560), (1, 640, 2560), (1100, 136, 48)])
def test_few_rows_and_other_k_only_slice(M, N, K):
    assert _bytes(M, N, K) == _bytes(M, N, K, slot=True)


def test_the_slot_form_takes_no_scratch_for_expanded_weights():
    """It never expands: whole wide outputs take none, narrow ones their slices, the same at 1024 rows as just below."""
    assert _bytes(1024, 2560, 6912, slot=True) == 0 and _bytes(8192, 13824, 2560, slot=True) == 0
    for N, K in ((256, 2560), (512, 6912), (1024, 6912)):
        assert 0 < _bytes(1024, N, K, slot=True) == _bytes(1023, N, K, slot=True) <= 148 * 64 * 1024


# "bn,slices" as asked for, also from 1024 rows on, where it switches the expansion off; what does not fit or is no tile leaves
# the plan alone
@pytest.mark.parametrize("tile,scratch", [("64,2", 8 * 4 * 2 * 64 * 512), ("128,4", 8 * 2 * 4 * 128 * 512), ("32,1", 0), ("48,1", None), ("128", None)])
def test_an_asked_for_tile_stands(tile, scratch, monkeypatch):
    from ronn_b200.ops import bitnet as B
    plain = _bytes(1024, 256, 2560)
    assert _expands(1024, 2560, 2560)
    monkeypatch.setenv("RONN_BITLINEAR_TILE", tile)
    assert _bytes(1024, 256, 2560) == (plain if scratch is None else scratch)
    assert _expands(1024, 2560, 2560) == (scratch is None)
    ws = B.slice_workspace(1024, 256, 2560, "cpu")
    assert (0 if ws is None else ws.numel()) == _bytes(1024, 256, 2560)
    monkeypatch.delenv("RONN_BITLINEAR_TILE")                # the size kept for the shape is not the other plan's
    ws = B.slice_workspace(1024, 256, 2560, "cpu")
    assert (0 if ws is None else ws.numel()) == plain


# expanded weights: rows past a tile and past its first half, columns cut inside a box, K of one and several blocks and cut inside
# one, rows of the result on and off the 16-byte grid; exact sums, so one rounding
@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(1024, 2568, 192), (1025, 2571, 192), (1030, 3000, 320), (1300, 2049, 64), (2049, 1544, 192), (1024, 2560, 1344)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_expanded_weights(M, N, K, dtype):
    from ronn_b200.ops import bitnet as B
    from ronn_b200.ops import kernels as Kn
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert _expands(M, N, K)
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    q = torch.randint(-127, 128, (M, K), generator=g, device="cuda", dtype=torch.int8)
    w = torch.randint(-1, 2, (N, K), generator=g, device="cuda", dtype=torch.int8)
    s = torch.rand(M, generator=g, device="cuda") * 0.01 + 0.001
    y = B.bitlinear_q(q, s, B.ternary_pack(w), 0.043, None, N, K, dtype)
    Kn.check_status()
    assert torch.equal(y, ((q.double() @ w.double().t()).float() * (s * torch.tensor(0.043, device="cuda"))[:, None]).to(dtype))


# the result lands in the slot that the state's parity names, with and without slices; exact sums, so one rounding
@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(1024, 256, 2560), (1030, 512, 320), (1024, 1024, 6912), (1024, 2560, 640), (96, 640, 2560)])
@pytest.mark.parametrize("parity", [0, 1])
def test_slot_form(M, N, K, parity):
    from ronn_b200.ops import bitnet as B
    from ronn_b200.ops import kernels as Kn
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    q = torch.randint(-127, 128, (M, K), generator=g, device="cuda", dtype=torch.int8)
    w = torch.randint(-1, 2, (N, K), generator=g, device="cuda", dtype=torch.int8)
    s = torch.rand(M, generator=g, device="cuda") * 0.01 + 0.001
    packed = B.ternary_pack(w)
    slots = torch.full((2, M, N), 7.0, dtype=torch.bfloat16, device="cuda")
    state = torch.tensor([4 + parity], dtype=torch.int32, device="cuda")
    ws = B.slice_workspace(M, N, K, q.device, slot=True)
    rc = _native.cuda().ronn_bitlinear_to_slot(q.data_ptr(), packed.data_ptr(), s.data_ptr(), 0.043, slots.data_ptr(), state.data_ptr(),
                                               M * N * 2, None if ws is None else ws.data_ptr(), M, N, K, K, 0,
                                               Kn.status_word(q.device).data_ptr(), Kn._stream())
    Kn.check_status()
    want = ((q.double() @ w.double().t()).float() * (s * torch.tensor(0.043, device="cuda"))[:, None]).bfloat16()
    assert rc == 0 and torch.equal(slots[parity], want) and bool((slots[1 - parity] == 7).all())


@pytest.mark.gpu
@pytest.mark.parametrize("tile", ["64,2", "128,1", "32,4"])
def test_an_asked_for_tile_computes_the_same(tile, monkeypatch):
    from ronn_b200.ops import bitnet as B
    from ronn_b200.ops import kernels as Kn
    g = torch.Generator(device="cuda").manual_seed(5)
    q = torch.randint(-127, 128, (1100, 2560), generator=g, device="cuda", dtype=torch.int8)
    packed = B.ternary_pack(torch.randint(-1, 2, (264, 2560), generator=g, device="cuda", dtype=torch.int8))
    s = torch.rand(1100, generator=g, device="cuda") * 0.01 + 0.001
    plain = B.bitlinear_q(q, s, packed, 0.043, None, 264, 2560, torch.bfloat16)
    monkeypatch.setenv("RONN_BITLINEAR_TILE", tile)
    assert torch.equal(B.bitlinear_q(q, s, packed, 0.043, None, 264, 2560, torch.bfloat16), plain)
    Kn.check_status()
