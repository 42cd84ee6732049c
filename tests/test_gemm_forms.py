"""Which kernel a GEMM runs: asked of the native rule, on the host."""
import os
import subprocess
import sys

import pytest

from ronn_b200 import _native

SKINNY, PAIR, SHALLOW, DEEP = 0x8000, 0x4000, 0x2000, 0x1000


def form(M, N, K, act="", residual=False, fp32=False, ldc=None, bn=0):
    from ronn_b200.ops.kernels import _ACT
    return _native.cuda().ronn_gemm_form(M, N, K, _ACT[act], int(residual), int(fp32), -(-N // 8) * 8 if ldc is None else ldc, bn)


# many rows and few, every width that the automatic choice may take, results on and off the 16-byte grid
@pytest.mark.parametrize("M,N,K", [(1024, 768, 768), (8192, 768, 768), (8192, 64, 256), (300, 4096, 1024), (200, 3072, 1024), (2048, 769, 512)])
@pytest.mark.parametrize("ring", [DEEP, SHALLOW])
def test_a_ring_that_is_asked_for_stands(M, N, K, ring):
    f = form(M, N, K, bn=ring, ldc=N)
    assert f & 0xfff in (32, 64, 128, 256) and (f & 0xfff == 256 or f & (DEEP | SHALLOW) == ring)
    for bn in (32, 64, 128):
        assert form(M, N, K, bn=bn | ring, ldc=N) == bn | ring


@pytest.mark.parametrize("name,ring", [("deep", DEEP), ("shallow", SHALLOW)])
def test_the_ring_of_the_environment_stands(name, ring):
    code = ("from ronn_b200 import _native; f = _native.cuda().ronn_gemm_form; "
            "print(*[f(M, N, K, 0, 0, 0, N, 0) for M, N, K in ((1024, 768, 768), (8192, 768, 768), (8192, 64, 256), (200, 3072, 1024))], "
            f"f(1024, 768, 768, 0, 0, 0, 768, 64 | {DEEP ^ SHALLOW ^ ring}))")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, RONN_GEMM_RING=name), cwd=root, capture_output=True, text=True)
    assert out.returncode == 0, out.stderr
    *auto, given = [int(v) for v in out.stdout.split()]
    assert all(f & 0xfff == 256 or f & (DEEP | SHALLOW) == ring for f in auto)
    assert given == 64 | (DEEP ^ SHALLOW ^ ring)             # a call that says goes before it


# one CTA per SM has the deep ring: it is fed by the bytes it keeps in flight
@pytest.mark.parametrize("M,N,K", [(1024, 768, 768), (1536, 768, 3072), (1024, 1024, 1024), (1024, 1152, 768)])
def test_a_tile_alone_on_its_sm_has_the_deep_ring(M, N, K):
    f = form(M, N, K)
    tiles = -(-M // 128) * -(-N // (f & 0xfff))
    assert f & 0xfff == 64 and tiles <= 148 and f & DEEP
