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


_NAMES = {"S": SHALLOW, "D": DEEP, "": 0}

# calls with many rows and the microseconds each form took (one B200, bf16, chains inside a CUDA graph): "res" with a
# residual, "f32" fp32 results, "rag" an odd row length; S the shallow, D the deep ring
_MEASURED = [
    (1024, 10, 64, "plain", "32S:4.3 32D:4.7"),
    (4096, 10, 128, "f32", "32S:4.7 32D:5.0"),
    (1024, 64, 1024, "f32", "32S:8.4 32D:7.7 64S:9.5 64D:8.8"),
    (8192, 32, 256, "gelu", "32S:5.1 32D:5.3"),
    (4096, 96, 512, "plain", "32S:6.0 32D:6.2 64S:6.4 64D:6.0 128D:7.1"),
    (1024, 128, 4096, "f32", "32S:22.8 32D:19.3 64S:23.4 64D:20.4 128D:22.8"),
    (8192, 128, 256, "plain", "32S:6.1 32D:6.4 64S:5.3 64D:5.4 128D:6.5"),
    (1024, 768, 64, "plain", "32S:4.7 32D:5.3 64S:4.7 64D:4.4 128D:5.7 256:8.1 PAIR:7.4"),
    (1024, 768, 768, "gelu", "32S:8.8 32D:10.8 64S:8.8 64D:8.1 128D:9.5 256:13.9 PAIR:12.7"),
    (1024, 768, 2048, "res", "32S:15.3 32D:20.1 64S:14.7 64D:13.0 128D:14.9 256:20.0 PAIR:18.0"),
    (1536, 768, 768, "gelures", "32S:9.8 32D:11.8 64S:9.1 64D:9.1 128D:10.9 256:16.6 PAIR:13.5"),
    (1536, 1024, 2048, "plain", "32S:24.5 32D:28.9 64S:15.6 64D:20.4 128D:14.0 256:18.0 PAIR:18.0"),
    (1536, 2304, 768, "plain", "64S:14.3 64D:14.9 128D:12.5 256:12.3 PAIR:12.2"),
    (2048, 1024, 4096, "res", "32S:44.6 32D:67.8 64S:27.2 64D:37.1 128D:24.6 256:33.3 PAIR:28.9"),
    (3000, 1024, 1024, "gelu", "32S:21.1 32D:29.9 64S:16.6 64D:18.0 128D:16.3 256:15.9 PAIR:14.9"),
    (512, 4096, 1024, "gelu", "64S:11.5 64D:13.9 128D:11.8 256:15.9 PAIR:14.2"),
    (768, 3072, 256, "plain", "64S:7.4 64D:7.8 128D:7.7 256:10.8 PAIR:8.8"),
    (1000, 8192, 512, "relu", "64S:18.3 64D:21.7 128D:19.0 256:18.7 PAIR:15.9"),
    (4096, 1536, 128, "res", "64S:14.9 64D:13.9 128D:13.9 256:18.3 PAIR:13.5"),
    (8192, 2304, 64, "res", "64S:34.4 64D:31.4 128D:30.3 256:32.7 PAIR:23.8"),
    (8192, 3072, 768, "gelu", "64S:60.2 64D:77.4 128D:52.5 256:55.7 PAIR:43.3"),
    (4662, 2304, 4096, "f32", "64S:117.7 64D:149.8 128D:100.1 256:88.3"),
    (8192, 4096, 2048, "plain", "64S:182.3 64D:261.9 128D:138.5 256:101.4 PAIR:101.7"),
    (4662, 8193, 128, "rag", "64D:90.7 128D:93.8 256:95.5 PAIR:64.4"),
    (2048, 769, 512, "rag", "32D:11.9 64D:9.5 128D:9.1 256:13.2 PAIR:12.5"),
    (8192, 193, 1024, "rag", "32D:22.1 64D:13.9 128D:11.5 256:15.2 PAIR:14.9"),
    (8192, 8192, 1024, "relu", "64S:189.8 64D:267.6 128D:153.1 256:111.6 PAIR:114.4"),
]


@pytest.mark.parametrize("M,N,K,variant,times", _MEASURED)
def test_the_chosen_form_is_near_the_fastest(M, N, K, variant, times):
    us = {}
    for entry in times.split():
        name, t = entry.split(":")
        us[PAIR | 256 if name == "PAIR" else int(name.rstrip("SD")) | _NAMES[name.lstrip("0123456789")]] = float(t)
    f = form(M, N, K, "gelu" if "gelu" in variant else "relu" if variant == "relu" else "", "res" in variant, variant == "f32",
             ldc=N if variant == "rag" else None)
    assert f in us and us[f] <= 1.1 * min(us.values())


# few rows: microseconds of the skinny and of the tcgen05 kernel, weights from DRAM, short and long K, on both sides of the line
@pytest.mark.parametrize("M,N,K,skinny,umma", [
    (1, 10, 64, 1.4, 3.6), (8, 50257, 1024, 19.3, 43.5), (16, 1024, 4096, 6.2, 18.5), (12, 8192, 8192, 40.0, 37.1),
    (32, 1024, 1024, 2.8, 7.0), (48, 2304, 768, 6.3, 6.5), (64, 3072, 1024, 10.1, 7.5), (72, 2304, 768, 9.3, 6.4),
    (64, 8192, 64, 9.1, 3.8), (96, 16384, 64, 19.7, 5.2), (32, 50257, 64, 18.4, 10.3), (56, 512, 8192, 10.7, 33.9),
    (64, 1024, 4096, 11.9, 18.7), (96, 768, 3072, 10.4, 14.7), (96, 4096, 256, 10.3, 4.7), (32, 1024, 8192, 11.4, 34.0),
    (17, 3072, 3072, 12.9, 22.6), (96, 2304, 2048, 21.0, 11.1)])
def test_few_rows_take_the_faster_kernel(M, N, K, skinny, umma):
    taken = skinny if form(M, N, K) == SKINNY else umma
    assert taken <= 1.1 * min(skinny, umma)


# the vocabulary of very narrow models: microseconds with the norm in front, fused into the few-rows kernel or on its own with
# the tcgen05 kernel
@pytest.mark.parametrize("M,N,K,fused,apart", [(1, 50257, 64, 11.4, 8.7), (8, 50257, 128, 12.2, 10.7), (4, 32000, 64, 7.6, 6.9),
                                               (8, 32000, 128, 8.7, 8.1), (1, 16384, 64, 5.4, 7.0), (8, 16384, 128, 5.7, 7.4), (4, 50257, 256, 12.8, 14.1),
                                               (8, 50257, 1024, 20.0, 44.0)])
def test_logits_of_a_few_rows(M, N, K, fused, apart):
    from ronn_b200.ops.kernels import norm_gemm_ok
    ok = norm_gemm_ok(M, K, N)
    assert (fused if ok else apart) == min(fused, apart) and (form(M, N, K) == SKINNY) == ok
    assert norm_gemm_ok(M, K)                                # the kernel takes the size either way


# microseconds with the norm that follows: one skinny launch and a norm kernel, four K slices and a reduction with the norm
@pytest.mark.parametrize("rows,n,k,one,slices", [
    (1, 1024, 4096, 6.9, 10.2), (16, 1024, 4096, 8.3, 10.2), (16, 4096, 2048, 10.2, 12.8), (32, 1024, 4096, 9.5, 10.2),
    (48, 768, 2048, 7.0, 8.5), (64, 512, 8192, 13.1, 14.1), (48, 1024, 2048, 9.3, 8.3), (48, 1024, 4096, 13.5, 10.4),
    (80, 512, 4096, 11.4, 10.4), (32, 2048, 2048, 10.7, 8.8), (64, 1024, 2048, 10.2, 8.5), (96, 512, 4096, 12.0, 10.5),
    (128, 256, 2048, 13.4, 9.2), (128, 256, 4096, 21.1, 11.1), (256, 256, 2048, 13.4, 9.2), (512, 512, 2048, 14.0, 10.0)])
def test_down_projections_take_the_faster_way(rows, n, k, one, slices):
    from ronn_b200.ops.kernels import skinny_down_ok
    ok = skinny_down_ok(rows, n, k)
    assert (one if ok else slices) <= 1.05 * min(one, slices)
    assert not ok or form(rows, n, k, residual=True) == SKINNY


def test_calls_between_the_rows_of_a_tile():
    """Every count of rows and columns gives a form that the launcher has, also far outside the measured range."""
    known = {w | r for w in (32, 64, 128) for r in (DEEP, SHALLOW)} | {256, PAIR | 256, SKINNY}
    for M in (1, 17, 97, 128, 257, 1023, 1024, 1025, 100000, 2 ** 30):
        for N in (1, 7, 32, 33, 64, 65, 128, 129, 50257, 2 ** 30):
            for fp32 in (False, True):
                f = form(M, N, 8, fp32=fp32, ldc=N)
                assert f in known and not (fp32 and f & PAIR), (M, N, fp32, hex(f))


# the grids of these forms, and the rules that choose them, count two CTAs per SM: registers have to fit as well
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [0, 1])
def test_two_ctas_fit_an_sm(dtype):
    lib = _native.cuda()
    for bn in (32, 64, 128):
        assert lib.ronn_gemm_ctas_per_sm(bn | SHALLOW, dtype) >= 2 and lib.ronn_gemm_ctas_per_sm(bn | DEEP, dtype) == 1
    assert lib.ronn_gemm_ctas_per_sm(256, dtype) == 1
    for bn, per_sm in ((32, 2), (64, 2), (128, 1)):
        assert lib.ronn_conv2d_ctas_per_sm(0, bn, dtype) >= per_sm
    assert lib.ronn_conv2d_ctas_per_sm(1, 64, dtype) == 2 and lib.ronn_conv2d_ctas_per_sm(1, 128, dtype) == 1
