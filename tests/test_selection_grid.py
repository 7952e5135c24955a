"""The launch that emits a top-k selection is wide enough for the passes over whole arrays
that its CTAs make together where a list came out short."""
import ctypes as C
import os
import shutil
import subprocess
from pathlib import Path

import pytest

from hipress_b200._native.build import CSRC, NVCC_FLAGS, nvcc_path

HAVE_NVCC = shutil.which("nvcc") is not None or os.path.exists("/usr/local/cuda/bin/nvcc")
TILE = 4096


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    so = tmp_path_factory.mktemp("grid") / "chain_grid.so"
    subprocess.run([nvcc_path(), *[f for f in NVCC_FLAGS if f not in ("-Xptxas", "-v")], "-shared", "-I", str(CSRC / "include"),
                    "-I", str(CSRC / "cuda"), str(Path(__file__).parent / "native/chain_grid.cu"), "-o", str(so)], check=True)
    return C.CDLL(str(so))


@pytest.fixture(scope="module")
def chain_ctas(library):
    L = library

    def f(units, n, k, sms):
        emitters = C.c_uint32()
        return L.chain_ctas(units, C.c_uint32(n), C.c_uint32(k), 2, sms, C.byref(emitters)), emitters.value
    return f


@pytest.mark.skipif(not HAVE_NVCC, reason="nvcc not available")
@pytest.mark.parametrize("sms", [16, 148])
def test_whole_array_passes_have_the_gpu(chain_ctas, sms):
    for units, n, k in [(1, 1, 1), (1, 1 << 20, 1049), (1, 6553600, 6554), (1, 1 << 24, 16777), (1, 1 << 24, 167773),
                        (4, 65536, 66), (4, 1 << 20, 1049), (2, 1 << 24, 1 << 24)]:
        ctas, emitters = chain_ctas(units, n, k, sms)
        tiles = units * -(-n // TILE)
        assert emitters <= ctas <= 2 * sms, (units, n, k)     # they wait for one another
        assert ctas >= min(tiles, sms), (units, n, k)
    assert chain_ctas(2 * sms // 7 + 1, 5000, 5, sms)[0] == 0     # the persistent kernels take those


@pytest.mark.skipif(not HAVE_NVCC, reason="nvcc not available")
@pytest.mark.parametrize("sms", [16, 148, 500])
@pytest.mark.parametrize("n", [[20_000_000] + [500] * 3, [500] * 30 + [20_000_000], [1 << (24 - i) for i in range(16)], [4096] * 40,
                               [0xFFFFF000], [1 << 20] * 6])
@pytest.mark.parametrize("part", [1000, 10, 1])
def test_a_list_is_emitted_by_ctas_as_its_length_asks(library, sms, n, part):
    k = [-(-x // part) for x in n]
    u32 = C.c_uint32 * len(n)
    ctas, most = u32(), 2 * sms // 7
    total = library.chain_shares(len(n), u32(*n), u32(*k), 2, sms, ctas)
    if most < len(n):
        assert total == 0       # the persistent kernels take those
        return
    assert sum(ctas) <= total <= 2 * sms and min(ctas) >= 7
    # as many as one round of its candidates takes (2048 a CTA), or its share of what there is
    want = [7 * (x * 3 // 2 // (2048 * 7)) for x in k]
    spare = 7 * (min(most, 64) - len(n))
    for c, w in zip(ctas, want):
        assert c >= 7 + min(w, w * spare // max(1, sum(want))) // 7 * 7, (list(ctas), want)
        assert c <= 7 + w
