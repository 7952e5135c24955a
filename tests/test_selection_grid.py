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
def chain_ctas(tmp_path_factory):
    so = tmp_path_factory.mktemp("grid") / "chain_grid.so"
    subprocess.run([nvcc_path(), *[f for f in NVCC_FLAGS if f not in ("-Xptxas", "-v")], "-shared", "-I", str(CSRC / "include"),
                    "-I", str(CSRC / "cuda"), str(Path(__file__).parent / "native/chain_grid.cu"), "-o", str(so)], check=True)
    L = C.CDLL(str(so))

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
