"""The one-rank quantiser kernels that hold error-feedback state keep their tiles in registers."""
import os
import re
import shutil
import subprocess

import pytest

from hipress_b200._native.build import CSRC, NVCC_FLAGS, nvcc_path

HAVE_NVCC = shutil.which("nvcc") is not None or os.path.exists("/usr/local/cuda/bin/nvcc")


@pytest.mark.skipif(not HAVE_NVCC, reason="nvcc not available")
def test_one_rank_kernels_with_state_do_not_spill(tmp_path):
    r = subprocess.run([nvcc_path(), *NVCC_FLAGS, "-I", str(CSRC / "include"), "-I", str(CSRC / "cuda"), "-c",
                        str(CSRC / "cuda/fused_dense.cu"), "-o", str(tmp_path / "x.o")], capture_output=True, text=True, check=True)
    found = 0
    for name, body in re.findall(r"Compiling entry function '(\S+)'(.*?)(?=Compiling|\Z)", r.stderr, re.S):
        # the last template argument of local_dense_kernel: whether, or which, state is kept
        m = re.search(r"local_dense_kernelI(?:Li\d+E){3}L[bi](\d)E", name)
        if m and m[1] != "0":
            found += 1
            assert re.search(r"(\d+) bytes spill stores", body)[1] == "0", (name, body)
    assert found
