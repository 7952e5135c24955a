"""Generated kernels where their loops without bounds tests begin and end, and the quotients
those loops take from products: the same bits as the C++ target and as `/`."""
import ctypes as C
import subprocess

import numpy as np
import pytest
import torch

from hipress_b200.compll import load_op
from hipress_b200._native.build import CSRC, GXX_FLAGS


@pytest.fixture(scope="module")
def quotients(tmp_path_factory):
    d = tmp_path_factory.mktemp("div")
    (d / "div.cpp").write_text("""
#include "hipress/compll_rt.cuh"
extern "C" void quotients(const float* a, float b, float* q, unsigned* bad, long n, int* ok) {
  const CompllDivisor d = compll_divisor(b);
  *ok = d.ok;
  for (long i = 0; i < n; ++i) { uint32_t x = 0; q[i] = compll_div(a[i], d, x); bad[i] = x >> 31; }
}""")
    subprocess.run(["g++", *GXX_FLAGS, "-Wno-unknown-pragmas", "-I", str(CSRC / "include"), "-shared", "-o", str(d / "div.so"),
                    str(d / "div.cpp")], check=True)
    L = C.CDLL(str(d / "div.so"))

    def f(a, b):
        q, bad, ok = np.empty_like(a), np.empty(a.size, np.uint32), C.c_int()
        L.quotients(a.ctypes.data_as(C.c_void_p), C.c_float(b), q.ctypes.data_as(C.c_void_p),
                    bad.ctypes.data_as(C.c_void_p), C.c_long(a.size), C.byref(ok))
        return q, bad != 0, bool(ok.value)
    return f


def test_quotients_round_as_division_does(quotients):
    rng = np.random.default_rng(0)
    hard = np.array([0x800000, 0x800001, 0xFFFFFF, 0xFFFFFE, 0xAAAAAA, 0xAAAAAB, 0xD55555, 0xC00000, 0xB504F3], np.uint32)
    for t in range(400):
        m = hard[t % hard.size] if t < 200 else rng.integers(1 << 23, 1 << 24)
        b = np.float32(np.ldexp(np.float64(m), int(rng.integers(-60, 61)) - 23))
        a = rng.integers(1 << 23, 1 << 24, 20000).astype(np.float64)
        a[:hard.size] = hard
        # neighbours of exact multiples of b and of half steps between them, the closest cases
        k = rng.integers(1 << 23, 1 << 25, 4000).astype(np.float64) / 2
        a[1000:5000] = np.frexp(k * float(m))[0] * (1 << 24)
        a = np.ldexp(np.rint(a), rng.integers(-63, 64, a.size) - 23).astype(np.float32)
        a *= rng.choice(np.array([-1, 1], np.float32), a.size)
        q, bad, ok = quotients(a, b)
        assert ok and not bad.any()
        assert np.array_equal((a / b).view(np.uint32), q.view(np.uint32))


def test_quotients_that_may_be_inexact_are_marked(quotients):
    for b in (0.0, -1.0, np.inf, np.nan, 2.0 ** -61, 2.0 ** 61, 1e-42):
        assert not quotients(np.ones(1, np.float32), b)[2], b
    a = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 2.0 ** -64, -2.0 ** 65, 1e-42], np.float32)
    assert quotients(a, 0.37)[1].all()
    assert not quotients(np.array([2.0 ** -63, -(2.0 ** 65 - 2.0 ** 41)], np.float32), 0.37)[1].any()


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [1, 2, 4, 8])
@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 592 * 1024 - 4, 592 * 1024 + 5, 3 * 592 * 1024 + 700])
def test_terngrad_encode_has_the_bits_of_the_cpu_target(n, bits):
    enc = load_op("TernGradEncode")
    torch.manual_seed(n)
    g = torch.randn(n + 1) * torch.randn(n + 1)
    sparse = torch.relu(g)        # most elements are the minimum: their quotient is zero
    cases = [g[:n], g[1:] * 1e-3, sparse[:n], torch.full((n,), 0.25), g[:n] * 1e-30, g[:n] * 1e30, g[:n] * 1e-40]
    for i, x in enumerate(cases):
        for off in (0, 1):         # the payload on and off a word boundary
            want = torch.zeros(off + 10 + (n * bits + 7) // 8, dtype=torch.uint8)
            enc(x.contiguous(), want[off:], bits, seed=5)
            got = torch.zeros_like(want, device="cuda")
            # case 1 lies off a 16-byte boundary
            xg = torch.cat([x[:1], x]).cuda()[1:] if i == 1 else x.cuda()
            enc(xg, got[off:], bits, seed=5)
            assert torch.equal(got.cpu(), want), (i, off)
