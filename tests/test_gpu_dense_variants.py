"""Branches of the quantisers' kernels at the values and sizes where they can go wrong,
against the CPU oracle."""
import pytest
import torch

from hipress_b200.ops import Compressor

pytestmark = pytest.mark.gpu


def _payloads_equal(c, g, **kw):
    n = g.numel()
    pc = c.encode(g, c.new_state(n, "cpu"), step=3, tensor_id=2, **kw)
    pg = c.encode(g.cuda(), c.new_state(n, "cuda"), step=3, tensor_id=2, **kw)
    assert torch.equal(pg.cpu(), pc)
    oc, og = torch.empty(n), torch.empty(n, device="cuda")
    c.decode(pc, oc, scale=0.5)
    c.decode(pg, og, scale=0.5)
    assert torch.equal(torch.nan_to_num(og.cpu()), torch.nan_to_num(oc))


@pytest.mark.parametrize("bits", [1, 2, 4, 8])
@pytest.mark.parametrize("what", ["normal", "tiny", "huge", "constant", "nan", "inf", "overflow"])
def test_terngrad_codes_at_extreme_ranges(bits, what):
    """The floor by rounding-down addition and the saturating multiply against the
    element-wise definition: ranges whose scale is infinite, zero or subnormal, and
    values that are not finite."""
    torch.manual_seed(bits)
    n = 3 * 4096 + 77
    g = torch.randn(n) * 0.02
    if what == "tiny":
        g *= 1e-36
    elif what == "huge":
        g *= 1e38
    elif what == "constant":
        g[:4096] = 0.25
        g[4096:8192] = 0.0
    elif what == "nan":
        g[5] = g[5000] = float("nan")
    elif what == "inf":
        g[9] = float("inf")
        g[4100] = float("-inf")
    elif what == "overflow":
        g[0], g[1] = 3e38, -3e38
    _payloads_equal(Compressor("terngrad", bitwidth=bits), g)


def test_status_words_in_pinned_host_memory():
    """The training loop keeps the status words in pinned host memory: a wait that runs
    out shows there without a copy."""
    from hipress_b200.parallel.fused import FusedDenseBucket, HipressTimeoutError
    c = Compressor("tbq")
    n = 20000
    b = FusedDenseBucket(c.spec, "ring", [n], 2, 0, ctas=16, timeout_s=0.3)
    arena = torch.zeros(2 * b.region_bytes(), dtype=torch.uint8, device="cuda")
    status = torch.zeros(4, dtype=torch.int32).pin_memory()
    b.bind([arena.data_ptr(), arena.data_ptr() + b.region_bytes()], status)
    g = torch.randn(n, device="cuda") * 0.02
    b.launch_ptrs([g.data_ptr()], [torch.zeros_like(g).data_ptr()], [g.data_ptr()], [None])
    torch.cuda.synchronize()
    assert int(status[0]) != 0
    with pytest.raises(HipressTimeoutError):
        b.check_status()
