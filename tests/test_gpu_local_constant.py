"""One rank, TernGrad through PS: tiles of one value, whose second quantisation needs no work."""
import pytest
import torch

from hipress_b200.ops import Compressor
from hipress_b200.parallel.fused import FusedDenseBucket
from hipress_b200.parallel.simulate import simulate_ps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 2, 4, 8])
# span: extremes that differ by less than a step can be told apart; nan: a NaN among equal values
@pytest.mark.parametrize("what", ["zero", "negative zero", "both zeros", "tiny", "huge", "span", "nan", "inf"])
def test_constant_tiles(bits, what):
    n = 5 * 4096 + 77
    c = Compressor("terngrad", bitwidth=bits)
    b = FusedDenseBucket(c.spec, "ps", [n], 1, 0).bind_local("cuda")
    g = torch.randn(n, generator=torch.Generator().manual_seed(bits))
    v = g[4096:4 * 4096]
    v.fill_({"negative zero": -0.0, "tiny": 1e-42, "huge": -3e38, "span": 1.0, "nan": -0.75, "inf": float("inf")}.get(what, 0.0))
    if what == "both zeros":
        v[::3] = -0.0
    elif what == "span":
        v.fill_(0.0)
        v[7::100] = 1e-45
    elif what == "nan":
        v[::500] = float("nan")
    ref = simulate_ps(c, [g.clone()], [{}], [{}], step=3, tensor_id=4)[0]
    out = torch.full((n,), 7.0, device="cuda")
    b.launch([g.cuda()], None, [out], None, step=3, tensor_ids=[4])
    got = out.cpu()
    same = (got.view(torch.int32) == ref.view(torch.int32)) | (got.isnan() & ref.isnan())
    assert bool(same.all()), (int((~same).sum()), got[~same][:4], ref[~same][:4])


@pytest.mark.parametrize("bits", [1, 2, 8])
def test_constant_tiles_cost_no_more_than_others(bits):
    n = 8192 * 4096
    b = FusedDenseBucket(Compressor("terngrad", bitwidth=bits).spec, "ps", [n], 1, 0).bind_local("cuda")
    grads = [torch.randn(n, device="cuda"), torch.zeros(n, device="cuda")]
    out = torch.empty(n, device="cuda")

    def us(g):
        a, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(20):
            b.launch([g], None, [out], None, step=1, tensor_ids=[4])
        e.record()
        torch.cuda.synchronize()
        return a.elapsed_time(e) * 50

    best = [1e9, 1e9]
    for _ in range(5):         # in turn
        for i in range(2):
            best[i] = min(best[i], us(grads[i]))
    # the same bytes and less arithmetic; a quarter for divisions of zero, which are slower
    assert best[1] < 1.25 * best[0], best
