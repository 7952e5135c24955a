"""One rank, TernGrad through PS: the server's quantisation made from the push's codes gives
the bits of decoding them and quantising the values."""
import pytest
import torch

from hipress_b200.ops import Compressor
from hipress_b200.parallel.fused import FusedDenseBucket
from hipress_b200.parallel.simulate import simulate_ps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 2, 4, 8])
# offset, tiny step: levels that lie a few or less than one unit in the last place apart;
# relu: the minimum many times; jump: one value far above the rest, so that levels are missing
@pytest.mark.parametrize("what", ["normal", "offset", "close", "collapsed", "constant", "relu", "jump", "tiny", "huge",
                                  "nan", "inf"])
def test_server_codes_from_push_codes(bits, what):
    gen = torch.Generator().manual_seed(bits)
    n = 48 * 4096 + 77
    c = Compressor("terngrad", bitwidth=bits)
    b = FusedDenseBucket(c.spec, "ps", [n], 1, 0).bind_local("cuda")
    for step in range(3):
        g = torch.randn(n, generator=gen) * torch.rand(n, generator=gen) * 0.02
        if what == "offset":
            g += 3.0
        elif what == "close":
            g = 1.0 + g * 1e-4
        elif what == "collapsed":
            g = 1.0 + (g > 0).float() * 2.0 ** -22
        elif what == "constant":
            g[:4096 * 20] = 0.25
        elif what == "relu":
            g = g.relu()
        elif what == "jump":
            g[::4096] = 5.0
        elif what == "tiny":
            g *= 1e-36
        elif what == "huge":
            g *= 1e39
        elif what == "nan":
            g[5::9000] = float("nan")
        elif what == "inf":
            g[7::9000] = float("inf")
        ref = simulate_ps(c, [g.clone()], [{}], [{}], step=step, tensor_id=4)[0]
        out = torch.full((n,), 7.0, device="cuda")
        b.launch([g.cuda()], None, [out], None, step=step, tensor_ids=[4])
        torch.cuda.synchronize()
        got = out.cpu()
        same = (got == ref) | (got.isnan() & ref.isnan())
        assert bool(same.all()), (step, int((~same).sum()), got[~same][:4], ref[~same][:4])
