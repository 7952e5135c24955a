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


@pytest.mark.parametrize("bits", [1, 2, 4, 8])
# which of two tensors keep state: the sender's; the owner's; both; one tensor each; one both, one none
@pytest.mark.parametrize("sender,owner", [((1, 1), (0, 0)), ((0, 0), (1, 1)), ((1, 1), (1, 1)), ((1, 0), (0, 1)),
                                          ((0, 1), (0, 0)), ((0, 1), (0, 1))])
def test_state_of_either_side(bits, sender, owner):
    gen = torch.Generator().manual_seed(bits)
    sizes = [6 * 4096 + 77, 3 * 4096]
    plain, kept = Compressor("terngrad", bitwidth=bits), Compressor("terngrad", bitwidth=bits, error_feedback=True)
    b = FusedDenseBucket(plain.spec, "ps", sizes, 1, 0).bind_local("cuda")
    state = [[torch.randn(n, generator=gen) * 0.01 if on else None for n, on in zip(sizes, side)] for side in (sender, owner)]
    dev = [[None if t is None else t.cuda() for t in side] for side in state]
    for step in range(2):
        grads = [torch.randn(n, generator=gen) for n in sizes]
        outs = [torch.empty(n, device="cuda") for n in sizes]
        b.launch([g.cuda() for g in grads], dev[0], outs, dev[1], step=step, tensor_ids=[4, 5])
        torch.cuda.synchronize()
        for i, n in enumerate(sizes):
            # the push, then the owner's pass over what it decodes to, as the oracle does one encode
            x = grads[i]
            for side in range(2):
                st = state[side][i]
                pay = (plain if st is None else kept).encode(x, {} if st is None else {"residual": st}, step=step, salt=side,
                                                             tensor_id=4 + i)
                x = plain.decode(pay, torch.zeros(n))
                if st is not None:
                    assert torch.equal(dev[side][i].cpu(), st), (step, i, side)
            assert torch.equal(outs[i].cpu(), x), (step, i)
