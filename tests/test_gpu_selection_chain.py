"""The top-k encode as a chain of launches, at the edges of its half tiles and list parts,
against the CPU oracle."""
import pytest
import torch

from hipress_b200.ops import Compressor, sparse_pairs

pytestmark = pytest.mark.gpu


def _off(t, words):
    """A copy `words` floats behind a 16-byte boundary."""
    return torch.cat([torch.zeros(4 + words), t]).cuda()[4 + words:]


@pytest.mark.parametrize("name", ["dgc", "graddrop"])
# around a half tile and a tile; sampled whole and in part; vectors and single elements
@pytest.mark.parametrize("n", [2047, 2048, 2049, 4095, 4097, 4 * 4096 + 2048, 9 * 4096 + 2049, 300 * 4096 + 1])
@pytest.mark.parametrize("ratio,off", [(0.002, 0), (0.02, 1), (0.6, 0)])
def test_chain_at_its_edges(name, n, ratio, off):
    gen = torch.Generator().manual_seed(n)
    c = Compressor(name, ratio=ratio)
    st_c = c.new_state(n, "cpu")
    for v in st_c.values():
        v.copy_(torch.randn(n, generator=gen) * 0.1)
    st_g = {k: _off(v, off) for k, v in st_c.items()}
    ws = c.new_workspace("cuda", n)
    for _ in range(2):
        g = torch.randn(n, generator=gen) * torch.randn(n, generator=gen)
        ic, vc = sparse_pairs(c.encode(g, st_c), c.kmax(n))
        ig, vg = sparse_pairs(c.encode(_off(g, off), st_g, workspace=ws), c.kmax(n))
        assert torch.equal(ic, ig) and torch.equal(vc, vg)
        for key in st_c:
            assert torch.equal(st_g[key].cpu(), st_c[key]), key


@pytest.mark.parametrize("what", ["equal", "clustered", "zeros", "infinite"])
def test_chain_where_the_list_does_not_hold_them(what):
    """Lists that overflow or come out short: the digits are counted over the whole array."""
    n, ratio = 70 * 4096 + 33, 0.01
    c = Compressor("graddrop", ratio=ratio)
    g = torch.randn(n, generator=torch.Generator().manual_seed(1)) * 1e-3
    if what == "equal":
        g = torch.full((n,), 0.5)
    elif what == "clustered":
        g[5 * 4096:6 * 4096] += 3.0
    elif what == "zeros":
        g = torch.zeros(n)
        g[4000:4100] = 1.0
    else:
        g[::5000] = float("inf")
    k = c.kmax(n)
    st = c.new_state(n, "cuda")
    idx, val = sparse_pairs(c.encode(g.cuda(), st, workspace=c.new_workspace("cuda", n)), k)
    want = g.abs().topk(k).values
    want = want[want != 0]
    assert idx.numel() == want.numel() and idx.unique().numel() == idx.numel()
    assert torch.equal(val.abs().sort(descending=True).values, want)
    assert torch.equal(g[idx], val)
    left = g.clone()
    left[idx] = 0.0
    assert torch.equal(st["residual"].cpu(), left)
