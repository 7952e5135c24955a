"""The one-launch top-k encoder and the one-launch decode at the edges of their ranges,
against the CPU oracle."""
import pytest
import torch

from hipress_b200.ops import Compressor, sparse_pairs

pytestmark = pytest.mark.gpu


def _check(name, g, ratio, steps=2, max_ctas=0):
    n = g.numel()
    c = Compressor(name, ratio=ratio)
    st_c, st_g = c.new_state(n, "cpu"), c.new_state(n, "cuda")
    ws = c.new_workspace("cuda", n)
    for _ in range(steps):
        pc = c.encode(g, st_c)
        pg = c.encode(g.cuda(), st_g, workspace=ws, max_ctas=max_ctas)
        k = c.kmax(n)
        ic, vc = sparse_pairs(pc, k)
        ig, vg = sparse_pairs(pg, k)
        assert torch.equal(ic, ig) and torch.equal(vc, vg)
        for key in st_c:
            assert torch.equal(st_g[key].cpu(), st_c[key]), key
        out_c, out_g = torch.empty(n), torch.full((n,), 7.0, device="cuda")
        c.decode(pc, out_c, scale=0.5)
        c.decode(pg, out_g, scale=0.5)
        assert torch.equal(out_g.cpu(), out_c)
        g = g.flip(0) * 0.7


@pytest.mark.parametrize("name", ["dgc", "graddrop"])
# below, at and above the size that is sampled whole; one tile and less; lists that one
# CTA finishes and lists that are refined first; payloads above the one-launch decode
@pytest.mark.parametrize("n,ratio", [(1, 0.5), (37, 0.1), (4096, 0.01), (65536, 0.001), (65537, 0.001),
                                     (1000003, 0.001), (3000001, 0.003), (600000, 0.05), (2000, 1.0)])
def test_selection_matches_oracle(name, n, ratio):
    torch.manual_seed(n)
    _check(name, torch.randn(n) * torch.randn(n), ratio)


def test_selection_with_few_ctas():
    torch.manual_seed(1)
    _check("dgc", torch.randn(500000) * torch.randn(500000), 0.002, max_ctas=3)


def test_selection_of_arrays_the_sample_misjudges():
    """Almost everything zero, the few large values in one place: the sample sees none of
    them, so the list is all that is not zero; and magnitudes the sample sees in full
    but the rest of the array does not have, so the list comes out short."""
    n = 1 << 20
    g = torch.zeros(n)
    g[70001:70001 + 900] = torch.linspace(1.0, 2.0, 900)
    _check("graddrop", g, 0.001, steps=1)
    torch.manual_seed(3)
    g = torch.randn(n) * 1e-3
    pieces = torch.arange(4096, dtype=torch.int64) * (n // 16) // 4096 * 16
    for q in range(16):
        g[pieces + q] = 1.0 + torch.rand(4096)
    g[5::97] *= 3.0
    _check("graddrop", g, 0.08, steps=1)


def test_selection_with_massive_ties_sends_exactly_k():
    n, ratio = 300000, 0.01
    c = Compressor("graddrop", ratio=ratio)
    g = (torch.randint(0, 3, (n,), generator=torch.Generator().manual_seed(2)).float() - 1.0).cuda()
    st = c.new_state(n, "cuda")
    k = c.kmax(n)
    idx, val = sparse_pairs(c.encode(g, st, workspace=c.new_workspace("cuda", n)), k)
    assert idx.numel() == k and idx.unique().numel() == k
    assert torch.equal(g.cpu()[idx], val) and bool((val != 0).all())
    assert int((st["residual"] != 0).sum()) == int((g != 0).sum()) - k


def test_selection_with_a_workspace_off_alignment():
    """Four bytes off: the launch that reads its counters 16 bytes at a time is not taken."""
    n = 100003
    torch.manual_seed(2)
    g, c = torch.randn(n), Compressor("graddrop", ratio=0.01)
    ws = torch.cat([c.new_workspace("cuda", n), torch.zeros(1, dtype=torch.int32, device="cuda")])[1:]
    ic, vc = sparse_pairs(c.encode(g, c.new_state(n, "cpu")), c.kmax(n))
    ig, vg = sparse_pairs(c.encode(g.cuda(), c.new_state(n, "cuda"), workspace=ws), c.kmax(n))
    assert torch.equal(ic, ig) and torch.equal(vc, vg)
