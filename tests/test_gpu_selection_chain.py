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


# large values that lie together: one row of 1024; a block of columns of a matrix whose rows
# are as long as the parts' turns; one half tile; the first hundredth; an array of one half
# tile, most of which is sent
@pytest.mark.parametrize("what", ["row", "columns", "half tile", "hundredth", "small"])
def test_concentrated_values_fit_the_list(what):
    n, ratio = 1 << 20, 0.001
    gen = torch.Generator().manual_seed(3)
    if what == "hundredth":
        n, ratio = 6553600, 0.0005
    elif what == "small":
        n, ratio = 2048, 0.9
    c = Compressor("graddrop", ratio=ratio)
    k = c.kmax(n)
    g = torch.randn(n, generator=gen)
    if what == "row":
        g[:300 * 1024] = 0.0
        g[301 * 1024:] = 0.0
    elif what == "columns":
        g *= 1e-3
        g[:n // 14336 * 14336].view(-1, 14336)[:, :20] += 1.0
    elif what == "half tile":
        g *= 1e-3
        g[6 * 2048:6 * 2048 + 1500] += 3.0
    elif what == "hundredth":
        g *= 1e-3
        g[:2 * k] *= 1e3
    st, ws = c.new_state(n, "cuda"), c.new_workspace("cuda", n)
    idx, val = sparse_pairs(c.encode(g.cuda(), st, workspace=ws), k)
    ic, vc = sparse_pairs(c.encode(g, c.new_state(n, "cpu")), k)
    assert torch.equal(idx, ic) and torch.equal(val, vc)
    # the word that says that the list did not hold them (kWsOverflow): no pass over the
    # whole array behind the update
    assert int(ws.view(torch.int32)[3 * 4096 + 5]) == 0


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


@pytest.mark.parametrize("topology", ["ps", "ring"])
@pytest.mark.parametrize("name", ["dgc", "graddrop"])
# one array; arrays of very different sizes; as many as a bucket holds, the smallest of one element
@pytest.mark.parametrize("sizes", [[300003], [200003, 8192, 300, 1 << 18, 4096], [1, 7000] + [3000 + 37 * i for i in range(38)]])
def test_buckets_of_one_rank(name, topology, sizes):
    from hipress_b200.parallel.fused_sparse import FusedSparseBucket
    from hipress_b200.parallel.simulate import chunk_elems, simulate_ps, simulate_ring
    gen = torch.Generator().manual_seed(len(sizes))
    c = Compressor(name, ratio=0.01)
    b = FusedSparseBucket(c.spec, sizes, 1, 0, topology=topology).bind_local("cuda")
    acc = "accum_v" if name == "dgc" else "residual"
    cpu = [c.new_state(s, "cpu") for s in sizes]
    srv = [{"residual": torch.zeros(chunk_elems(s, 1))} for s in sizes]
    gpu = [{k: v.cuda() for k, v in st.items()} for st in cpu]
    sums = [x["residual"].cuda() for x in srv]
    for step in range(3):
        grads = [torch.randn(s, generator=gen) * torch.randn(s, generator=gen) for s in sizes]
        dev = [g.cuda() for g in grads]       # the result takes the gradient's place
        b.launch_ptrs([g.data_ptr() for g in dev], [s[acc].data_ptr() for s in gpu],
                      [s["momentum_u"].data_ptr() for s in gpu] if name == "dgc" else None,
                      [g.data_ptr() for g in dev], [s.data_ptr() if topology == "ps" else None for s in sums])
        torch.cuda.synchronize()
        b.check_status()
        for i in range(len(sizes)):
            ref = simulate_ps(c, [grads[i]], [cpu[i]], [srv[i]]) if topology == "ps" else \
                simulate_ring(c, [grads[i]], [cpu[i]])
            assert torch.allclose(dev[i].cpu(), ref[0], rtol=1e-5, atol=1e-7), (step, i)
            for k in cpu[i]:
                assert torch.allclose(gpu[i][k].cpu(), cpu[i][k], rtol=1e-5, atol=1e-7), (step, i, k)
            if topology == "ps":
                assert torch.allclose(sums[i].cpu(), srv[i]["residual"], rtol=1e-5, atol=1e-7), (step, i)


@pytest.mark.parametrize("topology", ["ps", "ring"])
@pytest.mark.parametrize("name", ["dgc", "graddrop"])
# which arrays' lists overflow: the largest; some, of different sizes; all
@pytest.mark.parametrize("full", [[0], [1, 3, 6], list(range(8))])
def test_buckets_where_some_arrays_take_the_whole_array_passes(name, topology, full):
    from hipress_b200.parallel.fused_sparse import FusedSparseBucket
    gen = torch.Generator().manual_seed(len(full))
    sizes = [600007, 70001, 9000, 1 << 17, 20480, 33333, 16384, 50000]
    c = Compressor(name, ratio=0.001)
    b = FusedSparseBucket(c.spec, sizes, 1, 0, topology=topology).bind_local("cuda")
    acc = "accum_v" if name == "dgc" else "residual"
    st = [c.new_state(s, "cuda") for s in sizes]
    sums = [torch.zeros(s, device="cuda") for s in sizes]
    left = [torch.zeros(s) for s in sizes]
    for step in range(2 if name == "graddrop" else 1):
        grads = [torch.randn(s, generator=gen) * torch.randn(s, generator=gen) for s in sizes]
        for i in full:      # two values: far more ties than a list holds, but for the first few
            grads[i] = torch.where(torch.rand(sizes[i], generator=gen) < 0.5, -1.0, 1.0)
            grads[i][:3] = 5.0
        out = [g.cuda() for g in grads]       # the result takes the gradient's place
        b.launch_ptrs([g.data_ptr() for g in out], [s[acc].data_ptr() for s in st],
                      [s["momentum_u"].data_ptr() for s in st] if name == "dgc" else None,
                      [g.data_ptr() for g in out], [s.data_ptr() for s in sums])
        torch.cuda.synchronize()
        b.check_status()
        for i, n in enumerate(sizes):
            # kWsOverflow of the push's unit
            assert (int(b.ws[i * (3 * 4096 + 16) + 3 * 4096 + 5]) != 0) == (i in full), (step, i)
            total, got = left[i] + grads[i], out[i].cpu()
            sent = got.nonzero().flatten()
            want = total.abs().topk(c.kmax(n)).values
            assert torch.equal(got[sent].abs().sort(descending=True).values, want), (step, i)
            assert torch.equal(got[sent], total[sent]), (step, i)
            left[i] = total
            left[i][sent] = 0.0
            assert torch.equal(st[i][acc].cpu(), left[i]), (step, i)
            if name == "dgc":                 # the momentum of what was sent starts anew
                assert torch.equal(st[i]["momentum_u"].cpu(), left[i]), i
            if topology == "ps":              # the owner sent all it was given
                assert not sums[i].any(), (step, i)
