"""Which kernels a top-k selection of one rank takes, and that they are not the slower ones."""
import pytest
import torch

from hipress_b200.ops import Compressor, sparse_pairs
from hipress_b200.parallel.fused_sparse import FusedSparseBucket

pytestmark = pytest.mark.gpu


def _us(f, reps):
    a, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    for _ in range(reps):
        f()
    e.record()
    torch.cuda.synchronize()
    return a.elapsed_time(e) * 1e3 / reps


# two large arrays, of which many elements are sent: an array's CTAs count the same words
@pytest.mark.parametrize("name,topology,ratio", [("dgc", "ps", 0.03), ("graddrop", "ps", 0.03), ("graddrop", "ring", 0.05)])
def test_chain_of_large_arrays_is_no_slower_than_the_persistent_kernels(name, topology, ratio):
    sizes, c = [10_000_000] * 2, Compressor(name, ratio=ratio)
    runs = []
    for ctas in (0, 1024):     # 0: a chain of launches
        b = FusedSparseBucket(c.spec, sizes, 1, 0, topology=topology, ctas=ctas).bind_local("cuda")
        g = [torch.randn(n, device="cuda", generator=torch.Generator("cuda").manual_seed(n)) for n in sizes]
        out, sums = [torch.empty_like(x) for x in g], [torch.zeros_like(x) for x in g]
        st = [c.new_state(n, "cuda") for n in sizes]
        acc = "accum_v" if name == "dgc" else "residual"
        args = ([s[acc].data_ptr() for s in st], [s["momentum_u"].data_ptr() for s in st] if name == "dgc" else None,
                [x.data_ptr() for x in out], [x.data_ptr() for x in sums])
        h = [-x for x in g]     # gradients that cancel, so that the state stays as it is

        def run(b=b, args=args, g=g, h=h, keep=(out, sums, st)):
            b.launch_ptrs([x.data_ptr() for x in g], *args)
            b.launch_ptrs([x.data_ptr() for x in h], *args)
        runs.append(run)
    best = [1e9, 1e9]
    for _ in range(5):         # in turn
        for i in range(2):
            best[i] = min(best[i], _us(runs[i], 10))
    assert best[0] < 1.05 * best[1], best


# around one tile; around 42 M elements, where the share of the elements that are sent decides, and the update
@pytest.mark.parametrize("name,n,ratio,chain,chain_without_update", [
    ("dgc", 1, 0.5, 0, 0), ("dgc", 4096, 0.01, 0, 0), ("dgc", 4097, 0.01, 1, 1), ("graddrop", 4096, 0.5, 0, 0),
    ("graddrop", 4097, 0.001, 1, 1), ("graddrop", 10240 * 4096, 0.0002, 1, 1), ("graddrop", 10240 * 4096 + 1, 0.0002, 0, 0),
    ("graddrop", 10240 * 4096 + 1, 0.001, 0, 1), ("graddrop", 10240 * 4096 + 1, 0.002, 1, 1),
    ("dgc", 10240 * 4096 + 1, 0.0002, 1, 0), ("dgc", 10240 * 4096 + 1, 0.001, 1, 1)])
def test_routes_of_an_encode(name, n, ratio, chain, chain_without_update):
    """Sizes at which the persistent kernel is the faster one are its own again.  The counts
    of a chain's list parts are words of the workspace that the persistent kernel leaves zero."""
    c = Compressor(name, ratio=ratio)
    ws, k = c.new_workspace("cuda", n), c.kmax(n)
    for update in (True, False):
        g = torch.randn(n, device="cuda")
        st = c.new_state(n, "cuda")
        if not update:
            st["accum_v" if name == "dgc" else "residual"].copy_(g)
        pay = c.encode(g, st, workspace=ws, update=update)
        words = ws.view(torch.int32)
        head = 3 * 4096 + 16 + 160            # kWsWords, then kBarrierWords
        assert bool(words[head:head + 32 * 7].any()) == bool(chain if update else chain_without_update)
        idx, val = sparse_pairs(pay, k)
        want = g.abs().topk(k).values
        assert torch.equal(val.abs().sort(descending=True).values, want.cpu())
        assert torch.equal(g.cpu()[idx], val)


def test_chain_whose_list_overflows_is_no_slower_than_the_persistent_kernel():
    """Large values that lie together in a hundredth of the array: the sample sees few of them."""
    n, c = 6553600, Compressor("graddrop", ratio=0.001)
    g = torch.randn(n, device="cuda", generator=torch.Generator("cuda").manual_seed(1)) * 1e-3
    g[:n // 100] *= 1e3
    st, ws = c.new_state(n, "cuda"), c.new_workspace("cuda", n)
    pay = torch.empty(c.payload_bytes(n), dtype=torch.uint8, device="cuda")
    times = [[], []]
    for _ in range(15):        # in turn
        for i, ctas in enumerate((0, 10 ** 6)):
            st["residual"].zero_()
            times[i].append(_us(lambda: c.encode(g, st, workspace=ws, out=pay, max_ctas=ctas), 1))
            assert int(ws.view(torch.int32)[3 * 4096 + 5]) != 0      # kWsOverflow
    mid = [sorted(t)[len(t) // 2] for t in times]
    assert mid[0] < 1.1 * mid[1], mid


@pytest.mark.parametrize("name", ["dgc", "graddrop"])
@pytest.mark.parametrize("max_ctas", [1, 40, 10 ** 6])     # the last: as wide as the GPU is
def test_persistent_kernel_at_its_widths(name, max_ctas):
    n, c = 300 * 4096 + 5, Compressor(name, ratio=0.01)
    gen = torch.Generator().manual_seed(max_ctas)
    cpu, dev, ws = c.new_state(n, "cpu"), c.new_state(n, "cuda"), c.new_workspace("cuda", n)
    for _ in range(2):
        g = torch.randn(n, generator=gen) * torch.randn(n, generator=gen)
        want = sparse_pairs(c.encode(g, cpu), c.kmax(n))
        got = sparse_pairs(c.encode(g.cuda(), dev, workspace=ws, max_ctas=max_ctas), c.kmax(n))
        assert all(torch.equal(a, b) for a, b in zip(want, got))
        assert all(torch.equal(dev[k].cpu(), cpu[k]) for k in cpu)
