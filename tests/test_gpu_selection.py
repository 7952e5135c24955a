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


# around 96 tiles per CTA, where a CTA's tiles stop being one equal share of all
@pytest.mark.parametrize("tiles", [191, 192, 193, 400])
@pytest.mark.parametrize("name", ["dgc", "graddrop"])
def test_selection_with_tiles_that_are_handed_out(name, tiles):
    torch.manual_seed(tiles)
    n = tiles * 4096 - 5
    _check(name, torch.randn(n) * torch.randn(n), 0.002, max_ctas=2)


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


# the list's true length, 2048, cut by CTAs that each read another one: five slices that
# overlap and hold 2452 elements together; and a length beyond the list's room
@pytest.mark.parametrize("counts", [[511, 1023, 1535, 2047, 2048], [4096] * 8, [511, 4096, 1535, 4096, 2048, 4096]])
def test_emit_stays_in_its_lists_when_ctas_disagree_about_the_length(tmp_path, counts):
    import ctypes as C
    import subprocess
    from pathlib import Path
    from hipress_b200._native.build import CSRC, nvcc_path
    so = tmp_path / "emit_views.so"
    subprocess.run([nvcc_path(), "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-fmad=false",
                    "-Xcompiler", "-fPIC", "-shared", "-I", str(CSRC / "include"), "-I", str(CSRC / "cuda"),
                    str(Path(__file__).parent / "native/emit_views.cu"), "-o", str(so)], check=True)
    L = C.CDLL(str(so))
    n, cap, k = 8192, 2048, 1000
    # all candidates alike: every one is a tie and goes to the second list
    a = torch.ones(n, device="cuda")
    key = int(torch.ones(1).view(torch.int32).item())
    ws = torch.zeros(L.emit_workspace_words(), dtype=torch.int32, device="cuda")
    ws[0] = cap                            # histogram: all in the first bin above the bound
    # two lists of `cap` pairs, and behind them room for whatever the CTAs hold together
    guard = 0x5A5A5A5A
    lists = torch.full((4 * cap + 8 * max(counts),), guard, dtype=torch.int32, device="cuda")
    lists[:cap] = key
    lists[cap:2 * cap] = torch.arange(cap, dtype=torch.int32, device="cuda")
    out = torch.zeros(16 + 2 * 4 * (k + 4), dtype=torch.uint8, device="cuda")
    c = torch.tensor(counts, dtype=torch.int32, device="cuda")
    p = [C.c_void_p(t.data_ptr()) for t in (a, ws, lists, c, out)]
    rc = L.emit_views(p[0], C.c_uint32(n), C.c_uint32(k), p[1], p[2], C.c_uint32(cap), C.c_uint32(key), p[3],
                      C.c_int(len(counts)), p[4], C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    assert bool((lists[4 * cap:] == guard).all()), "the second list was written past its end"
    assert bool((lists[cap:2 * cap] == torch.arange(cap, dtype=torch.int32, device="cuda")).all())
    assert bool((a[cap:] == 1).all())


@pytest.mark.parametrize("name", ["dgc", "graddrop"])
def test_selection_on_a_stream_that_owns_a_few_sms(name):
    """The launch is sized for the stream's SMs: its CTAs wait for one another."""
    import ctypes as C
    from hipress_b200._native import lib
    st, sms, green = C.c_void_p(), C.c_int(), C.c_void_p()
    L = lib.cuda()
    if L.hp_cuda_partition_stream_create(torch.cuda.current_device(), 16, 0, C.byref(st), C.byref(sms), C.byref(green)):
        pytest.skip("the driver refuses SM partitions")
    assert 0 < sms.value < torch.cuda.get_device_properties(0).multi_processor_count
    stream = torch.cuda.ExternalStream(st.value)
    torch.manual_seed(7)
    n = 3000001
    g, c = torch.randn(n) * torch.randn(n), Compressor(name, ratio=0.001)
    gg, state, ws = g.cuda(), c.new_state(n, "cuda"), c.new_workspace("cuda", n)
    torch.cuda.synchronize()
    out = c.encode(gg, state, workspace=ws, stream=stream)
    stream.synchronize()
    ic, vc = sparse_pairs(c.encode(g, c.new_state(n, "cpu")), c.kmax(n))
    ig, vg = sparse_pairs(out, c.kmax(n))
    assert torch.equal(ic, ig) and torch.equal(vc, vg)
    assert int(ws[3 * 4096 + 9]) == 0, "a barrier expired"     # kWsStatus
    torch.cuda.synchronize()
    L.hp_cuda_partition_stream_destroy(st, green)
