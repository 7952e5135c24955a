"""The top-k chain of launches where its cooperative launch is refused, and where a barrier
of that launch expires.  The library is linked with a copy of the chain whose host refuses
the launch, or whose barrier waits, 20 us, for one CTA more than there are.  It runs in a
child process because the choice of library is made once per process."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


def _library(d: Path, source: str) -> Path:
    """The CUDA library with `source` in the place of sparse_chain.cu."""
    from hipress_b200._native import build as b
    flags = [f for f in b.NVCC_FLAGS if f not in ("-Xptxas", "-v")] + ["-I", str(b.CSRC / "include"), "-I", str(b.CSRC / "cuda")]
    nv, objs = b.nvcc_path(), []
    b.build()
    for s in sorted((b.CSRC / "cuda").glob("*.cu")):
        if s.name == "sparse_chain.cu":
            s, o = Path(__file__).parent / "native" / source, d / "chain.o"
        elif (b.OBJ / (s.stem + ".o")).exists():
            objs.append(b.OBJ / (s.stem + ".o"))
            continue
        else:
            o = d / (s.stem + ".o")
        subprocess.run([nv, *flags, "-c", str(s), "-o", str(o)], check=True)
        objs.append(o)
    out = d / "libhipress_cuda.so"
    subprocess.run([nv, "-shared", "-o", str(out), *map(str, objs), "-lcudart"], check=True)
    for name in ("libhipress_cpu.so", "_fastcall.so"):
        (d / name).symlink_to(b.HERE / name)
    return out


HEAD = """
import sys
from pathlib import Path
import torch
from hipress_b200._native import lib
lib.HERE = Path(sys.argv[1])
from hipress_b200.ops import Compressor, sparse_pairs
from hipress_b200.parallel.fused_sparse import FusedSparseBucket
from hipress_b200.parallel.simulate import chunk_elems, simulate_ps, simulate_ring
lib.cuda()
gen = torch.Generator().manual_seed(5)
def values(n):
    return torch.randn(n, generator=gen) * torch.randn(n, generator=gen)
"""

REFUSED = """
for name in ("dgc", "graddrop"):
    acc = "accum_v" if name == "dgc" else "residual"
    c = Compressor(name, ratio=0.01)
    for n in (300, 70 * 4096 + 33):
        cpu, dev, ws = c.new_state(n, "cpu"), c.new_state(n, "cuda"), c.new_workspace("cuda", n)
        for step in range(2):
            g = values(n)
            want = sparse_pairs(c.encode(g, cpu), c.kmax(n))
            got = sparse_pairs(c.encode(g.cuda(), dev, workspace=ws), c.kmax(n))
            assert all(torch.equal(a, b) for a, b in zip(want, got)), (name, n, step)
            assert all(torch.equal(dev[k].cpu(), cpu[k]) for k in cpu), (name, n, step)
    sizes = [200003, 8192, 300, 1]
    for topology in ("ps", "ring"):
        b = FusedSparseBucket(c.spec, sizes, 1, 0, topology=topology).bind_local("cuda")
        cpu = [c.new_state(s, "cpu") for s in sizes]
        srv = [{"residual": torch.zeros(chunk_elems(s, 1))} for s in sizes]
        dev = [{k: v.cuda() for k, v in st.items()} for st in cpu]
        sums = [x["residual"].cuda() for x in srv]
        for step in range(2):
            grads = [values(s) for s in sizes]
            out = [g.cuda() for g in grads]
            b.launch_ptrs([g.data_ptr() for g in out], [s[acc].data_ptr() for s in dev],
                          [s["momentum_u"].data_ptr() for s in dev] if name == "dgc" else None,
                          [g.data_ptr() for g in out], [s.data_ptr() for s in sums])
            torch.cuda.synchronize()
            b.check_status()
            for i in range(len(sizes)):
                ref = simulate_ps(c, [grads[i]], [cpu[i]], [srv[i]]) if topology == "ps" else \\
                    simulate_ring(c, [grads[i]], [cpu[i]])
                # plain multiply-adds and copies, one rank: the same bits
                assert torch.equal(out[i].cpu(), ref[0]), (name, topology, step, i)
                assert all(torch.equal(dev[i][k].cpu(), cpu[i][k]) for k in cpu[i]), (name, topology, step, i)
                if topology == "ps":
                    assert torch.equal(sums[i].cpu(), srv[i]["residual"]), (name, step, i)
print("OK")
"""


def _child(d, source, code):
    _library(d, source)
    r = subprocess.run([sys.executable, "-c", HEAD + code, str(d)], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "PYTHONPATH": str(ROOT)})
    assert r.returncode == 0 and "OK" in r.stdout, r.stderr[-3000:]


def test_a_refused_launch_is_made_up_for(tmp_path):
    """The arrays are updated when the last launch is refused: the call ends as it would have."""
    _child(tmp_path, "chain_refused.cu", REFUSED)


EXPIRED = """
from hipress_b200.parallel.fused import HipressTimeoutError
sizes = [200003, 8192]
c = Compressor("graddrop", ratio=0.01)
for topology in ("ps", "ring"):
    b = FusedSparseBucket(c.spec, sizes, 1, 0, topology=topology).bind_local("cuda")
    # equal values: the list overflows and the CTAs meet at the barrier
    grads = [torch.full((sizes[0],), 0.5), values(sizes[1])]
    out = [g.cuda() for g in grads]
    acc = [torch.zeros(s, device="cuda") for s in sizes]
    sums = [torch.zeros(s, device="cuda") for s in sizes]
    b.launch_ptrs([g.data_ptr() for g in out], [a.data_ptr() for a in acc], None, [g.data_ptr() for g in out],
                  [s.data_ptr() for s in sums])
    torch.cuda.synchronize()
    assert not out[0].any(), (topology, int(out[0].count_nonzero()))
    if topology == "ps":    # nor from the sum of a push that was not complete
        assert not out[1].any(), int(out[1].count_nonzero())
    else:                   # its list was complete
        assert torch.equal(out[1].cpu(), simulate_ring(c, [grads[1]], [c.new_state(sizes[1], "cpu")])[0])
    try:
        b.check_status()
    except HipressTimeoutError:
        pass
    else:
        raise AssertionError("no status")
print("OK")
"""


def test_a_result_is_left_alone_behind_a_barrier_that_expired(tmp_path):
    _child(tmp_path, "chain_expired.cu", EXPIRED)
