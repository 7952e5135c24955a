"""Phase times of a top-k bucket: the persistent kernels' stamps, and nothing for a chain of
launches, which has none."""
import pytest
import torch

from hipress_b200.ops import Compressor
from hipress_b200.parallel.fused_sparse import FusedSparseBucket

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("topology", ["ps", "ring"])
@pytest.mark.parametrize("what", ["normal", "equal"])     # equal values: the emitting launch has barriers too
def test_phase_times_of_one_rank(topology, what):
    n = 100 * 4096
    spec = Compressor("graddrop", ratio=0.01).spec
    g = torch.randn(n, device="cuda") if what == "normal" else torch.ones(n, device="cuda")
    for ctas in (0, 4, 0):
        b = FusedSparseBucket(spec, [n], 1, 0, topology=topology, ctas=ctas).bind_local("cuda")
        out, acc, sr = torch.empty_like(g), torch.zeros_like(g), torch.zeros_like(g)
        b.launch_ptrs([g.data_ptr()], [acc.data_ptr()], None, [out.data_ptr()], [sr.data_ptr()])
        torch.cuda.synchronize()
        b.check_status()
        times = b.last_phase_times()
        if ctas:
            assert times and all(0 < a <= c for a, c in zip(times, times[1:])), times
        else:
            assert times == [] and b.last_marks == []


def test_sweep_of_one_rank_reports_no_phases():
    from hipress_b200.bench.sweep import run_single
    rows = []
    run_single("graddrop", "ring", 1, 0, 2, rows)
    assert rows[0]["ms"] > 0 and not [k for k in rows[0] if "phase" in k or "marks" in k]
