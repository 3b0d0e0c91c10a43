"""The work counters of a walk do not depend on how the launch spreads it: the
same tracks m times over count m times the steps, FP64 escalations and tracks,
whether four lanes share a track (small batches), some tracks are shared
(mid-sized ones) or each lane walks its own; likewise the particles of the
walk_elements loop."""
import numpy as np
import pytest

from xdg_gb300 import synth
from xdg_gb300.engine import FP64, MIXED, CudaRayTracer

pytestmark = pytest.mark.gpu

BASE = 608


@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_counters_by_batch_size(cuda, oracle, prec):
    torch = cuda
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tm = synth.tet_cube(n=5, size=5.0, jitter=0.2, seed=3)
    rng = np.random.default_rng(11)
    p = rng.uniform(0.1, 4.9, (BASE, 3))
    u = synth.isotropic_dirs(rng, BASE)
    length = rng.exponential(2.0, BASE)
    rti = CudaRayTracer()
    rti.set_tet_mesh(tm)
    _, idx = oracle.TetTree(tm.tet_xyz(), tm.elem_ids).find_element(p)
    assert (idx >= 0).all()
    seeds = rti.seed_streams(5, BASE).view(np.int64)

    def dev(a, m):
        return torch.from_numpy(np.concatenate([a] * m)).cuda()

    def counted(call):
        rti.set_counting(True)
        try:
            out = call()
            torch.cuda.synchronize()
            return out, rti.counters()
        finally:
            rti.set_counting(False)

    def walk(m):
        (_, _, count, _), c = counted(lambda: rti.walk_elements(
            dev(idx.astype(np.int32), m), dev(p, m), dev(u, m), dev(length, m), 64, prec))
        assert c["steps"] == int(count.sum()) and c["rays"] == m * BASE
        return c

    def particles(m):
        z = torch.zeros(m * BASE, dtype=torch.float64, device="cuda")
        ev = torch.zeros(m * BASE, dtype=torch.int32, device="cuda")
        return counted(lambda: rti.transport_elements(
            dev(idx.astype(np.int32), m), dev(p, m), dev(u, m), dev(seeds, m), 1.0, 1000, z, ev,
            precision=prec))[1]

    team, mix = sms * 160 // BASE, sms * 704 // BASE  # the last batches of the shared launches
    for call, sizes in ((walk, (1, team, team + 1, mix, mix + 1)), (particles, (1, team, team + 1))):
        one = call(1)
        # an FP64 step decides all four faces exactly, a mixed one at least one
        if prec == FP64:
            assert one["escalate"] == 4 * one["steps"]
        else:
            assert one["steps"] <= one["escalate"] < 2 * one["steps"]
        for m in sizes:
            c = call(m)
            assert {k: c[k] for k in ("steps", "escalate", "rays")} == \
                {k: m * one[k] for k in ("steps", "escalate", "rays")}, (call.__name__, m)
