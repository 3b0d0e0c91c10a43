"""Calls on a device without free memory for their scratch, which
XDGCU_SCRATCH_LIMIT stands in for: what a call takes only to be faster it does
without, and the results are the same."""
import numpy as np
import pytest

from xdg_gb300 import synth
from xdg_gb300.engine import FP64, MIXED, XDG

pytestmark = pytest.mark.gpu


def _limited(monkeypatch, nbytes, model):
    if nbytes is not None:
        monkeypatch.setenv("XDGCU_SCRATCH_LIMIT", str(nbytes))
    else:
        monkeypatch.delenv("XDGCU_SCRATCH_LIMIT", raising=False)
    x = XDG(model)
    x.prepare_raytracer()
    return x


@pytest.mark.parametrize("op,n", [("ray_fire", 2_000_001), ("occluded", 2_000_000),
                                  ("point_in_volume", 2_000_000), ("find_volume", 500_000)])
def test_large_batches_without_scratch(cuda, monkeypatch, op, n):
    """The work queue of large batches needs a cursor in scratch memory;
    without it, and with trace_queue 0, the batch runs in fixed slices."""
    torch = cuda
    m = synth.single_sphere_in_box(level=2)
    o, d = (torch.from_numpy(a).cuda() for a in synth.lcg_ball_rays(n, 9.9, seed=5))

    def run(x):
        tree = x.volume_to_surface_tree[1]
        x.rti.set_tuning("scratch_bytes_high", 0)
        r = {"ray_fire": lambda: x.rti.ray_fire(tree, o, d, precision=MIXED),
             "occluded": lambda: x.rti.occluded(tree, o, d, MIXED),
             "point_in_volume": lambda: x.rti.point_in_volume(tree, o, d, precision=MIXED),
             "find_volume": lambda: x.find_volume(o, d, MIXED)}[op]()
        torch.cuda.synchronize()
        return (r if isinstance(r, tuple) else (r,)), x.rti.get_tuning("scratch_bytes_high")

    x = _limited(monkeypatch, None, m)
    want, used = run(x)
    assert used > 0  # the queue's cursor
    x.rti.set_tuning("trace_queue", 0)
    slices, used = run(x)
    assert used == 0
    got, used = run(_limited(monkeypatch, 1, m))
    assert used == 0
    for a, b, c in zip(want, slices, got):
        if torch.is_tensor(a):
            assert torch.equal(a, b) and torch.equal(a, c)
        else:
            assert np.array_equal(a, b) and np.array_equal(a, c)


@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("op", ["segments", "packed"])
def test_rounds_in_less_scratch(cuda, monkeypatch, op, prec):
    """The rounds of the global track loop and of the packed walk take a
    buffer of up to 4 GiB, and must still run where a buffer of 1 GiB and the
    rest of their scratch fit: whichever allocation fails first."""
    torch = cuda
    m = synth.tet_blocks([((12.0 * k, 0.0, 0.0), 6, 10.0) for k in range(3)], jitter=0.2, seed=17)
    n = 400_000
    rng = np.random.default_rng(3)
    lo, hi = [-3.0, -1.0, -1.0], [37.0, 11.0, 11.0]
    a, b = (torch.from_numpy(rng.uniform(lo, hi, (n, 3))).cuda() for _ in range(2))
    u, length = torch.nn.functional.normalize(b - a), (b - a).norm(dim=1)

    def run(x):
        x.rti.set_tuning("scratch_bytes_high", 0)
        if op == "segments":
            ipc = x.volume_to_surface_tree[m.implicit_complement]
            out = x.rti.segments_global(ipc, x.rti.global_element_tree, a, b, 64 * n,
                                        precision=prec)
        else:
            out = x.rti.walk_elements_packed(start, a, u, length, 64 * n, precision=prec)
        torch.cuda.synchronize()
        total = int(out[2][-1])
        assert total < 64 * n
        return (out[0][:total], out[1][:total], out[2], out[3]), total

    x = _limited(monkeypatch, None, m)
    if op == "packed":
        start = x.rti.find_element(x.rti.global_element_tree, a, prec)[1]
    want, total = run(x)
    peak = x.rti.get_tuning("scratch_bytes_high")
    # what the large buffer holds beyond 1 GiB, 12 bytes a segment
    spare = 12 * min(512 * n, (4 << 30) // 12) - (1 << 30)
    assert spare > 1 << 30
    for less in [3 * total, 6 * total, 9 * total, 12 * total,
                 *(int(f * spare) for f in (0.15, 0.3, 0.45, 0.6, 0.75, 0.9))]:
        got, _ = run(_limited(monkeypatch, peak - less, m))
        for k, (g, w) in enumerate(zip(got, want)):
            assert torch.equal(g, w), (less, k)
