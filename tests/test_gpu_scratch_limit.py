"""Calls on a device without free memory for their scratch, which
XDGCU_SCRATCH_LIMIT stands in for: what a call takes only to be faster it does
without, and the results are the same."""
import numpy as np
import pytest

from xdg_gb300 import synth
from xdg_gb300.engine import MIXED, XDG

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
