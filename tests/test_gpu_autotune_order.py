"""The walk's autotuner either turns the length order off or leaves the
threshold at which batches take it: the mid-sized batches below its sample
walk differently with the order, and it has not timed those."""
import numpy as np
import pytest

from xdg_gb300 import synth
from xdg_gb300.engine import FP64, MIXED, XDG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("n,before", [(200_000, None), (200_000, 60_000), (20_000, 50_000),
                                      (200_000, 0), (4000, None)])
def test_order_threshold(cuda, prec, n, before):
    torch = cuda
    tm = synth.tet_cube(n=30, size=10.0, jitter=0.2, seed=11)
    x = XDG(synth.model_from_tets(tm, np.ones(len(tm.conn), dtype=np.int32)))
    x.prepare_raytracer()
    rng = np.random.default_rng(3)
    p = rng.uniform(0.01, 9.99, (n, 3))
    idx = x.find_element(p)[1].astype(np.int32)
    dev = [torch.from_numpy(a).cuda() for a in (idx, p, synth.isotropic_dirs(rng, n),
                                                np.minimum(rng.exponential(5.0, n), 30.0))]
    default = x.rti.get_tuning("walk_sort_min")
    if before is not None:
        x.rti.set_tuning("walk_sort_min", before)
    _, tuned = x.rti.autotune_walk(*dev, max_segs=256, precision=prec, reps=3)
    after = tuned["walk_sort_min"]
    if n < default:           # not searched
        assert after == default
    elif before and before > n:
        assert after in (0, n, before)
    else:
        assert after in (0, before or default)
