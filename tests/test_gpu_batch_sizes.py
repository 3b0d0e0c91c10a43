"""Small batches are spread over more warps with fewer items each
(lanes_per_warp): every query of n items, for n at the edges of that rule,
gives the results its items have in one large batch, bit for bit."""
import numpy as np
import pytest

from xdg_gb300 import synth
from xdg_gb300.engine import FP64, MIXED, XDG, CudaRayTracer

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 33, 608, 913, 1825, 2433, 4865, 20000, 24320, 24321, 29999]
N = 30000


@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_batch_sizes(cuda, prec):
    m = synth.single_sphere_in_box(level=3)
    x = XDG(m)
    x.prepare_raytracer()
    o, d = synth.lcg_ball_rays(N, 9.9, seed=5)
    tree = x.volume_to_surface_tree[1]
    tm = synth.tet_cube(n=5, size=5.0, jitter=0.2, seed=3)
    rti = CudaRayTracer()
    rti.set_tet_mesh(tm)
    et = rti.create_element_tree(synth.Model(volumes=[1], tets=tm, elements={
        1: np.arange(len(tm.conn), dtype=np.int32)}), 1)
    rng = np.random.default_rng(7)
    p = rng.uniform(0.1, 4.9, (N, 3))
    length = rng.exponential(2.0, N)
    elem = rti.find_element(et, p, prec)[1]
    assert (elem >= 0).all()

    def calls(n):
        st = np.arange(n, dtype=np.uint64)
        e, r, u, s = elem[:n].copy(), p[:n].copy(), d[:n].copy(), st
        dist, ev = np.zeros(n), np.zeros(n, dtype=np.int32)
        status = rti.transport_elements(e, r, u, s, 1.0, 1000, dist, ev, precision=prec)
        walk = rti.walk_elements(elem[:n], p[:n], d[:n], length[:n], 64, prec)
        used = np.arange(64)[None, :] < walk[2][:, None]
        return [*x.rti.ray_fire(tree, o[:n], d[:n], precision=prec, status=True),
                *x.rti.occluded(tree, o[:n], d[:n], prec),
                x.rti.point_in_volume(tree, o[:n], d[:n], precision=prec),
                x.find_volume(o[:n], d[:n], prec), *x.rti.closest(tree, o[:n], prec),
                *rti.find_element(et, p[:n], prec), *rti.next_element(elem[:n], p[:n], d[:n], prec),
                np.where(used, walk[0], -1), np.where(used, walk[1], 0.0), walk[2], walk[3],
                e, r, u, s, dist, ev, status]

    want = calls(N)
    for n in SIZES:
        for k, (a, b) in enumerate(zip(calls(n), want)):
            assert np.array_equal(a, b[:n]), (n, k)
