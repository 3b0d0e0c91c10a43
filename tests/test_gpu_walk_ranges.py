"""The walk and next_element at the edges of the integer products' domain
(imul64.cuh): meshes and directions with values outside it take the FP64
unit's products, those with zeros the integer ones; both must equal the
oracle bit for bit."""
import numpy as np
import pytest

from xdg_gb300 import synth
from xdg_gb300.engine import FP64, MIXED, CudaRayTracer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("case", ["zeros", "tiny_vertex", "tiny_direction", "tiny_position", "short"])
def test_walk_ranges(cuda, oracle, prec, case):
    tm = synth.tet_cube(n=5, size=5.0, jitter=0.2, seed=3)
    rng = np.random.default_rng(5)
    n = 700
    r = rng.uniform(0.2, 4.8, (n, 3))
    u = synth.isotropic_dirs(rng, n)
    length = rng.exponential(3.0, n)
    if case == "zeros":        # zero direction components, boundary coordinates 0
        u[np.arange(n), rng.integers(0, 3, n)] = 0.0
        u /= np.linalg.norm(u, axis=1)[:, None]
    elif case == "tiny_vertex":
        tm.vertices[tm.vertices == 0.0] = 1e-60
    elif case == "tiny_direction":
        u[: n // 2, 0] = 1e-60
    elif case == "tiny_position":
        r[: n // 2, 1] = 1e-60
    else:                      # track lengths down to denormals
        length = 10.0 ** rng.uniform(-320, 0, n)
    rti = CudaRayTracer()
    rti.set_tet_mesh(tm)
    _, idx = oracle.TetTree(tm.tet_xyz(), tm.elem_ids).find_element(r)
    ok = np.nonzero(idx >= 0)[0]
    assert len(ok) > 600
    idx, r, u, length = idx[ok], r[ok], u[ok], length[ok]
    w = oracle.TetWalker(tm.vertices, tm.conn, tm.adj, tm.face_table)
    oe, ol, oc, ost = w.walk(idx, r, u, length, 128)
    se, sl, sc, st = rti.walk_elements(idx, r, u, length, 128, prec)
    assert np.array_equal(sc, oc) and np.array_equal(st, ost)
    for k in range(len(sc)):
        assert np.array_equal(se[k, :sc[k]], tm.elem_ids[oe[k, :sc[k]]]), k
        assert np.array_equal(sl[k, :sc[k]], ol[k, :sc[k]]), k
    # one step through next_element: the walk's first segment of long tracks
    nxt, dist, _ = rti.next_element(idx, r, u, prec)
    long = sc > 1
    assert np.array_equal(dist[long], ol[long, 0])
    assert np.array_equal(tm.elem_ids[nxt[long]], tm.elem_ids[oe[long, 1]])
