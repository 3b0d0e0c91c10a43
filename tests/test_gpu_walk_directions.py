"""Walks along directions far below the FP32 range: the mixed path's FP32
filter sees components under 2^-126 as zero, so it may not skip faces there.
Both precisions must equal the oracle bit for bit, whatever the length of the
direction vector."""
import numpy as np
import pytest

from xdg_gb300 import synth
from xdg_gb300.engine import FP64, MIXED, CudaRayTracer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("exponent", [-98, -101, -124, -126, -140, 100])
def test_direction_lengths(cuda, oracle, prec, exponent):
    # coordinates near 2^50, so that the edge coordinates stay above the
    # reference's zero tolerance
    tm = synth.tet_cube(n=5, size=5.0, jitter=0.2, seed=3)
    scale, s = 2.0 ** 50, 2.0 ** exponent
    tm.vertices *= scale
    rng = np.random.default_rng(9)
    n = 700
    r = rng.uniform(0.2, 4.8, (n, 3)) * scale
    u = synth.isotropic_dirs(rng, n) * s
    length = rng.exponential(3.0, n) * (scale / s)
    _, idx = oracle.TetTree(tm.tet_xyz(), tm.elem_ids).find_element(r)
    ok = np.nonzero(idx >= 0)[0]
    assert len(ok) > 600
    idx, r, u, length = idx[ok], r[ok], u[ok], length[ok]
    oe, ol, oc, ost = oracle.TetWalker(tm.vertices, tm.conn, tm.adj, tm.face_table).walk(
        idx, r, u, length, 128)
    assert oc.mean() > 3
    rti = CudaRayTracer()
    rti.set_tet_mesh(tm)
    se, sl, sc, st = rti.walk_elements(idx, r, u, length, 128, prec)
    assert np.array_equal(sc, oc) and np.array_equal(st, ost)
    for k in range(len(sc)):
        assert np.array_equal(se[k, :sc[k]], tm.elem_ids[oe[k, :sc[k]]]), k
        assert np.array_equal(sl[k, :sc[k]], ol[k, :sc[k]]), k
