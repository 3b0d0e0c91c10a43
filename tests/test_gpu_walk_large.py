"""Walks in batches above those whose tracks are shared among lanes, and at
the upper end of the mid-sized ones whose longest are: the oracle's tracks,
repeated, come out bit for bit, inside the integer products' domain
(imul64.cuh) and outside it, and without the edge table."""
import numpy as np
import pytest

from xdg_gb300 import synth
from xdg_gb300.engine import FP64, MIXED, CudaRayTracer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("case", ["plain", "zeros", "tiny_vertex", "tiny_direction", "tiny_position",
                                  "short", "no_edge_table"])
def test_large_batches(cuda, oracle, prec, case):
    torch = cuda
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tm = synth.tet_cube(n=5, size=5.0, jitter=0.2, seed=3)
    rng = np.random.default_rng(5)
    n = 700
    r = rng.uniform(0.2, 4.8, (n, 3))
    u = synth.isotropic_dirs(rng, n)
    length = rng.exponential(3.0, n)
    if case == "zeros":
        u[np.arange(n), rng.integers(0, 3, n)] = 0.0
        u /= np.linalg.norm(u, axis=1)[:, None]
    elif case == "tiny_vertex":
        tm.vertices[tm.vertices == 0.0] = 1e-60
    elif case == "tiny_direction":
        u[: n // 2, 0] = 1e-60
    elif case == "tiny_position":
        r[: n // 2, 1] = 1e-60
    elif case == "short":
        length = 10.0 ** rng.uniform(-320, 0, n)
    rti = CudaRayTracer()
    rti.set_tet_mesh(tm)
    if case == "no_edge_table":
        rti.set_tuning("walk_edge_table", 0)
    _, idx = oracle.TetTree(tm.tet_xyz(), tm.elem_ids).find_element(r)
    ok = np.nonzero(idx >= 0)[0][:600]
    assert len(ok) == 600
    idx, r, u, length = idx[ok].astype(np.int32), r[ok], u[ok], length[ok]
    oe, ol, oc, ost = oracle.TetWalker(tm.vertices, tm.conn, tm.adj, tm.face_table).walk(
        idx, r, u, length, 64)
    assert oc.max() < 64
    used = np.arange(64)[None, :] < oc[:, None]
    want_e = torch.from_numpy(np.where(used, tm.elem_ids[np.where(used, oe, 0)], -1).astype(np.int32)).cuda()
    want_l = torch.from_numpy(np.where(used, ol, -1.0)).cuda()
    want = [torch.from_numpy(a.astype(np.int32)).cuda() for a in (oc, ost)]
    used = torch.from_numpy(used).cuda()

    def rep(a, m):
        return torch.from_numpy(np.concatenate([a] * m)).cuda()

    mix = sms * 704 // 600
    for m in (mix, mix + 1):
        se, sl, sc, st = rti.walk_elements(rep(idx, m), rep(r, m), rep(u, m), rep(length, m), 64, prec)
        mask = used.repeat(m, 1)
        assert torch.equal(sc, want[0].repeat(m)) and torch.equal(st, want[1].repeat(m)), m
        assert torch.equal(torch.where(mask, se, -1), want_e.repeat(m, 1)), m
        assert torch.equal(torch.where(mask, sl, -1.0), want_l.repeat(m, 1)), m
