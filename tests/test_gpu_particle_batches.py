"""The particle loops in the batches whose lanes gather events (launch_rules.h)
and in those that do not: the oracle's histories, repeated to a batch on each
side of the limits, come out bit for bit; likewise with the waits set."""
import numpy as np
import pytest

from xdg_gb300 import synth
from xdg_gb300.engine import FP64, MIXED, XDG

pytestmark = pytest.mark.gpu

BASE = 2000


def _check(got, want, m, what):
    for k, (g, w) in enumerate(zip(got, want)):
        g = g.cpu().numpy()
        assert np.array_equal(g, np.concatenate([w.astype(g.dtype, copy=False)] * m)), (what, k)


@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_elements(cuda, oracle, prec):
    torch = cuda
    full = torch.cuda.get_device_properties(0).multi_processor_count * 512
    tm = synth.tet_cube(n=8, size=10.0, jitter=0.2, seed=11)
    x = XDG(synth.model_from_tets(tm, np.ones(len(tm.conn), dtype=np.int32)))
    x.prepare_raytracer()
    rng = np.random.default_rng(21)
    p = rng.uniform(0.05, 9.95, (BASE, 3))
    u = synth.isotropic_dirs(rng, BASE)
    elem = x.find_element(p)[1].astype(np.int32)
    seeds = x.rti.seed_streams(77, BASE)
    o = oracle.TetWalker(tm.vertices, tm.conn, tm.adj, tm.face_table).transport(
        elem, p, u, seeds, 1.0, 300)
    want = [o[0], o[1], o[2], o[3].view(np.int64), *o[4:7]]

    def run(m, wait):
        rep = lambda a: torch.from_numpy(np.concatenate([a] * m)).cuda()  # noqa: E731
        s = [rep(elem), rep(p), rep(u), rep(seeds.view(np.int64))]
        dist = torch.zeros(m * BASE, dtype=torch.float64, device="cuda")
        ev = torch.zeros(m * BASE, dtype=torch.int32, device="cuda")
        x.rti.set_tuning("transport_event_wait", wait)
        st = x.rti.transport_elements(*s, 1.0, 300, dist, ev, precision=prec)
        return [*s, dist, ev, st]

    default = x.rti.get_tuning("transport_event_wait")
    # four lanes a particle, one, a particle a lane, eight a lane
    for m in (1, 15, full // BASE, full // BASE + 1, 8 * full // BASE + 1):
        _check(run(m, default), want, m, m)
    for wait in (1, 32):
        for m in (1, 15, full // BASE + 1):
            _check(run(m, wait), want, m, (m, wait))


@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_surfaces(cuda, oracle, prec):
    torch = cuda
    full = torch.cuda.get_device_properties(0).multi_processor_count * 512
    m0 = synth.nested_spheres(n=8, level=3, jitter=1e-3, seed=7)
    x = XDG(m0)
    x.prepare_raytracer()
    rng = np.random.default_rng(8)
    p = rng.uniform(-4.5, 4.5, (BASE, 3))  # inside the outer sphere
    u = synth.isotropic_dirs(rng, BASE)
    tree = x._trees(x.find_volume(p, u)).astype(np.int32)
    grave = x.volume_to_surface_tree[m0.implicit_complement]
    assert (tree != grave).all()
    seeds = x.rti.seed_streams(7, BASE)
    o = oracle.SurfaceTransport(m0, x.volume_to_surface_tree).run(
        tree, p, u, seeds, 0.7, 1_000_000, graveyard_tree=grave)
    want = [o[0], o[1], o[2], o[3].view(np.int64), *o[4:7]]

    def run(m):
        rep = lambda a: torch.from_numpy(np.concatenate([a] * m)).cuda()  # noqa: E731
        s = [rep(tree), rep(p), rep(u), rep(seeds.view(np.int64))]
        n = m * BASE
        hist = torch.zeros((n, 16), dtype=torch.int32, device="cuda")
        hc = torch.zeros(n, dtype=torch.int32, device="cuda")
        dist = torch.zeros(n, dtype=torch.float64, device="cuda")
        ev = torch.zeros(n, dtype=torch.int32, device="cuda")
        st = x.rti.transport_surfaces(*s, 0.7, 1_000_000, hist, hc, dist, ev, None, grave, prec)
        return [*s, dist, ev, st]

    for m in (1, full // BASE, full // BASE + 1):
        _check(run(m), want, m, m)
    for flush, event in ((1, 24), (16, 1), (4, 32), (32, 32)):
        x.rti.set_tuning("trace_flush_wait", flush)
        x.rti.set_tuning("particle_event_wait", event)
        _check(run(full // BASE + 1), want, full // BASE + 1, (flush, event))
