"""Resident solves of more than one launch: each ends when its share of time is over and the
next goes on from there, or when an iteration needs the lake order first."""
import threading

import numpy as np
import pytest

from fastlem_gb300 import ParameterArrays, TerrainModel2D, _lib, workloads
from fastlem_gb300.batch import BatchGenerator, TerrainBatch
from tests import graphs
from tests.test_gpu_resident import _case, _same, _solve

pytestmark = pytest.mark.gpu


def _resident_launches(handle):
    return _lib.kernel_stats(handle)["resident_solve"][0]


@pytest.mark.parametrize("n, iters, slope", [(65537, 350, False), (60007, 200, True), (1500, 2000, False),
                                             (262144, 90, False), (250007, 60, True)])
def test_goes_on_in_the_next_launch(n, iters, slope):
    """Some 40 ms of iterations each, many more than one launch's share."""
    m, p = _case(n, 4, slope)
    f, jt, _ = _solve(m, p, iters, resident=False)
    e, it, used = _solve(m, p, iters)
    assert used and _resident_launches(m.handle()) >= 2
    assert it == jt == iters and _same(e, f)


def test_pack_of_several_waves():
    """More terrains than the blocks take at once: some start in a later launch."""
    base = [_case(n, i + 1, i == 2) for i, n in enumerate([9001, 15000, 700, 30011])]
    cases = [base[i % 4] for i in range(100)]                 # 1.4M sites
    batch = TerrainBatch([m for m, _ in cases])
    g = BatchGenerator().set_batch(batch).set_parameters([p for _, p in cases]).set_max_iteration(70)
    outs = [np.array(t.elevations()) for t in g.generate()]
    assert _resident_launches(batch.handle()) >= 2
    want = [_solve(m, p, 70, resident=False) for m, p in base]
    for i, (e, it) in enumerate(zip(outs, g.last_terrain_iterations)):
        assert it == want[i % 4][1] and _same(e, want[i % 4][0]), i


@pytest.mark.parametrize("slope", [None, 0.6])
def test_first_lake_after_the_first_iteration(orc, slope):
    """A smooth rise from the outlet has no lake; the first iteration's relief has."""
    g = graphs.random_delaunay(7000, 11, side=80.0)
    out = int(np.argmin(g.xs))
    dist = np.full(g.n, np.inf)
    dist[out] = 0.0
    src = np.repeat(np.arange(g.n), np.diff(g.row_ptr.astype(np.int64)))
    while True:                                               # path length from the outlet
        new = dist.copy()
        np.minimum.at(new, g.col, dist[src] + g.length)
        if np.array_equal(new, dist):
            break
        dist = new
    r = np.random.default_rng(3)
    m = TerrainModel2D(g.xs, g.ys, g.area, g.row_ptr, g.col, g.length, np.array([out], np.uint32))
    p = ParameterArrays(g.n, base_elevation=dist, erodibility=np.exp(r.normal(0, 0.5, g.n)),
                        uplift_rate=r.uniform(0.0, 2.0, g.n), max_slope=slope)
    e, it, used = _solve(m, p, 20)
    assert used and _resident_launches(m.handle()) >= 2       # stopped for the lake order
    want = orc.generate(graphs.from_model(m), p.base, p.erodibility, p.uplift, p.is_outlet,
                        max_slope=p.max_slope, max_iter=20)
    assert it == want["iters"] and _same(e, want["elev"])


def test_two_streams_at_once():
    cases = [_case(65537, 2, False), _case(20011, 3, True), _case(1024, 4, False), _case(100003, 5, False)]
    want = [_solve(m, p, 120, resident=False)[:2] for m, p in cases]
    from fastlem_gb300 import TerrainGenerator
    bad = []

    def work(m, p, e, it):
        g = TerrainGenerator.default().set_model(m).set_parameters(p).set_max_iteration(120)
        for _ in range(3):
            f = np.array(g.generate().elevations())
            if g.last_iterations != it or not _same(f, e):
                bad.append(m.n)

    threads = [threading.Thread(target=work, args=(*c, *w)) for c, w in zip(cases, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad and all(_resident_launches(m.handle()) > 0 for m, _ in cases)
