"""Rivers too long for the resident solve (one site after another, where the staged iterations
fold whole chains): the staged iterations take over, and the model starts with them from then
on.  With slope limits both go site by site, and the resident solve keeps such terrains."""
import numpy as np
import pytest

from fastlem_gb300 import ParameterArrays, TerrainModel2D, _lib, workloads
from fastlem_gb300.batch import BatchGenerator, TerrainBatch
from tests import graphs
from tests.test_gpu_resident import _same, _solve

pytestmark = pytest.mark.gpu


def _file(n):
    """A single file of sites."""
    g = graphs.from_edges(n, [(i, i + 1, 1.0 + 0.25 * (i % 7)) for i in range(n - 1)], default_outlets=[0])
    return TerrainModel2D(np.arange(n, dtype=np.float64), np.zeros(n), g.area, g.row_ptr, g.col, g.length,
                          g.default_outlets)


def _terrain_with_file(n, length, seed):
    """A terrain, and a single file of sites that drains into it from the side."""
    m = workloads.build_model(n, n ** 0.5, seed, 0)
    src = np.repeat(np.arange(n), np.diff(m.row_ptr.astype(np.int64)))
    first = src < m.col                         # every edge once, the rows' order from them
    edges = list(zip(src[first].tolist(), m.col[first].tolist(), m.length[first].tolist()))
    edge = int(np.argmax(m.xs))
    chain = [edge] + list(range(n, n + length))
    edges += [(a, b, 1.0 + 0.125 * (b % 5)) for a, b in zip(chain, chain[1:])]
    g = graphs.from_edges(n + length, edges, area=np.concatenate([m.area, np.ones(length)]),
                          default_outlets=[int(np.argmin(m.xs))])
    xs = np.concatenate([m.xs, m.xs[edge] + 1.0 + np.arange(length)])
    ys = np.concatenate([m.ys, np.full(length, m.ys[edge])])
    return TerrainModel2D(xs, ys, g.area, g.row_ptr, g.col, g.length, g.default_outlets)


def _params(m, slope=None):
    r = np.random.default_rng(m.n)
    return ParameterArrays(m.n, erodibility=r.uniform(0.5, 2.0, m.n), uplift_rate=r.uniform(0.5, 1.5, m.n),
                           max_slope=slope)


def _launches(handle):
    s = _lib.kernel_stats(handle)
    return s["resident_solve"][0], s["kahn_rounds"][0]


def _oracle(orc, m, p, iters):
    r = orc.generate(graphs.from_model(m), p.base, p.erodibility, p.uplift, p.is_outlet,
                     max_slope=p.max_slope, max_iter=iters)
    return r["elev"], r["iters"]


@pytest.mark.parametrize("n", [20000, 150001])
def test_file_leaves_once(orc, n):
    m = _file(n)
    p = _params(m)
    want, iters = _oracle(orc, m, p, 12)
    for call in range(2):
        e, it, used = _solve(m, p, 12, resident=None)
        assert used == (call == 0)
        assert _launches(m.handle())[1] > 0 and it == iters and _same(e, want)


def test_terrain_leaves_between_iterations(orc):
    """An iteration of 1 to 2 times the staged one's time: the solve leaves after some."""
    m = _terrain_with_file(20000, 2600, 3)
    p = _params(m)
    want, iters = _oracle(orc, m, p, 40)
    for call in range(2):
        e, it, used = _solve(m, p, 40, resident=None)
        assert used == (call == 0)
        assert _launches(m.handle())[1] > 0 and it == iters and _same(e, want)


def test_file_with_slope_limits_stays(orc):
    m = _file(20000)
    assert _solve(m, _params(m), 2, resident=None)[2]      # without them it leaves
    seen = _launches(m.handle())[1]
    p = _params(m, 0.5)
    want, iters = _oracle(orc, m, p, 12)
    for call in range(2):
        e, it, used = _solve(m, p, 12, resident=None)
        assert used and _launches(m.handle())[1] == seen
        assert it == iters and _same(e, want)


def test_file_in_a_pack(orc):
    ms = [workloads.build_model(9000, 95.0, 1, 0), _file(30000), workloads.build_model(2000, 45.0, 2, 0)]
    ps = [_params(m) for m in ms]
    want = [_oracle(orc, m, p, 25) for m, p in zip(ms, ps)]
    batch = TerrainBatch(ms)
    seen = (0, 0)
    for call in range(2):
        g = BatchGenerator().set_batch(batch).set_parameters(ps).set_max_iteration(25)
        outs = g.generate()
        now = _launches(batch.handle())
        assert now[0] > seen[0] and now[1] > seen[1]      # the others resident, the file staged
        seen = now
        for t, ((e, it), o) in enumerate(zip(want, outs)):
            assert int(g.last_terrain_iterations[t]) == it and _same(np.array(o.elevations()), e), t


@pytest.mark.parametrize("iters", [3, 7, 40])
def test_pack_leaves_at_different_iterations(orc, iters):
    """The staged iterations count on from each terrain's own: one that left after some, one
    that starts again, settled ones, and limits before and after they leave."""
    ms = [workloads.build_model(9000, 95.0, 1, 0), _terrain_with_file(9000, 2900, 3), _file(30000),
          _terrain_with_file(2500, 5000, 4), _file(40)]
    ps = [_params(m) for m in ms]
    want = [_oracle(orc, m, p, iters) for m, p in zip(ms, ps)]
    batch = TerrainBatch(ms)
    for call in range(2):
        g = BatchGenerator().set_batch(batch).set_parameters(ps).set_max_iteration(iters)
        outs = g.generate()
        for t, ((e, it), o) in enumerate(zip(want, outs)):
            assert int(g.last_terrain_iterations[t]) == it and _same(np.array(o.elevations()), e), t
        assert g.last_iterations == max(it for _, it in want)
    now = _launches(batch.handle())
    assert now[0] > 0 and now[1] > 0
