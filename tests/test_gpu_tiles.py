"""The staged iterations' tiles (basins inside one range of 2,048 sites, done in shared memory)
against the oracle: ragged last tiles, rivers with more levels than a tile takes, sites with
more donors or longer rows than a tile takes (the longest turn the tiles off), slope limits."""
import numpy as np
import pytest

from fastlem_gb300 import ParameterArrays, TerrainGenerator, TerrainModel2D, _lib
from tests import graphs

pytestmark = pytest.mark.gpu


def _files(count, length):
    """Parallel single files of sites behind a common outlet row."""
    edges = [(f * length + i, f * length + i + 1, 1.0 + 0.125 * ((f + i) % 5))
             for f in range(count) for i in range(length - 1)]
    edges += [(f * length, (f + 1) * length, 1.0) for f in range(count - 1)]
    return graphs.from_edges(count * length, edges, default_outlets=[0])


def _hubs(count, spokes):
    """A file of hubs, each with `spokes` donors of its own (in adjacency order around it)."""
    edges = [(h, h + 1, 1.5) for h in range(count - 1)]
    edges += [(h, count + h * spokes + s, 1.0 + 0.01 * s) for h in range(count) for s in range(spokes)]
    return graphs.from_edges(count * (spokes + 1), edges, default_outlets=[0])


@pytest.mark.parametrize("slope", [False, True])
@pytest.mark.parametrize("make", [
    lambda: graphs.random_delaunay(2047, 1), lambda: graphs.random_delaunay(2048, 2),
    lambda: graphs.random_delaunay(2049, 3), lambda: graphs.random_delaunay(9000, 4),
    lambda: graphs.grid(70, 60, unit_lengths=True), lambda: _files(40, 19), lambda: _files(3, 1500),
    lambda: _hubs(300, 2), lambda: _hubs(300, 3), lambda: _hubs(300, 4), lambda: _hubs(200, 5),
    lambda: _hubs(200, 9), lambda: _hubs(150, 10), lambda: _hubs(150, 11), lambda: _hubs(8, 400)])
def test_staged_equals_oracle(orc, make, slope):
    g = make()
    n = g.n
    r = np.random.default_rng(n)
    xs = np.arange(n, dtype=np.float64) if g.xs is None else g.xs
    ys = np.zeros(n) if g.ys is None else g.ys
    m = TerrainModel2D(xs, ys, g.area, g.row_ptr, g.col, g.length, g.default_outlets)
    p = ParameterArrays(n, erodibility=np.exp(r.normal(0, 0.5, n)), uplift_rate=r.uniform(0.0, 2.0, n),
                        base_elevation=r.uniform(0, 1e-3, n),
                        max_slope=np.where(r.random(n) < 0.3, np.nan, r.uniform(0.05, 0.6, n)) if slope else None)
    want = orc.generate(g, p.base, p.erodibility, p.uplift, p.is_outlet, max_slope=p.max_slope, max_iter=8)
    old = _lib.set_tuning(resident=0)
    try:
        gen = TerrainGenerator.default().set_model(m).set_parameters(p).set_max_iteration(8)
        e = np.array(gen.generate().elevations())
        before = _lib.kernel_stats(m.handle())["resident_solve"][0]
    finally:
        _lib.set_tuning(**old)
    assert before == 0 and gen.last_iterations == want["iters"]
    assert np.array_equal(e.view(np.uint64), np.ascontiguousarray(want["elev"]).view(np.uint64))
