"""Whole solves in one launch (resident.cu): the staged iterations' and the oracle's results,
bit for bit, at the sizes where the cut into blocks changes, with slope limits, lakes, odd
graphs and packed terrains."""
import numpy as np
import pytest

from fastlem_gb300 import ParameterArrays, TerrainGenerator, TerrainModel2D, _lib, workloads
from fastlem_gb300.batch import BatchGenerator
from tests import graphs

pytestmark = pytest.mark.gpu


def _solve(model, params, iters, resident=True):
    """(elevations, iterations, whether the resident kernel ran); resident None: by the rule."""
    old = _lib.set_tuning(resident=-1 if resident is None else 1 if resident else 0)
    try:
        g = TerrainGenerator.default().set_model(model).set_parameters(params)
        if iters:
            g.set_max_iteration(iters)
        stats = _lib.kernel_stats(model.handle()).get("resident_solve", (0,))[0]
        e = g.generate().elevations()
        used = _lib.kernel_stats(model.handle())["resident_solve"][0] > stats
        return np.array(e), g.last_iterations, used
    finally:
        _lib.set_tuning(**old)


def _same(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint64), np.ascontiguousarray(b).view(np.uint64))


def _case(n, seed, slope):
    m = workloads.build_model(n, n ** 0.5, seed, 0)
    rng = np.random.default_rng(seed)
    ms = None
    if slope:
        ms = np.where(rng.random(n) < 0.2, np.nan, rng.uniform(-0.05, 0.6, n))
    p = ParameterArrays(n, erodibility=np.exp(rng.normal(0, 0.5, n)), uplift_rate=rng.uniform(0.0, 2.0, n),
                        base_elevation=rng.uniform(0, 1e-3, n) if seed % 2 else 0.0,
                        is_outlet=workloads.border_outlets(m, n ** 0.5, 0.02 * n ** 0.5), max_slope=ms)
    return m, p


@pytest.mark.parametrize("slope", [False, True])
@pytest.mark.parametrize("n", [3, 33, 448, 449, 897, 1025, 2049, 5000, 20011, 160001])
def test_equals_staged_iterations(n, slope):
    m, p = _case(n, n % 7 + 1, slope)
    iters = 40 if n < 100000 else 6
    e, it, used = _solve(m, p, iters)
    f, jt, staged = _solve(m, p, iters, resident=False)
    assert used and not staged
    assert it == jt and _same(e, f)


@pytest.mark.parametrize("slope", [None, 0.314])
def test_equals_oracle_to_convergence(orc, slope):
    w = workloads.small(scale=0.7, max_slope=slope)
    p = w.params
    e, it, used = _solve(w.model, p, 0)
    r = orc.generate(graphs.from_model(w.model), p.base, p.erodibility, p.uplift, p.is_outlet,
                     max_slope=p.max_slope)
    assert used and it == r["iters"] and _same(e, r["elev"])


def test_largest_part_size():
    """More sites than one per thread and block: every block holds several rounds."""
    m, p = _case(700001, 3, False)
    e, it, used = _solve(m, p, 3)
    f, jt, _ = _solve(m, p, 3, resident=False)
    assert used and it == jt and _same(e, f)


def test_caller_order_without_coordinates():
    """Without coordinates the blocks' ranges are arbitrary: nearly every donor is in another
    block, more than a block has room for, and the solve takes the staged iterations."""
    m, p = _case(30000, 5, False)
    perm = np.random.default_rng(1).permutation(m.n).astype(np.uint32)
    inv = np.argsort(perm).astype(np.uint32)
    deg = np.diff(m.row_ptr.astype(np.int64))[perm]
    row = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint32)
    take = np.concatenate([np.arange(m.row_ptr[v], m.row_ptr[v + 1]) for v in perm])
    q = TerrainModel2D(m.xs[perm], m.ys[perm], m.area[perm], row, inv[m.col[take]], m.length[take],
                       inv[m.default_outlets])
    import ctypes
    h = ctypes.c_void_p()
    _lib.check(_lib.lib().fl_graph_create(q.n, _lib.ptr(q.row_ptr), _lib.ptr(q.col), _lib.ptr(q.length),
                                          _lib.ptr(q.area), _lib.ptr(q.default_outlets),
                                          len(q.default_outlets), None, None, ctypes.byref(h)))
    q._handle = h
    r = ParameterArrays(q.n, erodibility=p.erodibility[perm], uplift_rate=p.uplift[perm],
                        base_elevation=p.base[perm], is_outlet=p.is_outlet[perm])
    e, it, _ = _solve(q, r, 5)
    f, jt, staged = _solve(q, r, 5, resident=False)
    assert not staged and it == jt and _same(e, f)


def test_long_river_goes_on_in_the_staged_iterations():
    """A single file of sites is one river as long as the terrain: the resident solve gives up
    after some iterations and the staged ones go on from there."""
    n = 20000
    g = graphs.from_edges(n, [(i, i + 1, 1.0 + 0.25 * (i % 7)) for i in range(n - 1)], default_outlets=[0])
    m = TerrainModel2D(np.arange(n, dtype=np.float64), np.zeros(n), g.area, g.row_ptr, g.col, g.length,
                       g.default_outlets)
    p = ParameterArrays(n, erodibility=np.random.default_rng(1).uniform(0.5, 2.0, n))
    e, it, used = _solve(m, p, 12, resident=None)
    f, jt, _ = _solve(m, p, 12, resident=False)
    assert used and it == jt and _same(e, f)


def test_graphs_that_are_not_simple_keep_the_staged_iterations():
    g = graphs.from_edges(4, [(0, 1, 1.0), (1, 2, 1.0), (1, 2, 2.0), (2, 3, 1.0)], default_outlets=[0])
    m = TerrainModel2D(np.arange(4.0), np.zeros(4), g.area, g.row_ptr, g.col, g.length, g.default_outlets)
    _, _, used = _solve(m, ParameterArrays(4), 3)
    assert not used


@pytest.mark.parametrize("make", [graphs.line, graphs.star, graphs.two_components,
                                  lambda: graphs.grid(40, 37, unit_lengths=True),
                                  lambda: graphs.grid(61, 50, jitter=0.3, seed=2)])
@pytest.mark.parametrize("slope", [None, 0.2])
def test_small_graphs_against_oracle(orc, make, slope):
    g = make()
    xs = np.arange(g.n, dtype=np.float64) if g.xs is None else g.xs
    ys = np.zeros(g.n) if g.ys is None else g.ys
    m = TerrainModel2D(xs, ys, g.area, g.row_ptr, g.col, g.length, g.default_outlets)
    p = ParameterArrays(g.n, max_slope=slope)
    e, it, used = _solve(m, p, 30)
    r = orc.generate(g, p.base, p.erodibility, p.uplift, p.is_outlet, max_slope=p.max_slope, max_iter=30)
    assert used and it == r["iters"] and _same(e, r["elev"])


@pytest.mark.parametrize("bad", [np.nan, np.inf, -1.0, 0.0])
def test_odd_erodibility(bad):
    """Values out of the ordinary travel through the published markers unchanged."""
    m, p = _case(3000, 4, False)
    p.erodibility[::97] = bad
    e, it, used = _solve(m, p, 6)
    f, jt, _ = _solve(m, p, 6, resident=False)
    assert used and it == jt
    nan = np.isnan(f)
    assert np.array_equal(np.isnan(e), nan) and _same(e[~nan], f[~nan])


def test_packed_terrains_equal_solo_solves():
    sizes = [1500, 40, 26000, 3, 9001, 1024, 60007, 700]
    cases = [_case(n, i + 1, i == 2) for i, n in enumerate(sizes)]
    g = BatchGenerator().set_models([m for m, _ in cases]).set_parameters([p for _, p in cases])
    outs = [np.array(t.elevations()) for t in g.set_max_iteration(60).generate()]
    for (m, p), e, it in zip(cases, outs, g.last_terrain_iterations):
        f, jt, _ = _solve(m, p, 60, resident=False)
        assert it == jt and _same(e, f)
