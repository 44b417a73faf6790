"""Graphs with rows too long for the tiles: those sites are left to the rounds, all others stay
in the tiles.  Rows that name a site twice, or not at all although it names theirs, turn the
tiles off only where they are short."""
import numpy as np
import pytest

from fastlem_gb300 import ParameterArrays, TerrainModel2D, _lib
from tests import graphs
from tests.test_gpu_resident import _same, _solve

pytestmark = pytest.mark.gpu


def _rows(g):
    return [list(zip(g.col[a:b].tolist(), g.length[a:b].tolist())) for a, b in zip(g.row_ptr, g.row_ptr[1:])]


def _model(rows, g):
    row = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint32)
    return TerrainModel2D(g.xs, g.ys, g.area, row, np.array([j for r in rows for j, _ in r], np.uint32),
                          np.array([w for r in rows for _, w in r]), g.default_outlets)


def _hub(n, spokes, seed):
    """A random terrain with one site that also borders `spokes` far ones."""
    g = graphs.random_delaunay(n, seed)
    rows = _rows(g)
    r = np.random.default_rng(seed)
    near = {j for j, _ in rows[n // 2]} | {n // 2}
    for f in r.choice(n, spokes, replace=False).tolist():
        if f not in near:
            rows[n // 2].append((f, 1.0 + r.random()))
            rows[f].append((n // 2, rows[n // 2][-1][1]))
    return _model(rows, g), rows, g


def _outside_tiles(m):
    """Sites of the last pass's rounds and skeleton: without tiles all."""
    off, _, _ = _lib.round_trace(m.handle())
    return int(off[-1]) + _lib.basin_stats(m.handle())["skeleton_sites"]


def _params(n):
    r = np.random.default_rng(n)
    return ParameterArrays(n, erodibility=np.exp(r.normal(0, 0.5, n)), uplift_rate=r.uniform(0.0, 2.0, n),
                           base_elevation=r.uniform(0, 1e-3, n))


@pytest.mark.parametrize("spokes", [20, 60, 100, 1500])
def test_long_rows_keep_the_tiles(orc, spokes):
    n = 9000
    m, _, _ = _hub(n, spokes, spokes)
    p = _params(n)
    want = orc.generate(graphs.from_model(m), p.base, p.erodibility, p.uplift, p.is_outlet, max_iter=8)
    e, it, used = _solve(m, p, 8, resident=False)
    assert not used and it == want["iters"] and _same(e, want["elev"])
    assert _outside_tiles(m) < n // 2


@pytest.mark.parametrize("what", ["short_twice", "long_twice", "one_sided"])
def test_odd_rows(what):
    n = 9000
    m, rows, g = _hub(n, 100, 7)
    hub = n // 2
    plain = _model(rows, g)
    if what == "short_twice":
        rows[100].append(rows[100][0])
    elif what == "long_twice":
        rows[hub].append(rows[hub][0])
    else:                                       # a short row no longer names a neighbour of its site
        rows[100] = rows[100][1:]
    m = _model(rows, g)
    p = _params(n)
    _, _, used = _solve(m, p, 1, resident=False)
    assert not used
    if what == "long_twice":
        assert _outside_tiles(m) < n // 2
    else:
        assert _outside_tiles(m) == n
    _solve(plain, p, 1, resident=False)
    assert _outside_tiles(plain) < n // 2
