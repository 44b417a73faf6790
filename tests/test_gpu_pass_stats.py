"""What the basin statistics say of the last pass, staged or resident: its leaves, and nothing
that an earlier pass left behind; algorithmic bytes for every kernel class that ran."""
import numpy as np
import pytest

from fastlem_gb300 import _lib
from fastlem_gb300._lib import check, lib
from tests import graphs
from tests.test_gpu_resident import _case, _solve

pytestmark = pytest.mark.gpu


def _leaves(orc, m, p, iters):
    """Sites that nothing drains to in the last of `iters` iterations."""
    g = graphs.from_model(m)
    e = orc.generate(g, p.base, p.erodibility, p.uplift, p.is_outlet, max_iter=iters - 1)["elev"]
    table = p.is_outlet.astype(np.uint8)
    nxt = orc.initial_tree(g, e, table)
    sub, lakes = orc.roots(table, nxt)
    if lakes:
        nxt = orc.remove_lakes_heap(g, nxt, np.flatnonzero(table).astype(np.uint32), sub)
    drains = nxt != np.arange(g.n)
    return g.n - len(np.unique(nxt[drains]))


@pytest.mark.parametrize("n", [3, 2049, 20011])
@pytest.mark.parametrize("resident", [True, False])
def test_leaves(orc, n, resident):
    m, p = _case(n, 4, False)
    if not p.is_outlet.any():
        p.is_outlet[0] = True
    for iters in (2, 5):
        _, it, used = _solve(m, p, iters, resident=resident)
        assert used == resident
        assert _lib.basin_stats(m.handle())["leaves"] == _leaves(orc, m, p, it)


def test_nothing_of_an_earlier_pass():
    m, p = _case(20011, 4, False)
    _solve(m, p, 3, resident=False)
    staged = _lib.basin_stats(m.handle())
    assert staged["skeleton_sites"] > 0 and staged["chains"] > 0
    _solve(m, p, 3)
    after = _lib.basin_stats(m.handle())
    assert after["leaves"] > 0 and all(v == 0 for k, v in after.items() if k != "leaves")
    assert len(_lib.round_trace(m.handle())[0]) == 1


@pytest.mark.parametrize("resident", [True, False])
def test_bytes(resident):
    """Every class that did anything has bytes (the rounds none when there are none, as in this
    terrain's passes outside the tiles), and none more than a few times what 5 iterations read and
    write altogether (93 B a site and 12 a slot)."""
    m, p = _case(60007, 4, False)
    _solve(m, p, 5, resident=resident)
    lib().fl_graph_reset_stats(m.handle())
    _solve(m, p, 5, resident=resident)
    whole = 5 * (93.0 * m.n + 12.0 * len(m.col))
    rounds = _lib.basin_stats(m.handle())["kahn_rounds"]
    for name, (launches, _, moved) in _lib.kernel_stats(m.handle()).items():
        if name == "kahn_rounds" and rounds == 0:
            assert moved == 0
        elif launches:
            assert 0 < moved < 4 * whole, name
