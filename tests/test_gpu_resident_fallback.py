"""Terrains that the resident solve cannot finish: the staged iterations take them over, and
only them; a pack's other terrains keep what the resident solve computed."""
import numpy as np
import pytest

from fastlem_gb300 import ParameterArrays, TerrainModel2D, _lib, workloads
from fastlem_gb300.batch import BatchGenerator, TerrainBatch
from tests import graphs
from tests.test_gpu_resident import _case, _same, _solve

pytestmark = pytest.mark.gpu


def _scrambled(n, seed, slope):
    """A terrain whose coordinates say nothing about its edges, so that its blocks' ranges are
    arbitrary and nearly every donor is in another block: more than a block's 512 where its
    share is more sites than that (100,000 over 152 blocks)."""
    m, p = _case(n, seed, slope)
    r = np.random.default_rng(seed)
    return TerrainModel2D(r.permutation(m.xs), r.permutation(m.ys), m.area, m.row_ptr, m.col, m.length,
                          m.default_outlets), p


def _launches(handle):
    s = _lib.kernel_stats(handle)
    return s["resident_solve"][0], s["kahn_rounds"][0]


def _oracle(orc, m, p, iters):
    r = orc.generate(graphs.from_model(m), p.base, p.erodibility, p.uplift, p.is_outlet,
                     max_slope=p.max_slope, max_iter=iters)
    return r["elev"], r["iters"]


@pytest.mark.parametrize("slope", [False, True])
def test_no_room_alone(orc, slope):
    m, p = _scrambled(100000, 5, slope)
    want, iters = _oracle(orc, m, p, 5)
    for call in range(2):
        e, it, used = _solve(m, p, 5)
        res, kahn = _launches(m.handle())
        assert used == (call == 0)            # not tried again
        assert kahn > 0 and it == iters and _same(e, want)


@pytest.mark.parametrize("slope", [False, True])
def test_no_room_in_a_pack(orc, slope):
    """Before, one such terrain sent the whole pack back to the start."""
    cases = [_case(2500, 1, slope), _scrambled(30000, 5, slope), _case(40, 2, False), _case(90001, 4, slope)]
    batch = TerrainBatch([m for m, _ in cases])
    want = [_oracle(orc, m, p, 12) for m, p in cases]
    seen = 0
    for call in range(2):
        g = BatchGenerator().set_batch(batch).set_parameters([p for _, p in cases]).set_max_iteration(12)
        outs = g.generate()
        res, kahn = _launches(batch.handle())
        assert res > seen and kahn > 0        # the others stay with the resident solve
        seen = res
        for t, ((e, it), o) in enumerate(zip(want, outs)):
            assert int(g.last_terrain_iterations[t]) == it, t
            assert _same(np.array(o.elevations()), e), t
        assert g.last_iterations == max(it for _, it in want)
