"""Packed terrains by both routes, the staged passes and the resident solve, against the oracle:
terrains that settle at different iterations and sit out the others' (tiles, rounds, skeleton),
tiles that hold parts of several terrains, slope limits, lakes; and which route a pack takes."""
import numpy as np
import pytest

from fastlem_gb300 import ParameterArrays, _lib, workloads
from fastlem_gb300.batch import BatchGenerator, TerrainBatch
from tests import graphs
from tests.test_gpu_resident import _same

pytestmark = pytest.mark.gpu


def _terrains(slope):
    """Sizes around and far from the tile's 2,048; outlets along the border, the hull or at one
    site (every other basin is a lake); default uplift, which settles, and uneven."""
    out = []
    for i, (n, outlets) in enumerate([(3, "one"), (300, "border"), (2048, "hull"), (2047, "border"), (7000, "one"),
                                      (64, "border"), (2500, "hull"), (12000, "border"), (1, None), (900, "one")]):
        r = np.random.default_rng(i + 1)
        if n == 1:
            g = graphs.from_edges(1, [], default_outlets=[0])
            from fastlem_gb300 import TerrainModel2D
            m = TerrainModel2D(np.zeros(1), np.zeros(1), g.area, g.row_ptr, g.col, g.length, g.default_outlets)
        else:
            m = workloads.build_model(n, n ** 0.5, i + 1, 0)
        is_outlet = np.zeros(n, bool)
        if outlets == "border":
            is_outlet = workloads.border_outlets(m, n ** 0.5, 0.05 * n ** 0.5)
        elif outlets == "one":
            is_outlet[int(np.argmin(m.xs))] = True
        uneven = i % 3 == 1
        out.append((m, ParameterArrays(
            n, erodibility=np.exp(r.normal(0, 0.5, n)), uplift_rate=r.uniform(0.5, 1.5, n) if uneven else 1.0,
            base_elevation=r.uniform(0, 2, n) if uneven else 0.0, is_outlet=is_outlet,
            max_slope=np.where(r.random(n) < 0.3, np.nan, r.uniform(0.05, 0.8, n)) if slope and i % 2 else None)))
    return out


@pytest.mark.parametrize("resident", [0, 1])
@pytest.mark.parametrize("slope", [False, True])
def test_both_routes(orc, slope, resident):
    cases = _terrains(slope)
    want = []
    for m, p in cases:
        r = orc.generate(graphs.from_model(m), p.base, p.erodibility, p.uplift, p.is_outlet,
                         max_slope=p.max_slope, max_iter=70)
        want.append((r["elev"], r["iters"]))
    assert len({it for _, it in want}) > 3 and min(it for _, it in want) < 10
    batch = TerrainBatch([m for m, _ in cases])
    old = _lib.set_tuning(resident=resident)
    try:
        for _ in range(2):
            g = BatchGenerator().set_batch(batch).set_parameters([p for _, p in cases]).set_max_iteration(70)
            outs = g.generate()
            for t, ((e, it), o) in enumerate(zip(want, outs)):
                assert int(g.last_terrain_iterations[t]) == it, t
                assert _same(np.array(o.elevations()), e), t
            assert g.last_iterations == max(it for _, it in want)
    finally:
        _lib.set_tuning(**old)
    stats = _lib.kernel_stats(batch.handle())
    assert (stats["resident_solve"][0] > 0) == bool(resident)
    assert (stats["kahn_rounds"][0] > 0) == (not resident)


@pytest.mark.parametrize("sites, slope, resident", [(3_100_000, False, True), (3_200_000, False, False),
                                                    (3_200_000, True, True), (5_300_000, True, False)])
def test_large_packs_by_the_rule(sites, slope, resident):
    n = 50000
    models = [workloads.build_model(n, n ** 0.5, s, 0) for s in (1, 2)]
    params = [ParameterArrays(n, is_outlet=workloads.border_outlets(m, n ** 0.5, 3.0), max_slope=0.5 if slope else None)
              for m in models]
    k = sites // n
    batch = TerrainBatch([models[i % 2] for i in range(k)])
    g = BatchGenerator().set_batch(batch).set_parameters([params[i % 2] for i in range(k)]).set_max_iteration(3)
    outs = [np.array(t.elevations()) for t in g.generate()]
    stats = _lib.kernel_stats(batch.handle())
    assert (stats["resident_solve"][0] > 0) == resident and (stats["kahn_rounds"][0] > 0) == (not resident)
    old = _lib.set_tuning(resident=0)
    try:
        small = BatchGenerator().set_models(models).set_parameters(params).set_max_iteration(3)
        want = [np.array(t.elevations()) for t in small.generate()]
    finally:
        _lib.set_tuning(**old)
    assert all(_same(e, want[i % 2]) for i, e in enumerate(outs))
