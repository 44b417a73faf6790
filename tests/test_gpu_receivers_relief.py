"""Receivers on small relief: elevation differences below 2^-24 of the elevations, which the float
pairs leave to estimates from the doubles' bits; flat ground; both sides of the switch."""
import ctypes

import numpy as np
import pytest

from fastlem_gb300 import ParameterArrays, TerrainGenerator, _lib, workloads
from fastlem_gb300._lib import check, lib, ptr
from tests import graphs
from tests.test_gpu_parity import Handle
from tests.test_gpu_resident import _same, _solve

pytestmark = pytest.mark.gpu


def _fields(rng, n):
    flat = np.zeros(n)
    yield "flat", flat + 7.0
    yield "sea", np.where(rng.random(n) < 0.5, 0.0, rng.uniform(0, 1, n))
    for base in (1.0, 1e3, 1e7, 1e12, 2.0 ** 96, 2.0 ** 100, 2.0 ** -70, 2.0 ** -75, 1e-300, 1e300):
        for rel in (2.0 ** -22, 2.0 ** -24, 2.0 ** -25, 2.0 ** -30, 2.0 ** -50):
            e = base * (1.0 + rng.uniform(0, 4, n) * rel)
            yield f"{base} {rel}", e
            yield f"around {base} {rel}", base * (1.0 + rng.uniform(-2, 2, n) * rel)
            e = np.where(rng.random(n) < 0.05, rng.choice([0.0, -0.0, -base, np.nan, np.inf, 1e-3 * base], n), e)
            yield f"mixed {base} {rel}", e
    yield "steps", 1e6 + np.round(rng.uniform(0, 8, n)) * 2.0 ** -30
    yield "negative", -1e6 - rng.uniform(0, 1e-3, n)


@pytest.mark.parametrize("make", [lambda: graphs.random_delaunay(3000, seed=21), lambda: graphs.star(40),
                                  lambda: graphs.grid(40, 37, unit_lengths=True)])
def test_receivers(orc, make):
    g = make()
    rng = np.random.default_rng(5)
    with Handle(g) as h:
        for name, elev in _fields(rng, g.n):
            table = (rng.uniform(size=g.n) < 0.05).astype(np.uint8)
            want = orc.initial_tree(g, elev, table)
            got = np.empty(g.n, np.uint32)
            hl = ctypes.c_int()
            check(lib().fl_probe_receivers(h.h, ptr(elev), ptr(table), ptr(got), ctypes.byref(hl)))
            assert np.array_equal(got, want), name


def _case(n, base):
    m = workloads.build_model(n, n ** 0.5, 1, 0)
    return m, ParameterArrays(n, erodibility=np.exp(np.random.default_rng(2).normal(0, 0.5, n)), base_elevation=base,
                              is_outlet=workloads.border_outlets(m, n ** 0.5, 0.02 * n ** 0.5))


@pytest.mark.parametrize("base", [1e6, 1e9])
def test_solve_on_a_large_base(orc, base):
    m, p = _case(5000, base)
    want = orc.generate(graphs.from_model(m), p.base, p.erodibility, p.uplift, p.is_outlet, max_iter=20)
    for resident in (True, False):
        e, it, used = _solve(m, p, 20, resident=resident)
        assert used == resident and it == want["iters"] and _same(e, want["elev"])


def test_large_base_costs_no_f64_scan():
    """The receivers of a million sites took five times as long on a base elevation of 10^7 as on
    none while every row was scanned in f64."""
    ms = []
    m, _ = _case(1000000, 0.0)
    for base in (0.0, 1e7):
        g = TerrainGenerator.default().set_model(m).set_parameters(_case(1000000, base)[1]).set_max_iteration(12)
        g.generate()
        check(lib().fl_graph_set_timing(m.handle(), 1))
        lib().fl_graph_reset_stats(m.handle())
        g.generate()
        ms.append(_lib.kernel_stats(m.handle())["receivers"][1])
        check(lib().fl_graph_set_timing(m.handle(), 0))
    print(ms)
    assert ms[1] < 4.0 * ms[0]
