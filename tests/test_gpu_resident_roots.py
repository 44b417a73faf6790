"""Resident solve: a basin's sites need their root's response time and elevation from whichever
block has the root, over several blocks on the way.  Roots whose times and elevations change
from iteration to iteration (outlets with a falling slope limit), basins over many blocks and
thousands of basins across block borders: the staged iterations' bits."""
import numpy as np
import pytest

from fastlem_gb300 import ParameterArrays, workloads
from tests.test_gpu_resident import _same, _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slope", [False, True])
@pytest.mark.parametrize("n, outlets", [(6000, 1), (20011, 400), (60007, 1), (60007, 6000)])
def test_roots_in_other_blocks(n, outlets, slope):
    m = workloads.build_model(n, n ** 0.5, outlets + 3, 0)
    r = np.random.default_rng(n + outlets)
    out = np.zeros(n, bool)
    out[r.choice(n, outlets, replace=False)] = True
    ms = np.where(out, -0.03, r.uniform(0.1, 0.8, n)) if slope else None
    p = ParameterArrays(n, erodibility=np.exp(r.normal(0, 0.7, n)), uplift_rate=r.uniform(0.0, 2.0, n),
                        base_elevation=r.uniform(0, 2.0, n), is_outlet=out, max_slope=ms)
    f, jt, staged = _solve(m, p, 60, resident=False)
    assert not staged
    for _ in range(3):
        e, it, used = _solve(m, p, 60)
        assert used and it == jt and _same(e, f)
