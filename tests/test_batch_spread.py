"""The planner's default packing spreads idle CTAs (host only): teams only grow, the budget and the
per-CTA limits hold, the slowest member's team grows first, and a full machine is left as it is."""
import numpy as np
import pytest

from ufemism_gb300 import api
from ufemism_gb300 import workloads as wl


@pytest.mark.parametrize("n,lo,hi", [(1, 400, 401), (3, 500, 9000), (24, 2000, 16000), (64, 300, 6000), (256, 2000, 50000)])
@pytest.mark.parametrize("resident", [1, 7, 152, 608])
def test_default_packing_spreads_idle_ctas(n, lo, hi, resident):
    rows = 4 * np.asarray(wl.ensemble_sizes(n, lo=lo, hi=hi), dtype=np.int64)
    try:
        base, _, base_grid = api.batch_plan(rows, resident, rows_per_cta=8192)
    except Exception:
        with pytest.raises(Exception):
            api.batch_plan(rows, resident)
        return
    t, classes, grid = api.batch_plan(rows, resident)
    assert np.all(t >= base) and grid <= resident and len(classes) <= 16
    assert np.all(rows // t >= 32) and np.all(rows / t <= 1024 * 32 * 3 // 4)
    assert grid == sum(s * k for s, k in classes)
    if base.sum() >= resident:
        assert np.array_equal(t, base)
    else:
        assert t.sum() <= resident   # every member still has its team at once
        grown = t > base
        if n > 1 and grown.any():
            assert grown[np.argmax(rows)] or t[np.argmax(rows)] * 2 > resident // 2 + 1
