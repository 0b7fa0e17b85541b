"""The planner's default packing accepts what the packing without spreading accepts (host only), also
where spreading idle CTAs over many uneven members would give more team sizes than there are classes."""
import numpy as np
import pytest

from ufemism_gb300 import api


@pytest.mark.parametrize("resident", [152, 608, 1300, 8000])
@pytest.mark.parametrize("seed", range(40))
def test_spreading_refuses_nothing(resident, seed):
    rng = np.random.default_rng(seed)
    rows = np.exp(rng.uniform(np.log(200), np.log(3e6), int(rng.integers(17, 60)))).astype(np.int64)
    try:
        packed, _, _ = api.batch_plan(rows, resident, rows_per_cta=8192)
    except api.nat.UfeError:
        return
    team, classes, grid = api.batch_plan(rows, resident)
    assert np.all(team >= packed) and len(classes) <= 16 and grid <= resident
