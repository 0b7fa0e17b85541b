"""The batch autotuner tries the default packing, which spreads idle CTAs over a few members' teams, so that
what it returns is no slower than a batch that was never tuned (run with -m gpu)."""
import pytest

from ufemism_gb300 import _native as nat
from ufemism_gb300 import api
from ufemism_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("members", [1, 5])
def test_the_default_packing_is_a_candidate(members):
    api.init(0)
    ensemble = [wl.ensemble_member(n, 8200 + i) for i, n in enumerate((3000, 1200, 2100, 800, 1700)[:members])]
    p = api.default_params(precision=nat.UFE_MIXED, sliding_law=nat.UFE_SLIDING_LINEAR)
    best, tried = api.batch_autotune(ensemble, p)
    default = [e for e in tried if e["rows_per_cta"] == 0 and e["block"] == 1024]
    assert len(default) == 1
    fastest = min(tried, key=lambda e: e["device_ms"])
    assert (best["rows_per_cta"], best["block"]) == (fastest["rows_per_cta"], fastest["block"])
    assert fastest["device_ms"] <= default[0]["device_ms"]
    packed = [e for e in tried if e["rows_per_cta"] == 8192 and e["block"] == 1024]
    assert default[0]["grid_ctas"] > packed[0]["grid_ctas"]   # idle CTAs are used
    b = api.Batch([m for _, m, _ in ensemble], **{k: best[k] for k in ("team_ctas", "rows_per_cta", "block")})
    assert b.n == members
    b.close()
