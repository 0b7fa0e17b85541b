"""A linear solve with NaN rows is not reported as converged (run with -m gpu): every mode runs to the
sweep limit, on the halo sweeps, on the phased ones and in a batch."""
import numpy as np
import pytest

from conftest import oracle_aaac, oracle_inputs

from ufemism_gb300 import _native as nat
from ufemism_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("halo", ["1", "0"])
@pytest.mark.parametrize("mode", ["mixed", "fp64", "exact"])
@pytest.mark.parametrize("everywhere", [False, True])
def test_nan_rows_do_not_converge(mode, halo, everywhere, monkeypatch):
    api.init(0)
    monkeypatch.setenv("UFE_SSA_HALO", halo)
    m = oracle_aaac("1k")
    ssa, _, _ = oracle_inputs(m)
    beta = np.full(m.nVAaAc, 1e3)
    beta[np.arange(m.nVAaAc) if everywhere else [m.nVAaAc // 2]] = np.nan
    ssa = dict(ssa, beta_sq_AaAc=beta)
    p = api.default_params(precision=nat.UFE_MIXED if mode == "mixed" else nat.UFE_FP64, fp64_exact=int(mode == "exact"),
                           SSA_max_inner_loops=60, SSA_max_outer_loops=3)
    dm = api.DeviceMesh(m)
    rc, out, st = dm.solve_ssa(ssa, p, check=False)
    dm.close()
    assert np.isnan(out["U_SSA"]).any()
    assert rc == nat.UFE_NOT_CONVERGED and st["not_converged"] == st["linear_solves"] == 3
    assert list(st["sweeps"]) == [60] * 3 and np.isnan(st["last_max_residual"])
    if halo == "1":
        b = api.Batch([m, m])
        b.upload(0, ssa, p)
        b.upload(1, dict(ssa, beta_sq_AaAc=np.full(m.nVAaAc, 1e3)), p)
        rc, stats, _ = b.run(p, check=False)
        b.close()
        assert stats[0]["not_converged"] == 3 and list(stats[0]["sweeps"]) == [60] * 3
        assert np.isfinite(stats[1]["last_max_residual"])
