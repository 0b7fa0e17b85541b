"""The VJP's bounded waits (run with -m gpu), on the transposed halo sweeps and on the phased ones
(UFE_SSA_HALO=0): a wait that runs out is reported as UFE_TIMEOUT, nothing of the call is left on the
handle's stream (columns are queued ahead), and the next call gives the same gradients as before."""
import numpy as np
import pytest
import torch

from conftest import oracle_aaac, oracle_inputs, rel_l2

from ufemism_gb300 import _native as nat
from ufemism_gb300 import api

pytestmark = pytest.mark.gpu

GRADIENTS = ("dJ_dlogbeta_sq_AaAc", "dJ_dhx_AaAc", "lambda_U_AaAc", "lambda_V_AaAc")


@pytest.fixture(scope="module")
def solved():
    api.init(0)
    m = oracle_aaac("1k")
    ssa, _, _ = oracle_inputs(m)
    p = api.default_params(precision=nat.UFE_FP64, SSA_RN_tol=1e-9, SSA_max_residual_UV=1e-9,
                           SSA_max_outer_loops=200, SSA_max_inner_loops=200000)
    dm = api.DeviceMesh(m)
    rc, out, _ = dm.solve_ssa(ssa, p)
    assert rc == 0
    rng = np.random.default_rng(11)
    dJ = {k: rng.standard_normal(out[k].shape) for k in ("U_SSA", "V_SSA", "Ux_SSA_Ac", "Uy_SSA_Ac")}
    rc, ref, _ = dm.ssa_vjp(dJ, p, method=nat.UFE_VJP_SOR)
    assert rc == 0
    yield dm, p, dJ, ref
    dm.close()


@pytest.mark.parametrize("halo", ["1", "0"])
@pytest.mark.parametrize("restart", [12, 100])
def test_wait_timeout_reported_and_handle_usable(solved, halo, restart, monkeypatch):
    dm, p, dJ, ref = solved
    monkeypatch.setenv("UFE_SSA_HALO", halo)
    rc, first, st = dm.ssa_vjp(dJ, p, restart=restart)
    assert rc == 0
    for k in GRADIENTS:
        assert rel_l2(first[k], ref[k]) <= 1e-8, k
    monkeypatch.setenv("UFE_WAIT_TIMEOUT_NS", "5")
    rc, _, _ = dm.ssa_vjp(dJ, p, restart=restart, check=False)
    assert rc == nat.UFE_TIMEOUT and "timed out" in nat.last_error()
    assert torch.cuda.ExternalStream(dm.stream).query()
    monkeypatch.delenv("UFE_WAIT_TIMEOUT_NS")
    rc, again, st2 = dm.ssa_vjp(dJ, p, restart=restart)
    assert rc == 0 and st2["sweeps"] == st["sweeps"]
    for k in GRADIENTS:
        assert np.array_equal(again[k], first[k]), k


def test_no_device_memory_for_the_program(monkeypatch):
    """Where the device has no room for the transposed halo sweeps' program, the phased sweeps run. (The
    program of this mesh takes about 80 MB; all but 32 MB of the device is taken.)"""
    api.init(0)
    m = oracle_aaac("50k")
    ssa, _, _ = oracle_inputs(m)
    p = api.default_params(precision=nat.UFE_MIXED)
    dm = api.DeviceMesh(m)
    dm.solve_ssa(ssa, p)
    rng = np.random.default_rng(12)
    dJ = {k: rng.standard_normal(n) for k, n in (("U_SSA", m.base.nV), ("V_SSA", m.base.nV), ("Ux_SSA_Ac", m.nAc),
                                                 ("Uy_SSA_Ac", m.nAc))}
    monkeypatch.setenv("UFE_SSA_HALO", "0")
    rc0, phased, _ = dm.ssa_vjp(dJ, p)
    monkeypatch.delenv("UFE_SSA_HALO")
    assert rc0 == 0
    torch.cuda.empty_cache()
    taken = torch.empty(max(0, torch.cuda.mem_get_info()[0] - (32 << 20)), dtype=torch.uint8, device="cuda")
    try:
        rc, got, _ = dm.ssa_vjp(dJ, p)
    finally:
        del taken
        torch.cuda.empty_cache()
    assert rc == 0
    for k in GRADIENTS:
        assert np.array_equal(got[k], phased[k]), k
    dm.close()
