"""The SIA, the 3-D SIA and the ice's physical properties with numbers of levels other than 15 (run with
-m gpu), against the oracle (tolerances of the 15-level tests)."""
import numpy as np
import pytest

import oracle as orc
from conftest import oracle_aaac, oracle_inputs, rel_l2

from ufemism_gb300 import _native as nat
from ufemism_gb300 import api

pytestmark = pytest.mark.gpu


def levels(nZ):
    return np.linspace(0.0, 1.0, nZ) ** 0.7


@pytest.mark.parametrize("nZ", [2, 3, 14, 16, 64])
def test_sia(nZ):
    api.init(0)
    m = oracle_aaac("1k")
    _, sia, _ = oracle_inputs(m, "marine")
    rng = np.random.default_rng(nZ)
    sia = dict(sia, A_flow_Ac=np.asfortranarray(1e-16 * rng.uniform(0.5, 2.0, (m.nAc, nZ))))
    ref = orc.solve_sia(m, sia, orc.default_params(zeta=levels(nZ)))
    dm = api.DeviceMesh(m)
    p = api.default_params(zeta=levels(nZ))
    got = dm.solve_sia(sia, p)
    without = dm.solve_sia(sia, p, want_3d=False)
    dm.close()
    for k in ("D_SIA_3D_Ac", "D_SIA_Ac", "Ux_SIA_Ac", "Uy_SIA_Ac", "Up_SIA_Ac", "Uo_SIA_Ac", "U_SIA", "V_SIA", "D_SIA"):
        assert rel_l2(got[k], ref[k]) <= 1e-12, k
        if k != "D_SIA_3D_Ac":
            assert np.array_equal(without[k], got[k]), k


@pytest.mark.parametrize("nZ", [2, 3, 14, 16, 64])
def test_sia_3d(nZ):
    api.init(0)
    m = oracle_aaac("1k")
    ssa, _, g = oracle_inputs(m, "marine")
    nV = m.base.nV
    rng = np.random.default_rng(nZ)
    A3 = np.asfortranarray(1e-16 * rng.uniform(0.5, 2.0, (nV, nZ)))
    dHb_dt = rng.normal(size=nV) * 1e-3
    p = api.default_params(zeta=levels(nZ))
    dm = api.DeviceMesh(m)
    dm.geometry_attach(m)
    dm.geometry_update(ssa["Hi"], ssa["Hb"], ssa["SL"])
    got = dm.solve_sia_3d(A3, dHb_dt, p)
    dm.close()
    ref = orc.solve_sia_3d(m, g, A3, dHb_dt, np.zeros(nV), np.zeros(nV), zeta=levels(nZ))
    for x, y, k in zip(got, ref, "UVW"):
        assert rel_l2(x, y) <= 1e-12, k


@pytest.mark.parametrize("nZ", [2, 14, 64])
def test_physical_properties(nZ):
    api.init(0)
    m = oracle_aaac("1k")
    ssa, _, g = oracle_inputs(m, "marine")
    rng = np.random.default_rng(nZ)
    Ti = np.asfortranarray(240.0 + 30.0 * rng.random((m.base.nV, nZ)))
    dm = api.DeviceMesh(m)
    dm.geometry_attach(m)
    dm.geometry_update(ssa["Hi"], ssa["Hb"], ssa["SL"])
    got = dm.ice_physical_properties(api.default_params(zeta=levels(nZ)), Ti, flow_law=nat.UFE_FLOW_ARRHENIUS)
    dm.close()
    ref = orc.ice_physical_properties(m, ssa["Hi"], g["mask_sheet"], g["mask_sheet_Ac"], Ti, zeta=levels(nZ))
    assert set(got) <= set(ref)
    for k in got:
        assert rel_l2(got[k], ref[k]) <= 1e-12, k
