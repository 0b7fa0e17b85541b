"""SIA columns with an infinite or overflowing thickness (run with -m gpu): the diffusivities are cut off
level by level as in the oracle (the power of the thickness is infinite, not NaN), and the other columns
keep their values. Only the base level and the averages of such a column are NaN."""
import numpy as np
import pytest

import oracle as orc
from conftest import oracle_aaac, oracle_inputs, rel_l2

from ufemism_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nZ", [15, 7])
@pytest.mark.parametrize("thickness", [np.inf, -np.inf, 1e110, 1e160, np.nan])
def test_sia_edges(thickness, nZ):
    api.init(0)
    m = oracle_aaac("1k")
    _, sia, _ = oracle_inputs(m)
    sheet = np.flatnonzero(sia["mask_sheet_Ac"] == 1)
    at = sheet[::7]
    Hi = sia["Hi_Ac"].copy()
    Hi[at] = thickness
    zeta = np.linspace(0.0, 1.0, nZ)
    sia = dict(sia, Hi_Ac=Hi, A_flow_Ac=np.asfortranarray(sia["A_flow_Ac"][:, :nZ]))
    with np.errstate(all="ignore"):
        ref = orc.solve_sia(m, sia, orc.default_params(zeta=zeta))
    dm = api.DeviceMesh(m)
    got = dm.solve_sia(sia, api.default_params(zeta=zeta))
    dm.close()
    others = np.setdiff1d(np.arange(m.nAc), at)
    for k in ("D_SIA_3D_Ac", "D_SIA_Ac", "Ux_SIA_Ac", "Uy_SIA_Ac", "Up_SIA_Ac", "Uo_SIA_Ac"):
        assert np.array_equal(np.isnan(got[k][at]), np.isnan(ref[k][at])), k
        finite = np.isfinite(ref[k][at])
        assert np.allclose(got[k][at][finite], ref[k][at][finite], rtol=1e-12, atol=0.0), k
        assert rel_l2(got[k][others], ref[k][others]) <= 1e-12, k


@pytest.mark.parametrize("thickness", [np.inf, 1e110])
def test_sia_3d_columns(thickness):
    api.init(0)
    m = oracle_aaac("1k")
    ssa, _, g = oracle_inputs(m)
    Hi = ssa["Hi"].copy()
    inner = np.flatnonzero((m.base.edge_index == 0) & (ssa["mask_sheet"] == 1))
    Hi[inner[::9]] = thickness
    A3 = np.asfortranarray(np.full((m.base.nV, 15), 1e-16))
    with np.errstate(all="ignore"):
        g = orc.update_geometry(m, Hi, ssa["Hb"], ssa["SL"])
        ref = orc.solve_sia_3d(m, g, A3, np.zeros(m.base.nV), np.zeros(m.base.nV), np.zeros(m.base.nV))
    dm = api.DeviceMesh(m)
    dm.geometry_attach(m)
    dm.geometry_update(Hi, ssa["Hb"], ssa["SL"])
    got = dm.solve_sia_3d(A3, np.zeros(m.base.nV), api.default_params())
    dm.close()
    for x, y, k in zip(got[:2], ref[:2], "UV"):
        assert np.array_equal(np.isnan(x), np.isnan(y)), k
        both = np.isfinite(x) & np.isfinite(y)
        assert rel_l2(x[both], y[both]) <= 1e-12, k
