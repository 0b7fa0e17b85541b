"""The transposed halo sweeps of the VJP's GMRES iteration (run with -m gpu) where their launches can go
wrong: fewer and more sweeps per iteration than one launch does, meshes of one patch and of many, both
sliding laws. Every number of sweeps per iteration solves the same system, so the gradients agree with
the plain transposed SOR iteration (the phased kernel) to the adjoint tests' 1e-8."""
import numpy as np
import pytest

from conftest import oracle_aaac, oracle_inputs, rel_l2

from ufemism_gb300 import _native as nat
from ufemism_gb300 import api
from ufemism_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,law", [("tiny", nat.UFE_SLIDING_LINEAR), ("1k", nat.UFE_SLIDING_COULOMB_REGULARISED)])
def test_sweeps_per_iteration(name, law):
    api.init(0)
    m = oracle_aaac(name)
    ssa, _, _ = oracle_inputs(m, "dome")
    ssa["beta_sq_AaAc"] = np.exp(wl.log_beta_field(m, std=0.5, ell=100e3, seed=3))
    p = api.default_params(precision=nat.UFE_FP64, sliding_law=law, SSA_RN_tol=1e-9, SSA_max_residual_UV=1e-9,
                           SSA_max_outer_loops=200, SSA_max_inner_loops=200000)
    dm = api.DeviceMesh(m)
    rc, out, _ = dm.solve_ssa(ssa, p)
    assert rc == 0
    rng = np.random.default_rng(4)
    dJ = {k: rng.standard_normal(out[k].shape) for k in ("U_SSA", "V_SSA", "Ux_SSA_Ac", "Uy_SSA_Ac")}
    rc, ref, _ = dm.ssa_vjp(dJ, p, geom_mesh=m, method=nat.UFE_VJP_SOR)
    assert rc == 0
    for n in (1, 3, 8, 9, 17):
        rc, got, st = dm.ssa_vjp(dJ, p, geom_mesh=m, sweeps_per_iteration=n, restart=60)
        assert rc == 0 and st["sweeps"] % n == 0, (n, rc, st)
        for k in ("dJ_dlogbeta_sq_AaAc", "dJ_dHi", "lambda_U_AaAc"):
            assert rel_l2(got[k], ref[k]) <= 1e-8, (n, k)
    dm.close()
