"""The work that a user of this library has it do, as cases to time: velocity solves of one mesh
(mixed and FP64, both sliding laws, cold and warm starts), an ensemble, a gradient, the SIA on
host and on device arrays, the thermodynamics' inputs, the geometry and thickness updates, and a
whole time step. Meshes are the seeded generator's: its presets (``mesh`` a text) or a number of
vertices. A model keeps its mesh for many steps, so a case has one mesh; the ice on it (thickness,
bed, friction, temperature, mass balance) comes from the seed.
"""
import ctypes as ct
import math
from functools import lru_cache

import numpy as np
import torch

from ufemism_gb300 import _native as nat
from ufemism_gb300 import api, meshgen, workloads

RHO_I, RHO_W, GRAV = 910.0, 1028.0, 9.81
ZETA = api.ZETA_DEFAULT
NZ = len(ZETA)
SSA_OUT = ("U_SSA", "V_SSA", "Ux_SSA_Ac", "Uy_SSA_Ac", "N_AaAc", "Up_SSA_Ac", "Uo_SSA_Ac", "eta_AaAc", "S_AaAc",
           "tau_c_AaAc", "phi_fric_AaAc")


def listed():
    return [
        # the headline configuration: one cold solve of the 200k-vertex dome in the mixed precision
        dict(name="ssa-200k-mixed", kind="ssa", mesh="200k", geometry="dome", law="linear", precision="mixed",
             warm=False, gl=False),
        # the solve of a time step: the velocities of the step before as the start, 16k vertices
        dict(name="ssa-16k-mixed-warm", kind="ssa", mesh="16k", geometry="dome", law="linear", precision="mixed",
             warm=True, gl=False),
        # a marine ice sheet under the reference's own sliding law, 4k vertices: many sweeps of small work
        dict(name="ssa-4k-marine-coulomb-mixed", kind="ssa", mesh="4k", geometry="marine", law="coulomb",
             precision="mixed", warm=False, gl=False),
        # the FP64 default on a regional mesh of 50k vertices
        dict(name="ssa-50k-fp64", kind="ssa", mesh="50k", geometry="dome", law="linear", precision="fp64",
             warm=False, gl=False),
        # a check against the Fortran model's own numbers: the parity mode on a small marine mesh
        dict(name="ssa-1k-marine-coulomb-exact", kind="ssa", mesh="1k", geometry="marine", law="coulomb",
             precision="exact", warm=False, gl=False),
        # a friction ensemble of uneven members, inputs up and results down every time
        dict(name="ensemble-24-mixed", kind="ensemble", members=24, lo=2000, hi=16000, precision="mixed"),
        # an inversion's gradient: the adjoint of a solve on 16k vertices
        dict(name="vjp-16k", kind="vjp", mesh="16k", law="linear"),
        # SIA velocities of a 100k-vertex ice sheet from and to the Fortran model's host arrays
        dict(name="sia-100k", kind="sia", mesh="100k", where="host"),
        # the smallest call: the SIA of a small mesh on arrays that stay on the device
        dict(name="sia-1k-device", kind="sia", mesh="1k", where="device"),
        # what the thermodynamics takes: physical properties, 3-D velocities, upwind derivatives
        dict(name="thermo-50k", kind="thermo", mesh="50k"),
        # geometry, masks and ice thickness of a time step, 100k vertices
        dict(name="geometry-100k", kind="geometry", mesh="100k"),
        # one whole velocity and thickness step with the fields kept on the device, 50k vertices
        dict(name="step-50k", kind="step", mesh="50k"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["ssa", "ssa", "ssa", "ssa", "ensemble", "vjp", "sia", "thermo", "geometry", "step"])
    if kind == "ssa":
        precision = rng.choice(["mixed", "mixed", "fp64", "exact"])
        geometry = rng.choice(["dome", "dome", "marine"])
        law = "linear" if geometry == "dome" else "coulomb"
        hi = dict(mixed=150000, fp64=40000, exact=8000)[precision] if geometry == "dome" else 2500
        return dict(kind="ssa", mesh=size(300, hi), geometry=geometry, law=law, precision=precision,
                    warm=rng.random() < 0.5, gl=geometry == "marine" and rng.random() < 0.25)
    if kind == "ensemble":
        lo = size(1000, 4000)
        return dict(kind="ensemble", members=rng.randint(3, 24), lo=lo, hi=size(lo + 500, 14000),
                    precision=rng.choice(["mixed", "mixed", "fp64"]))
    if kind == "vjp":
        return dict(kind="vjp", mesh=size(700, 15000), law=rng.choice(["linear", "coulomb"]))
    if kind == "sia":
        where = rng.choice(["host", "device"])
        return dict(kind="sia", mesh=size(300, 100000 if where == "host" else 60000), where=where)
    return dict(kind=kind, mesh=size(700, dict(thermo=50000, geometry=100000, step=40000)[kind]))


# ---------------------------------------------------------------------------------------- inputs
@lru_cache(maxsize=48)
def _mesh(size, mesh_seed=20261204):
    base = meshgen.dome_mesh(size) if isinstance(size, str) else meshgen.sized_mesh(size, mesh_seed)
    return base, api.build_aaac(base)


@lru_cache(maxsize=16)
def _cells(size):
    return workloads.areas_and_widths(_mesh(size)[0])


@lru_cache(maxsize=16)
def _triangles(size):
    """mesh%R and the triangles' derivative weights (NxTri, NyTri)."""
    base, _ = _mesh(size)
    V, T = np.asarray(base.V), np.asarray(base.Tri, dtype=np.int64) - 1
    (ax, ay), (bx, by), (cx, cy) = (V[T[:, k]].T for k in range(3))
    D = ax * (by - cy) + bx * (cy - ay) + cx * (ay - by)
    Nx = np.stack([(by - cy) / D, (cy - ay) / D, (ay - by) / D], axis=1)
    Ny = np.stack([(cx - bx) / D, (ax - cx) / D, (bx - ax) / D], axis=1)
    C = np.asarray(base.C, dtype=np.int64) - 1
    d = np.linalg.norm(V[np.maximum(C, 0)] - V[:, None, :], axis=2)
    R = np.where(C >= 0, d, np.inf).min(axis=1)
    return R, np.asfortranarray(Nx), np.asfortranarray(Ny)


def _params(law="linear", precision="mixed", gl=False):
    return api.default_params(
        sliding_law=nat.UFE_SLIDING_LINEAR if law == "linear" else nat.UFE_SLIDING_COULOMB_REGULARISED,
        precision=nat.UFE_MIXED if precision == "mixed" else nat.UFE_FP64, fp64_exact=int(precision == "exact"),
        use_analytical_GL_flux=int(gl))


def _ice(base, geometry, seed):
    """Hi, Hb, SL: a dome of 3600 m give or take 5 % on a flat bed, or on a marine bed."""
    rng = np.random.default_rng(seed)
    H0 = rng.uniform(3420.0, 3780.0)
    make = workloads.dome_geometry if geometry == "dome" else workloads.marine_geometry
    Hi, Hb, SL = make(base, H0=H0) if geometry == "dome" else make(base, seed=seed, H0=H0)
    return Hi, Hb, SL


def _friction(mesh, seed, std=1.0):
    return np.exp(workloads.log_beta_field(mesh, std=std, ell=100e3, seed=seed + 1))


def _temperature(base, seed):
    """Ice temperature (nV, nZ): colder inland and towards the surface, both Arrhenius branches."""
    x, y = np.asarray(base.V).T
    surface = 243.0 + 22.0 * np.hypot(x, y) / 750e3 + workloads.grf(x, y, 2.0, 150e3, seed)
    return np.asfortranarray(np.minimum(surface[:, None] + (271.0 - surface[:, None]) * ZETA[None, :] ** 2, 272.0))


def _earlier_velocities(dm, mesh, base, geometry, law, gl, seed, beta):
    """The velocities of the step before: the parity mode's solve of slightly thicker ice."""
    Hi, Hb, SL = _ice(base, geometry, seed)
    ssa, _ = workloads.prepare_inputs(mesh, 1.003 * Hi, Hb, SL)
    ssa["beta_sq_AaAc"] = beta
    _, out, _ = dm.solve_ssa(ssa, _params(law, "exact", gl), check=False)
    return {k: out[k] for k in ("U_SSA", "V_SSA", "Ux_SSA_Ac", "Uy_SSA_Ac", "N_AaAc")}


def prepare(case, seed):
    api.init(0)
    if case["kind"] == "ensemble":
        return _prepare_ensemble(case, seed)
    base, mesh = _mesh(case["mesh"])
    s = dict(kind=case["kind"], base=base, mesh=mesh, dm=api.DeviceMesh(mesh))
    if case["kind"] == "ssa":
        s["params"] = _params(case["law"], case["precision"], case["gl"])
        s["fields"], s["warm"] = _ssa_inputs(case, seed, s["dm"])
    elif case["kind"] == "vjp":
        s["params"] = _params(case["law"], "exact")
        ssa, _ = _ssa_inputs(dict(case, geometry="dome", gl=False, warm=False), seed, s["dm"])
        _, out, _ = s["dm"].solve_ssa(ssa, s["params"])
        # the misfit to observed surface velocities: 5 % off, smoothly
        rng = np.random.default_rng(seed + 7)
        s["dJ"] = {k: out[k] * rng.uniform(0.02, 0.08) + 0.1 * rng.standard_normal(out[k].shape)
                   for k in ("U_SSA", "V_SSA", "Ux_SSA_Ac", "Uy_SSA_Ac")}
    elif case["kind"] == "sia":
        s.update(_sia_inputs(case, seed))
        if case["where"] == "device":
            _sia_on_device(s)
    else:
        s["params"] = _params("linear", "mixed")
        s["dm"].geometry_attach(mesh)
        Hi, Hb, SL = _ice(base, "marine", seed)
        rng = np.random.default_rng(seed + 3)
        x, y = np.asarray(base.V).T
        s.update(Hi=Hi, Hb=Hb, SL=SL, Ti=_temperature(base, seed + 5), dHb_dt=1e-3 * rng.standard_normal(base.nV),
                 SMB=0.3 - 0.8 * np.hypot(x, y) / 750e3 + 0.05 * rng.standard_normal(base.nV),
                 BMB=-0.2 * rng.random(base.nV))
        s["A"], s["Cw"] = _cells(case["mesh"])
        if case["kind"] == "geometry":
            s["Up_SIA"], s["Up_SSA"] = _some_fluxes(mesh, Hi, seed)
        else:
            R, NxTri, NyTri = _triangles(case["mesh"])
            s["dm"].triangles_attach(base, R, NxTri, NyTri)
            if case["kind"] == "thermo":
                s["dm"].geometry_update(Hi, Hb, SL)
            else:
                s["beta"] = _friction(mesh, seed)
                s["warm"] = _earlier_velocities(s["dm"], mesh, base, "dome", "linear", False, seed, s["beta"])
                s["Hi"], s["Hb"], s["SL"] = _ice(base, "dome", seed)
                g = workloads.prepare_inputs(mesh, s["Hi"], s["Hb"], s["SL"])[0]
                s["mask_sheet"] = g["mask_sheet"]
    return s


def _ssa_inputs(case, seed, dm):
    base, mesh = _mesh(case["mesh"])
    ssa, _ = workloads.prepare_inputs(mesh, *_ice(base, case["geometry"], seed))
    if case["law"] == "linear":
        ssa["beta_sq_AaAc"] = _friction(mesh, seed, std=0.5 if base.nV > 20000 else 1.0)
    warm = None
    if case["warm"] and dm is not None:
        warm = _earlier_velocities(dm, mesh, base, case["geometry"], case["law"], case["gl"], seed,
                                   ssa.get("beta_sq_AaAc"))
    return ssa, warm


def _some_fluxes(mesh, Hi, seed):
    """Velocities along the Ac edges (m/yr) of the size that the thickness update meets."""
    rng = np.random.default_rng(seed + 11)
    Aci = np.asarray(mesh.Aci) - 1
    dH = Hi[Aci[:, 1]] - Hi[Aci[:, 0]]
    return -0.2 * dH * rng.random(mesh.nAc), 30.0 * rng.standard_normal(mesh.nAc) * (Hi[Aci[:, 0]] > 0.0)


def _sia_inputs(case, seed):
    base, mesh = _mesh(case["mesh"])
    _, sia = workloads.prepare_inputs(mesh, *_ice(base, "dome", seed))
    T = _temperature(base, seed + 5)
    Aci = np.asarray(mesh.Aci) - 1
    Tc = 0.5 * (T[Aci[:, 0]] + T[Aci[:, 1]])
    sia["A_flow_Ac"] = np.asfortranarray(1.14e-5 * np.exp(-6.0e4 / (8.314 * Tc)))
    return dict(fields=sia, params=_params())


def _sia_on_device(s):
    """Device arrays for the call that takes them: (nAc, nZ) column-major is (nZ, nAc) here."""
    f, mesh, dev = s["fields"], s["mesh"], torch.device("cuda", 0)
    names = ("mask_sheet_Ac", "Hi_Ac", "dHs_dx_Ac", "dHs_dy_Ac", "dHs_dp_Ac", "dHs_do_Ac")
    ins = [torch.as_tensor(f[k], device=dev) for k in names]
    ins.append(torch.as_tensor(np.ascontiguousarray(f["A_flow_Ac"].T), device=dev))
    new = dict(dtype=torch.float64, device=dev)
    out = dict(D_SIA_3D_Ac=torch.zeros((NZ, mesh.nAc), **new))
    out.update({k: torch.zeros(mesh.nAc, **new) for k in ("D_SIA_Ac", "Ux_SIA_Ac", "Uy_SIA_Ac", "Up_SIA_Ac", "Uo_SIA_Ac")})
    out.update({k: torch.zeros(s["base"].nV, **new) for k in ("U_SIA", "V_SIA", "D_SIA")})
    s["ins"], s["out"] = ins, out
    s["c_in"] = nat.SiaIn(*(t.data_ptr() for t in ins))
    s["c_out"] = nat.SiaOut(*(t.data_ptr() for t in out.values()))
    s["zeta"] = np.ascontiguousarray(ZETA)
    p = s["params"]
    s["c_par"] = nat.Params(p["SSA_RN_tol"], p["SSA_max_outer_loops"], p["SSA_max_residual_UV"], p["SSA_SOR_omega"],
                            p["SSA_max_inner_loops"], p["m_enh_ssa"], p["m_enh_sia"], p["sliding_law"], p["beta_sq"],
                            0, 0, NZ, s["zeta"].ctypes.data, p["precision"], 0, 0, 0)
    s["kind"] = "sia-device"


def _prepare_ensemble(case, seed):
    sizes = workloads.ensemble_sizes(case["members"], lo=case["lo"], hi=case["hi"])
    members = []
    for i, n in enumerate(sizes):
        base, mesh = _mesh(int(n), 1000 + i)
        rng = np.random.default_rng(seed * 1000 + i)
        ssa, _ = workloads.prepare_inputs(mesh, *workloads.dome_geometry(base, H0=rng.uniform(2000.0, 4000.0)))
        ssa["beta_sq_AaAc"] = _friction(mesh, seed * 1000 + i)
        members.append(ssa)
    batch = api.Batch([_mesh(int(n), 1000 + i)[1] for i, n in enumerate(sizes)])
    return dict(kind="ensemble", batch=batch, members=members, params=_params("linear", case["precision"]))


# ---------------------------------------------------------------------------------------- one pass
def run(s):
    kind = s["kind"]
    if kind == "ssa":
        rc, out, _ = s["dm"].solve_ssa(s["fields"], s["params"], warm=s["warm"], check=False)
        return rc, out
    if kind == "ensemble":
        for i, f in enumerate(s["members"]):
            s["batch"].upload(i, f, s["params"])
        rc, _, _ = s["batch"].run(s["params"])
        got = [s["batch"].download(i) for i in range(len(s["members"]))]
        # all members' results, field by field
        return rc, {k: np.concatenate([g[k] for g in got]) for k in SSA_OUT}
    if kind == "vjp":
        rc, out, _ = s["dm"].ssa_vjp(s["dJ"], s["params"], geom_mesh=s["mesh"], check=False)
        return rc, out
    if kind == "sia":
        return s["dm"].solve_sia(s["fields"], s["params"])
    if kind == "sia-device":
        rc = nat.load().ufe_sia_solve_noalloc(s["dm"].handle, ct.byref(s["c_par"]), ct.byref(s["c_in"]),
                                              ct.byref(s["c_out"]))
        if rc:
            raise nat.UfeError(rc, "ufe_sia_solve_noalloc")
        return s["out"]
    dm, p = s["dm"], s["params"]
    if kind == "thermo":
        props = dm.ice_physical_properties(p, s["Ti"])
        u, v, w = dm.solve_sia_3d(None, s["dHb_dt"], p)
        dx, dy, missing = dm.upwind_derivatives_3d(p)
        return dict(props, U_3D=u, V_3D=v, W_3D=w, dTi_dx=dx, dTi_dy=dy, missing=missing)
    if kind == "geometry":
        g = dm.geometry_update(s["Hi"], s["Hb"], s["SL"])
        masks = dm.geometry_masks()
        H, prev, rate, flux = dm.thickness_update(s["Hi"], s["A"], s["Cw"], s["SMB"], s["BMB"], 1.0,
                                                  Up_SIA_Ac=s["Up_SIA"], Up_SSA_Ac=s["Up_SSA"])
        return dict(geometry=g, masks=masks, Hi=H, Hi_prev=prev, dHi_dt=rate, dVi_in=flux)
    # one time step, in the order of the model's loop
    dm.geometry_update(s["Hi"], s["Hb"], s["SL"])
    props = dm.ice_physical_properties(p, s["Ti"])
    sia = dm.solve_sia_geometry(None, p)
    dm.ssa_upload_geometry(s["Hi"], s["Hb"], s["SL"], None, None, p, beta=s["beta"], warm=s["warm"])
    rc, _ = dm.ssa_run(p, check=False)
    ssa = dm.ssa_download()
    u, v, w = dm.solve_sia_3d(None, s["dHb_dt"], p)
    dx, dy, missing = dm.upwind_derivatives_3d(p)
    heat = dm.frictional_heating(s["mask_sheet"])
    H, prev, rate, flux = dm.thickness_update(s["Hi"], s["A"], s["Cw"], s["SMB"], s["BMB"], 1.0)
    return dict(status=rc, props=props, sia=sia, ssa=ssa, U_3D=u, V_3D=v, W_3D=w, dTi_dx=dx, dTi_dy=dy,
                missing=missing, heating=heat, Hi=H, Hi_prev=prev, dHi_dt=rate, dVi_in=flux)


# ---------------------------------------------------------------------------------------- work
_VERTICES = {"tiny": 248, "1k": 740, "4k": 3992, "16k": 14340, "50k": 42672, "100k": 95000, "200k": 203020}


def _ssa_work(nV, geometry, law):
    """Bytes: the operator (five coefficients and a column per entry, six or seven entries a row),
    seven input fields, the warm start and the eleven results, once each. Flops: the iteration's
    measured number of sweeps on these meshes, two fused multiply-adds an entry and about twenty
    operations a row."""
    rows = 4.0 * nV
    sweeps = min(13500.0, 0.055 * rows + 100.0) if geometry == "dome" else min(1e5, 3.0 * rows + 4000.0)
    return dict(bytes=rows * (7 * 44 + 8 * (7 + 4 + 11)), flops=sweeps * rows * (6 * 4 + 20))


def work(case):
    if case["kind"] == "ensemble":
        w = [_ssa_work(float(n), "dome", "linear")
             for n in workloads.ensemble_sizes(case["members"], lo=case["lo"], hi=case["hi"])]
        return {k: sum(q[k] for q in w) for k in ("bytes", "flops")}
    nV = float(_VERTICES.get(case["mesh"], case["mesh"]))
    nAc = 3.0 * nV
    ssa = _ssa_work(nV, case.get("geometry", "dome"), case.get("law", "linear"))
    if case["kind"] == "ssa":
        return ssa
    if case["kind"] == "vjp":
        # the adjoint operator twice as wide, a few hundred transposed sweeps, the Krylov basis once
        rows = nV + nAc
        return dict(bytes=rows * (7 * 76 + 8 * 30), flops=400.0 * rows * (6 * 8 + 30))
    sia = dict(bytes=8.0 * (nAc * (2 * NZ + 10) + nV * 3), flops=nAc * NZ * 12.0)
    if case["kind"] == "sia":
        return sia
    thermo = dict(bytes=8.0 * NZ * (nV * (1 + 4 + 3 + 2) + nAc * 2) + 12.0 * 17 * nV, flops=NZ * (nV * 260.0 + nAc * 45.0))
    geom = dict(bytes=8.0 * (nV * 12 + nAc * 40) + 4.0 * (nV * 15 + nAc * 16) + 8.0 * nV * 50, flops=nV * 80.0 + nAc * 130.0)
    if case["kind"] == "thermo":
        return thermo
    if case["kind"] == "geometry":
        return geom
    return {k: thermo[k] + geom[k] + sia[k] + ssa[k] for k in ("bytes", "flops")}


# ---------------------------------------------------------------------------------------- exact
# What a pass returns, in 64 bits with numpy alone. Solves of more than a few thousand rows and the
# adjoint (a sparse direct solve of its Jacobian) would take longer than is worth it here: None.
def exact(case, seed):
    kind = case["kind"]
    if kind == "ssa":
        base, mesh = _mesh(case["mesh"])
        if base.nV > 1100 or case["warm"] or case["gl"]:
            return None
        return None, _exact_ssa(mesh, _ssa_inputs(case, seed, None)[0], _params(case["law"], case["precision"]))
    if kind == "sia":
        return _exact_sia(case, _sia_inputs(case, seed)["fields"])
    if kind in ("thermo", "geometry"):
        return _exact_fields(case, seed)
    return None


def _floating(Hi, Hb, SL):
    return Hi < (SL - Hb) * RHO_W / RHO_I


def _exact_ssa(mesh, f, p):
    """Picard iteration around the five-colour SOR, row by row of a colour at once."""
    base = mesh.base
    nV, nA, ncm = base.nV, mesh.nVAaAc, mesh.CAaAc.shape[1]
    cat = lambda k: np.concatenate([f[k], f[k + "_Ac"]])  # noqa: E731
    Hi, Hb, SL, A = cat("Hi"), cat("Hb"), cat("SL"), cat("A_flow_mean")
    tx, ty = RHO_I * GRAV * cat("dHs_dx_shelf"), RHO_I * GRAV * cat("dHs_dy_shelf")
    n = np.asarray(mesh.nCAaAc, dtype=np.int64)
    C = np.asarray(mesh.CAaAc, dtype=np.int64) - 1
    used = np.arange(ncm)[None, :] < n[:, None]
    J = np.where(used, C, 0)
    rows = np.arange(nA)

    def split(N):
        N = np.asarray(N)
        return N[rows, n], np.where(used, N[:, :ncm], 0.0)

    (hx, Nx), (hy, Ny), (hxx, Nxx), (hxy, Nxy), (hyy, Nyy) = (
        split(getattr(mesh, k + "_AaAc")) for k in ("Nx", "Ny", "Nxx", "Nxy", "Nyy"))
    cu, cv, s3 = 4 * Nxx + Nyy, 4 * Nyy + Nxx, 3 * (hxy + Nxy.sum(axis=1))
    edge = np.concatenate([np.asarray(base.edge_index), np.asarray(mesh.edge_index_Ac)]) > 0
    colours = [np.flatnonzero((np.asarray(mesh.colour) == k + 1) & ~edge) for k in range(5)]
    lists = [(r, J[r], cu[r], cv[r], s3[r]) for r in colours]
    er = np.flatnonzero(edge & (rows >= 4))
    ew = (used[er] & ~edge[J[er]]).astype(float)
    ew /= ew.sum(axis=1, keepdims=True)
    kr = np.arange(4)
    kw = used[kr] / n[kr][:, None]
    lam = np.clip(1.0 - (Hb - SL) / 1000.0, 0.0, 1.0)
    mH = np.maximum(0.1, Hi)
    phi = np.clip(5.0 + 15.0 * (1.0 + Hb / 1000.0), 5.0, 20.0)
    tau = np.tan(np.pi / 180.0 * phi) * (RHO_I * GRAV * mH - 0.96 * RHO_I * GRAV * mH * lam)
    ground = ~_floating(Hi, Hb, SL)
    U, V, N = np.zeros(nA), np.zeros(nA), np.zeros(nA)
    eta = np.zeros(nA)
    S = np.zeros(nA)
    for _ in range(p["SSA_max_outer_loops"]):
        ux, uy = hx * U + (Nx * U[J]).sum(1), hy * U + (Ny * U[J]).sum(1)
        vx, vy = hx * V + (Nx * V[J]).sum(1), hy * V + (Ny * V[J]).sum(1)
        e2 = ux ** 2 + vy ** 2 + ux * vy + 0.25 * (uy + vx) ** 2 + 1e-12
        eta = (0.5 * p["m_enh_ssa"] * A) ** (-1 / 3) * e2 ** (-1 / 3)
        Nold, N = N, eta * mH
        if math.sqrt(((N - Nold) ** 2).sum() / (N ** 2).sum()) < p["SSA_RN_tol"]:
            break
        if p["sliding_law"] == nat.UFE_SLIDING_LINEAR:
            S = np.asarray(f["beta_sq_AaAc"], dtype=float)
        else:
            S = tau * (1e-6 + U ** 2 + V ** 2) ** (0.5 * (0.3 - 1.0)) / 100.0 ** 0.3
        fr = np.where(ground, S / (mH * eta), 0.0)
        eu, ev, bx, by = 4 * hxx + hyy - fr, 4 * hyy + hxx - fr, tx / eta, ty / eta
        data = [(r, j, a, b, s, eu[r], ev[r], bx[r], by[r]) for r, j, a, b, s in lists]
        for _ in range(p["SSA_max_inner_loops"]):
            worst = 0.0
            for r, j, a, b, s, e, g, x, y in data:
                u, v = U[r], V[r]
                ru = (np.einsum("ij,ij->i", a, U[j]) + s * v + e * u - x) / e
                rv = (np.einsum("ij,ij->i", b, V[j]) + s * u + g * v - y) / g
                U[r], V[r] = u - p["SSA_SOR_omega"] * ru, v - p["SSA_SOR_omega"] * rv
                worst = max(worst, np.abs(ru).max(), np.abs(rv).max())
            U[er], V[er] = (ew * U[J[er]]).sum(1), (ew * V[J[er]]).sum(1)
            U[kr], V[kr] = (kw * U[J[kr]]).sum(1), (kw * V[J[kr]]).sum(1)
            if worst < p["SSA_max_residual_UV"]:
                break
    Aci, xy = np.asarray(mesh.Aci) - 1, np.asarray(base.V)
    d = xy[Aci[:, 1]] - xy[Aci[:, 0]]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    x, y = U[nV:], V[nV:]
    return dict(U_SSA=U[:nV], V_SSA=V[:nV], Ux_SSA_Ac=x, Uy_SSA_Ac=y, N_AaAc=N, Up_SSA_Ac=x * d[:, 0] + y * d[:, 1],
                Uo_SSA_Ac=y * d[:, 0] - x * d[:, 1], eta_AaAc=eta, S_AaAc=S, tau_c_AaAc=tau, phi_fric_AaAc=phi)


def _integral_up(f):
    """-integral from the base (k = nZ) to each level of f over zeta."""
    d = np.zeros_like(f)
    for k in range(NZ - 2, -1, -1):
        d[:, k] = d[:, k + 1] - 0.5 * (f[:, k + 1] + f[:, k]) * (ZETA[k + 1] - ZETA[k])
    return d


def _average(f):
    return (0.5 * (f[:, 1:] + f[:, :-1]) * np.diff(ZETA)).sum(axis=1)


def _exact_sia(case, f):
    base, mesh = _mesh(case["mesh"])
    H, sx, sy, sp, so = (f[k] for k in ("Hi_Ac", "dHs_dx_Ac", "dHs_dy_Ac", "dHs_dp_Ac", "dHs_do_Ac"))
    sheet = f["mask_sheet_Ac"] == 1
    D0 = (RHO_I * GRAV * H) ** 3 * (sp ** 2 + so ** 2)
    D3 = np.maximum(D0[:, None] * 2.0 * H[:, None] * _integral_up(f["A_flow_Ac"] * ZETA ** 3), -1e5) * sheet[:, None]
    avg = _average(D3)
    D, Ux, Uy = H * avg, avg * sx, avg * sy
    iAci, nC = np.asarray(mesh.iAci, dtype=np.int64) - 1, np.asarray(base.nC)
    used = np.arange(iAci.shape[1])[None, :] < nC[:, None]
    mean = lambda d: np.where(used, d[np.maximum(iAci, 0)], 0.0).sum(axis=1) / nC  # noqa: E731
    return dict(D_SIA_3D_Ac=D3 if case["where"] == "host" else np.ascontiguousarray(D3.T), D_SIA_Ac=D, Ux_SIA_Ac=Ux,
                Uy_SIA_Ac=Uy, Up_SIA_Ac=avg * sp, Uo_SIA_Ac=avg * so, U_SIA=mean(Ux), V_SIA=mean(Uy), D_SIA=mean(D))


def _arrhenius(T):
    return np.where(T < 263.15, 1.14e-5 * np.exp(-6.0e4 / (8.314 * T)), 5.47e10 * np.exp(-13.9e4 / (8.314 * T)))


def _exact_fields(case, seed):
    base, mesh = _mesh(case["mesh"])
    nV = base.nV
    Hi, Hb, SL = _ice(base, "marine", seed)
    Aci = np.asarray(mesh.Aci, dtype=np.int64) - 1
    vi, vj = Aci[:, 0], Aci[:, 1]
    nC, C = np.asarray(base.nC, dtype=np.int64), np.asarray(base.C, dtype=np.int64) - 1
    used = np.arange(C.shape[1])[None, :] < nC[:, None]
    J = np.where(used, C, 0)
    rows = np.arange(nV)

    def grad(d):
        out = []
        for N in (np.asarray(mesh.Nx), np.asarray(mesh.Ny)):
            x = N[rows, nC].reshape((nV,) + (1,) * (d.ndim - 1)) * d
            for c in range(C.shape[1]):
                w = np.where(used[:, c], N[:, c], 0.0)
                x = x + w.reshape((nV,) + (1,) * (d.ndim - 1)) * d[J[:, c]]
            out.append(x)
        return out

    surface = lambda H, B, S: H + np.maximum(S - RHO_I / RHO_W * H, B)  # noqa: E731
    to_ac = lambda d: 0.5 * (d[vi] + d[vj])  # noqa: E731
    Hs = surface(Hi, Hb, SL)
    ocean = _floating(Hi, Hb, SL)
    sheet, shelf = (Hi > 0) & ~ocean, (Hi > 0) & ocean
    ix, iy = grad(Hi)
    sx, sy = grad(Hs)
    rng = np.random.default_rng(seed + 3)
    x, y = np.asarray(base.V).T
    dHb_dt = 1e-3 * rng.standard_normal(nV)
    SMB = 0.3 - 0.8 * np.hypot(x, y) / 750e3 + 0.05 * rng.standard_normal(nV)
    BMB = -0.2 * rng.random(nV)
    f = 1.0 - RHO_I / RHO_W
    if case["kind"] == "geometry":
        g = dict(Hs=Hs, dHi_dx=ix, dHi_dy=iy, dHs_dx=sx, dHs_dy=sy, dHs_dx_shelf=np.where(ocean, f * ix, sx),
                 dHs_dy_shelf=np.where(ocean, f * iy, sy), Hi_Ac=to_ac(Hi), Hb_Ac=to_ac(Hb), SL_Ac=to_ac(SL))
        g["Hs_Ac"] = surface(g["Hi_Ac"], g["Hb_Ac"], g["SL_Ac"])
        for name, d in (("Hi", Hi), ("Hb", Hb), ("Hs", Hs), ("SL", SL)):
            for suffix, N in (("dx", mesh.Nx_Ac), ("dy", mesh.Ny_Ac), ("do", mesh.No_Ac)):
                g["d%s_%s_Ac" % (name, suffix)] = (np.asarray(N) * d[Aci]).sum(axis=1)
            g["d%s_dp_Ac" % name] = np.asarray(mesh.Np_Ac) * (d[vj] - d[vi])
        ocean_Ac = _floating(g["Hi_Ac"], g["Hb_Ac"], g["SL_Ac"])
        for q in ("dx", "dy"):
            g["dHs_%s_shelf_Ac" % q] = np.where(ocean_Ac, f * g["dHi_%s_Ac" % q], g["dHs_%s_Ac" % q])
        return dict(geometry=g, masks=None, **_exact_thickness(case, mesh, Hi, SMB, BMB, *_some_fluxes(mesh, Hi, seed)))
    T = _temperature(base, seed + 5)
    Tc = to_ac(T)
    A, Ac = _arrhenius(T), _arrhenius(Tc)
    Hc, Bc, Sc = to_ac(Hi), to_ac(Hb), to_ac(SL)
    sheet_Ac = (Hc > 0) & ~_floating(Hc, Bc, Sc)
    out = dict(A_flow=A, A_flow_mean=np.where(sheet, _average(A), _arrhenius((T[:, 0] + 271.15) / 2)), A_flow_Ac=Ac,
               A_flow_mean_Ac=np.where(sheet_Ac, _average(Ac), _arrhenius((Tc[:, 0] + 271.15) / 2)),
               Ti_pmp=273.16 - 8.7e-4 * Hi[:, None] * ZETA, Cpi=2115.3 + 7.79293 * (T - 273.16),
               Ki=3.101e8 * np.exp(-0.0057 * T), Ti_Ac=Tc)
    # 3-D velocities without a sliding velocity (no solve on the handle)
    moves = ~shelf & (Hi != 0.0)
    D = (RHO_I * GRAV * Hi) ** 3 * (sx ** 2 + sy ** 2)
    D = np.maximum(D[:, None] * 2.0 * Hi[:, None] * _integral_up(A * ZETA ** 3), -1e5) * moves[:, None]
    edge = np.asarray(base.edge_index) > 0
    er, kr = np.flatnonzero(edge)[np.flatnonzero(edge) >= 4], np.arange(4)

    def neumann(d):
        w = used[er] & ~edge[J[er]]
        d[er] = np.where(w[:, :, None], d[J[er]], 0.0).sum(axis=1) / w.sum(axis=1)[:, None]
        d[kr] = np.where(used[kr][:, :, None], d[J[kr]], 0.0).sum(axis=1) / nC[kr][:, None]
        return d

    U, V = neumann(D * sx[:, None]), neumann(D * sy[:, None])
    Ux, Vy = grad(U)[0], grad(V)[1]
    W = np.zeros_like(U)
    W[:, -1] = dHb_dt + U[:, -1] * (sx - ix) + V[:, -1] * (sy - iy)
    mH = np.maximum(0.1, Hi)
    for k in range(NZ - 2, -1, -1):
        dz, zm = ZETA[k + 1] - ZETA[k], 0.5 * (ZETA[k + 1] + ZETA[k])
        W[:, k] = W[:, k + 1] - Hi * dz * (
            0.5 * (Ux[:, k] + Ux[:, k + 1]) + 0.5 * (Vy[:, k] + Vy[:, k + 1])
            + (sx - zm * ix) / mH * (U[:, k + 1] - U[:, k]) / dz + (sy - zm * iy) / mH * (V[:, k + 1] - V[:, k]) / dz)
    W[edge | ~sheet] = 0.0
    out.update(U_3D=U, V_3D=V, W_3D=neumann(W))
    # upwind derivatives of Ti: the first triangle around the vertex that holds the upwind point
    R, NxT, NyT = _triangles(case["mesh"])
    speed = np.hypot(U, V)
    still = (np.abs(U) < 1e-10) & (np.abs(V) < 1e-10)
    s = np.where(still, 1.0, 4.0 * speed)
    px, py = x[:, None] - U * R[:, None] / s, y[:, None] - V * R[:, None] / s
    tri = np.asarray(base.Tri, dtype=np.int64) - 1
    iTri, niTri = np.asarray(base.iTri, dtype=np.int64) - 1, np.asarray(base.niTri)
    dx, dy = grad(T)
    dx, dy = np.where(still, dx, 0.0), np.where(still, dy, 0.0)
    todo = ~still
    for c in range(iTri.shape[1]):
        t = np.where(c < niTri, iTri[:, c], 0)
        a, b, q = tri[t].T
        ax, ay, bx, by, cx, cy = (v[:, None] for v in (x[a], y[a], x[b], y[b], x[q], y[q]))
        inside = ((bx - ax) * (py - ay) - (by - ay) * (px - ax) > -1e-8) & \
            ((cx - ax) * (py - ay) - (cy - ay) * (px - ax) < 1e-8) & \
            ((cx - bx) * (py - by) - (cy - by) * (px - bx) > -1e-8)
        hit = todo & inside & (c < niTri)[:, None]
        for d, N in ((dx, NxT), (dy, NyT)):
            d[:] = np.where(hit, N[t, 0][:, None] * T[a] + N[t, 1][:, None] * T[b] + N[t, 2][:, None] * T[q], d)
        todo &= ~hit
    out.update(dTi_dx=dx, dTi_dy=dy, missing=None)   # the count is no computed number
    return out


def _exact_thickness(case, mesh, Hi, SMB, BMB, up_sia, up_ssa):
    base = mesh.base
    A, Cw = _cells(case["mesh"])
    nV = base.nV
    Aci = np.asarray(mesh.Aci, dtype=np.int64) - 1
    vi, vj = Aci[:, 0], Aci[:, 1]
    C, nC = np.asarray(base.C, dtype=np.int64) - 1, np.asarray(base.nC)
    used = np.arange(C.shape[1])[None, :] < nC[:, None]
    ci = (used[vi] & (C[vi] == vj[:, None])).argmax(axis=1)
    cj = (used[vj] & (C[vj] == vi[:, None])).argmax(axis=1)
    u = up_sia + up_ssa
    d = np.where(u > 0.0, Hi[vi], Hi[vj]) * u * Cw[vi, ci]
    flux = np.zeros(Cw.shape)
    flux[vi, ci], flux[vj, cj] = -d, d
    smb, have = (SMB + BMB) * A, A * Hi
    out = np.where(flux < 0.0, -flux, 0.0).sum(axis=1)
    dry = -smb >= have
    smb = np.where(dry, -have, smb)
    fac = np.where(dry, 0.0, 1.0)
    over = out > have + smb
    fac[over] = ((have + smb) / np.where(out > 0, out, 1.0))[over]
    flux = np.where(flux < 0.0, flux * fac[:, None], np.where(used, flux * fac[np.maximum(C, 0)], 0.0))
    rate = (flux.sum(axis=1) + smb) / A
    H = np.where(np.asarray(base.edge_index) > 0, 0.0, Hi + rate)
    return dict(Hi=H, Hi_prev=Hi, dHi_dt=rate, dVi_in=flux)
