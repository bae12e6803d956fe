"""The kernels around the linear solve of a Picard iteration, where their split can go wrong: layer counts below, at and
above the six warps that share a vertex's layers, both forms of Glen's power, rows at the domain border and prescribed
rows, and triangle and vertex counts that leave the last 32 incomplete -- against the oracle."""
import numpy as np
import pytest

from helpers import rel_l2

# The linear solves end at 1e-12 |D^-1 b|; with friction a step of them moves the velocities by less than 1e-9 of
# their size (the condition number of these small meshes is below 1e3), and the rest are roundings.
TOL = 1e-8


def _params(pkg, params, **kw):
    p = pkg.abi.SolverParams.from_buffer_copy(params)
    p.stress_balance_PETSc_rtol, p.stress_balance_PETSc_abstol, p.visc_it_nit = 1e-12, 0.0, 1
    for k, v in kw.items():
        setattr(p, k, v)
    return p


@pytest.mark.gpu
@pytest.mark.parametrize("n_glen", [3.0, 2.5, 1.0])
@pytest.mark.parametrize("nz", [3, 5, 6, 7, 13, 64])
def test_diva_iterations_match_oracle(pkg, oracle_mod, gpu_lib, nz, n_glen):
    mesh, ice, params = pkg.geometry.small_channel(nz=nz)
    p = _params(pkg, params, Glens_flow_law_exponent=n_glen)
    orc = oracle_mod.Oracle(mesh)
    a, b = pkg.new_diva_state(mesh.nTri, mesh.nz), pkg.new_diva_state(mesh.nTri, mesh.nz)
    with pkg.VelocitySolver(mesh, operators=orc.operators()) as s:
        na, _, sa = s.solve_DIVA(ice, a, p)
    nb, _, sb = orc.solve_DIVA(ice, b, p)
    assert na == nb and sa["status"] == sb["status"]
    for k in ("u_vav_b", "v_vav_b", "u_base_b", "tau_bx_b", "eta_3D_b"):
        assert rel_l2(a[k], b[k]) < TOL, k


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("cross", [0, 1])
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_ssa_iterations_with_prescribed_rows_match_oracle(pkg, oracle_mod, gpu_lib, seed, cross, precision):
    mesh, ice, params = pkg.geometry.small_dome(seed=seed)
    p = _params(pkg, params, do_include_SSADIVA_crossterms=cross, precision=precision, BC_u_west=1, BC_v_north=1)
    mask = np.zeros(mesh.nTri, np.int32)
    mask[::37] = 1
    bc = dict(mask_b=mask, u_b=np.linspace(-5, 5, mesh.nTri), v_b=np.linspace(3, -3, mesh.nTri))
    orc = oracle_mod.Oracle(mesh)
    a, b = pkg.new_ssa_state(mesh.nTri), pkg.new_ssa_state(mesh.nTri)
    with pkg.VelocitySolver(mesh, operators=orc.operators()) as s:
        na, _, sa = s.solve_SSA(ice, a, p, BC=bc)
    q = _params(pkg, p, precision=0)
    nb, _, sb = orc.solve_SSA(ice, b, q, BC=bc)
    assert na == nb and sa["status"] == sb["status"]
    assert rel_l2(np.r_[a["u_b"], a["v_b"]], np.r_[b["u_b"], b["v_b"]]) < TOL
