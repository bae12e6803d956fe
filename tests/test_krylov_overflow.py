"""A linear velocity solve whose sums overflow ends with an error, in the persistent kernel as in the three-kernel form."""
import numpy as np
import pytest

from helpers import load_small_dome


def overflowing_inputs(pkg, oracle_mod, mesh, p):
    """Inputs of the linearised solve whose first iteration has (t,t) beyond the FP64 range and every earlier sum well
    inside it.  A system with strong first-derivative terms has |t| far above |s| = O(|r|); the solve is linear in the
    driving stress, so its sums are formed here at an ordinary scale and the stress is scaled up."""
    nT = mesh.nTri
    rng = np.random.default_rng(1)
    args = [np.full(nT, 1e11), rng.normal(0, 1e8, nT), rng.normal(0, 1e8, nT), np.zeros(nT),
            rng.normal(0, 1e5, nT), rng.normal(0, 1e5, nT)]
    A, b = oracle_mod.Oracle(mesh).assemble_linearised(p, *args)
    M = A.to_scipy().tocsr()
    d = M.diagonal()
    d = np.where(d != 0.0, 1.0 / np.where(d != 0.0, d, 1.0), 1.0)
    r = d * b
    v = d * (M @ r)
    alpha = (r @ r) / (v @ r)
    s = r - alpha * v
    t = d * (M @ s)
    others = max(abs(x) for x in (r @ r, v @ r, s @ s, s @ t, s @ r, t @ r))
    scale = 1e155 / np.linalg.norm(t)   # (t,t) = 1e310
    assert others * scale * scale < 1e308
    args[4] = args[4] * scale
    args[5] = args[5] * scale
    return args


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["PREC_FP64", "PREC_FP32_PAIR"])
def test_overflowed_sums_are_an_error(pkg, oracle_mod, gpu_lib, precision):
    """The pair's range is left at once, so its solve is the persistent FP64 kernel's; PREC_FP64 of this entry point
    takes three kernels an iteration."""
    mesh, _, _, ops, _ = load_small_dome(pkg)
    p = pkg.abi.default_params(stress_balance_PETSc_rtol=1e-12, stress_balance_PETSc_abstol=0.0)
    args = overflowing_inputs(pkg, oracle_mod, mesh, p)
    p.precision = getattr(pkg.abi, precision)
    with pkg.VelocitySolver(mesh, operators=ops) as s, pytest.raises(pkg.UfeError) as e:
        s.solve_SSA_DIVA_linearised(p, np.zeros(mesh.nTri), np.zeros(mesh.nTri), *args)
    assert e.value.code in (pkg.abi.UFE_ERR_NAN, pkg.abi.UFE_ERR_DIVERGED)
