"""The persistent BiCGStab kernels at the sizes where the launch rule changes: one row per thread with 512, 768 and
1024 threads per block (k_bicgstab_resident; a block's rows grow with the mesh, one block per SM), and several rows
per thread beyond (k_bicgstab_halo), in FP64 and in double-word arithmetic, against the three-kernel form."""
import math

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("nV", [320, 30_000, 45_000, 70_000, 85_000])
def test_persistent_forms_solve_the_same_system(pkg, gpu_lib, monkeypatch, nV):
    """One Picard iteration of the SSA dome from rest, each linear solve to |D^-1 r| <= 1e-12 |D^-1 b|.  Two such
    solutions of M x = D^-1 b differ by at most 2e-12 cond(M) |x|; friction keeps cond(M) below 5e3 on these meshes
    (the solves take tens of iterations), so by 1e-8."""
    mesh, ice, p = pkg.geometry.dome_case(res_scale=math.sqrt(8492.0 / nV))
    p.visc_it_nit = 1
    p.stress_balance_PETSc_rtol, p.stress_balance_PETSc_abstol = 1e-12, 0.0

    def solve(precision):
        q = pkg.abi.SolverParams.from_buffer_copy(p)
        q.precision = precision
        with pkg.VelocitySolver(mesh) as s:
            s.ice_upload(ice)
            st = s.solve_resident(q, diva=False)
            return np.concatenate(s.velocity_download()), st

    got = {prec: solve(prec) for prec in (pkg.abi.PREC_FP64, pkg.abi.PREC_FP32_PAIR)}
    monkeypatch.setenv("UFE_NO_HALO", "1")
    ref, st = solve(pkg.abi.PREC_FP64)
    assert np.linalg.norm(ref) > 0 and st["n_Axb_its"] < 500
    for prec, (x, s) in got.items():
        assert s["status"] in (pkg.abi.UFE_OK, pkg.abi.UFE_WARN_PICARD_MAXIT)
        assert (s["n_pair_its"] > 0) == (prec == pkg.abi.PREC_FP32_PAIR)
        assert np.linalg.norm(x - ref) <= 1e-8 * np.linalg.norm(ref)
