"""Quotients that share a divisor's reciprocal keep the divisions' bits where the numerator is zero, its sign among
them: connections of zero width, whose flux is -0 where it would enter the cell."""
import numpy as np
import pytest


@pytest.mark.gpu
def test_zero_widths_bitexact(pkg, oracle_mod, gpu_lib):
    mesh, f, p = pkg.geometry.thickness_case()
    A, Cw = pkg.mesh.voronoi_geometry(mesh)
    Cw = np.array(Cw, order="F")
    Cw[::3, ::2] = 0.0
    f = dict(f)
    for k in ("Hi_tplusdt", "divQ", "AMB", "dHi_dt"):
        f[k] = np.zeros(mesh.nV)
    pp = pkg.abi.default_thickness_params(BC_H_west="infinite", BC_H_east="infinite")
    want = oracle_mod.Oracle(mesh).thickness_assemble(A, Cw, pp, {k: np.copy(v) for k, v in f.items()}, 3.0)
    pe = pkg.abi.default_thickness_params(choice_ice_integration_method="explicit")
    q = {k: np.copy(v) for k, v in f.items()}
    oracle_mod.Oracle(mesh).calc_dHi_dt(A, Cw, pe, q, 3.0)
    with pkg.VelocitySolver(mesh) as s:
        s.voronoi_upload(A, Cw)
        got = s.thickness_assemble(pp, f, 3.0)
        g = s.calc_dHi_dt(pe, f, 3.0)
    assert np.signbit(want[2][want[2] == 0.0]).any()
    for a, b in zip(got, want):
        assert a.tobytes() == b.tobytes()
    for k in ("divQ", "Hi_tplusdt", "dHi_dt", "AMB"):
        assert np.array_equal(g[k], q[k])
