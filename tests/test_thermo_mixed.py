"""Column steps and the mesh's resident heat steps on one context keep to their own vertical grids."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("nz", [7, 40])
def test_column_steps_leave_the_resident_state_alone(pkg, gpu_lib, nz):
    mesh, fields, p = pkg.geometry.small_thermo(seed=3)
    zeta, cols = pkg.geometry.random_columns(2 * mesh.nV, nz, seed=nz)
    pc = pkg.abi.default_thermo_params(dt=1.0)
    with pkg.ColumnSolver() as c:
        want_cols = c.thermo_step(pc, zeta, cols)[0]
    with pkg.VelocitySolver(mesh) as s:
        s.heat_upload(fields)
        s.heat_step_resident(p, 4)
        want = s.heat_download()
    assert mesh.nz != nz
    with pkg.VelocitySolver(mesh) as s:
        s.heat_upload(fields)
        s.heat_step_resident(p, 2)
        assert np.array_equal(pkg.ColumnSolver.thermo_step(s, pc, zeta, cols)[0], want_cols)
        s.heat_step_resident(p, 2)
        assert np.array_equal(s.heat_download(), want)
