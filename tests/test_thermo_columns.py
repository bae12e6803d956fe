"""The full-step column pass at the ends of its range: one to 33 columns (blocks of 32), 3 to 256 layers, uniform heat
capacity and conductivity -- bit for bit the oracle's values, which its shared reciprocals and comparisons on bit
patterns are to leave alone."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [10.0, 0.7, 3.0])
@pytest.mark.parametrize("nV,nz", [(1, 3), (31, 4), (32, 12), (33, 30), (200, 33), (70, 255), (33, 256)])
def test_full_step_columns_are_the_oracles(pkg, oracle_mod, gpu_lib, nV, nz, dt):
    p = pkg.abi.default_thermo_params(dt=dt)
    p.choice_ice_heat_capacity, p.choice_ice_thermal_conductivity = pkg.abi.CP["uniform"], pkg.abi.KI["uniform"]
    zeta, cols = pkg.geometry.random_columns(4 * nV + 20, nz, seed=nz)
    flags = np.asarray(oracle_mod.thermo_step(p, zeta, cols)[3])
    pick = np.flatnonzero(flags == 0)[:nV]
    assert len(pick) == nV
    cols = {k: np.asfortranarray(v[pick]) for k, v in cols.items()}
    ref, n_ref, status, _ = oracle_mod.thermo_step(p, zeta, cols)
    with pkg.ColumnSolver() as s:
        got, n = s.thermo_step(p, zeta, cols)
    assert status == pkg.abi.UFE_OK and n == n_ref == 0
    assert np.array_equal(got, ref)
