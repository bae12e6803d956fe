"""The dt-halving retry kernel at the layer counts where its rows-per-lane rule changes (1, 2, 4, 8 rows per lane for up
to 32, 64, 128, 256 layers), against the oracle's sequential recurrences."""
import numpy as np
import pytest


def stiff_columns(pkg, oracle_mod, p, nz, nV=1500, pool=9000):
    """nV columns: from a pool with large vertical velocities those that recover at a smaller time step and a few that
    end in the Robin profile, among ordinary ones.  Returns (zeta, columns)."""
    zeta, cols = pkg.geometry.random_columns(pool, nz, seed=nz, stiff_frac=0.6, stiffness=3000.0)
    rng = np.random.default_rng(nz)
    cols["w_3D"] *= np.where(rng.random(pool) < 0.5, 1.0, 10.0 ** rng.uniform(0.0, 2.0, pool))[:, None]
    flags = np.asarray(oracle_mod.thermo_step(p, zeta, cols)[3])
    pick = np.r_[np.flatnonzero(flags == 2)[:60], np.flatnonzero(flags == 1)[:10]]
    pick = np.sort(np.r_[pick, np.flatnonzero(flags == 0)[:nV - len(pick)]])
    return zeta, {k: np.asfortranarray(v[pick]) for k, v in cols.items()}


@pytest.mark.gpu
@pytest.mark.parametrize("glbc", [0, 1])
@pytest.mark.parametrize("nz", [5, 12, 31, 32, 33, 63, 65, 128, 129, 160])
def test_retried_columns_match_oracle(pkg, oracle_mod, gpu_lib, nz, glbc):
    """1e-8 K: the warp-parallel sums differ from the sequential ones by a few ulp per substep (an ulp of 273 K is
    6e-14 K), over at most 1,022 substeps of a clamped profile."""
    p = pkg.abi.default_thermo_params(dt=10.0)
    p.choice_GL_temperature_BC = glbc
    zeta, cols = stiff_columns(pkg, oracle_mod, p, nz)
    ref, n_ref, status, flags = oracle_mod.thermo_step(p, zeta, cols)
    assert status == pkg.abi.UFE_OK and (np.asarray(flags) > 0).sum() > 0
    with pkg.ColumnSolver() as s:
        got, n = s.thermo_step(p, zeta, cols)
    assert n == n_ref
    assert np.abs(got - ref).max() < 1e-8


@pytest.mark.gpu
@pytest.mark.parametrize("glbc", [0, 1])
@pytest.mark.parametrize("nz", [3, 8, 30, 32])
@pytest.mark.parametrize("n", [1, 304, 305, 700])
def test_short_and_long_lists_match_oracle(pkg, oracle_mod, gpu_lib, n, nz, glbc):
    """Up to 304 listed columns of up to 32 layers are retried by four warps each, longer lists by one: both against
    the oracle, 1e-8 K as above (the inverse's sums are of at most 32 terms of the profile's size per substep)."""
    p = pkg.abi.default_thermo_params(dt=10.0)
    p.choice_GL_temperature_BC = glbc
    zeta, cols = pkg.geometry.random_columns(6000, nz, seed=nz, stiff_frac=0.6, stiffness=3000.0)
    rng = np.random.default_rng(nz)
    cols["w_3D"] *= np.where(rng.random(6000) < 0.5, 1.0, 10.0 ** rng.uniform(0.0, 2.0, 6000))[:, None]
    flags = np.asarray(oracle_mod.thermo_step(p, zeta, cols)[3])
    listed = np.flatnonzero(flags == 2)
    if len(listed) == 0:
        pytest.skip("no column recovers at this layer count")
    pick = np.r_[np.resize(listed, n), np.flatnonzero(flags == 0)[:50]]
    cols = {k: np.asfortranarray(v[pick]) for k, v in cols.items()}
    ref, n_ref, status, flags = oracle_mod.thermo_step(p, zeta, cols)
    assert status == pkg.abi.UFE_OK and (np.asarray(flags) > 0).sum() == n
    with pkg.ColumnSolver() as s:
        got, n_got = s.thermo_step(p, zeta, cols)
    assert n_got == n_ref
    assert np.abs(got - ref).max() < 1e-8
