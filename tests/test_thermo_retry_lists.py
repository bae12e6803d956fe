"""Lists of distinct retried columns of every kind -- grounded, floating and at the grounding line, there with either
basal condition -- through the two retry kernels (four warps a column for lists of up to 304 columns of up to 32 layers,
one warp beyond): no list entry touches another."""
import functools

import numpy as np
import pytest

NZ = [3, 5, 8, 30, 32]


def params(pkg, glbc):
    p = pkg.abi.default_thermo_params(dt=10.0)
    p.choice_GL_temperature_BC = pkg.abi.GLBC[glbc]
    return p


@functools.lru_cache(maxsize=None)
def listed_columns(pkg, oracle_mod, nz, glbc, want=90):
    """(zeta, columns that recover at a smaller time step, that end in the Robin profile, that are stable): pools of stiff
    columns through the oracle until `want` distinct ones recover, or for three layers, where none does, six pools."""
    p, got = params(pkg, glbc), {0: [], 1: [], 2: []}
    for seed in range(60):
        n = 20_000
        zeta, cols = pkg.geometry.random_columns(n, nz, seed=100 * nz + seed, stiff_frac=0.6, stiffness=3000.0)
        rng = np.random.default_rng(seed)
        cols["w_3D"] *= np.where(rng.random(n) < 0.5, 1.0, 10.0 ** rng.uniform(-1.0, 2.0, n))[:, None]
        kinds = [pkg.abi.COL_GROUNDED, pkg.abi.COL_FLOATING, pkg.abi.COL_GL_GR]
        cols["mask"] = rng.choice(kinds, n, p=[0.3, 0.2, 0.5]).astype(np.int32)
        flags = np.asarray(oracle_mod.thermo_step(p, zeta, cols)[3])
        for f in got:
            pick = np.flatnonzero(flags == f)[:want if f else 300]
            got[f].append({k: np.asarray(v)[pick] for k, v in cols.items()})
        if sum(len(g["mask"]) for g in got[2]) >= want or (nz == 3 and seed == 5):
            break
    merged = [{k: np.concatenate([g[k] for g in got[f]]) for k in got[f][0]} for f in (2, 1, 0)]
    return zeta, merged[0], merged[1], merged[2]


def join(*parts):
    return {k: np.asfortranarray(np.concatenate([p[k] for p in parts])) for k in parts[0]}


def take(cols, index):
    return {k: v[index] for k, v in cols.items()}


@pytest.mark.parametrize("glbc", ["grounded", "subgrid"])
@pytest.mark.parametrize("nz", NZ)
def test_the_pool_holds_distinct_columns_of_every_kind(pkg, oracle_mod, nz, glbc):
    _, recover, robin, stable = listed_columns(pkg, oracle_mod, nz, glbc)
    cols = recover if nz > 3 else robin
    assert len(stable["mask"]) >= 300 and len(cols["mask"]) >= 60
    assert len(np.unique(cols["w_3D"], axis=0)) == len(cols["mask"])
    for kind in (pkg.abi.COL_GROUNDED, pkg.abi.COL_GL_GR):
        assert (cols["mask"] == kind).sum() >= 5, kind


@pytest.mark.gpu
@pytest.mark.parametrize("glbc", ["grounded", "subgrid"])
@pytest.mark.parametrize("nz", NZ)
def test_a_columns_answer_does_not_depend_on_its_list(pkg, oracle_mod, gpu_lib, nz, glbc):
    """Every listed column gets, to the bit, what it gets alone: in a list of distinct columns in another order, which
    the four-warp kernel takes, and for each of several copies in a list of more than 304, the one-warp kernel's."""
    p = params(pkg, glbc)
    zeta, recover, robin, stable = listed_columns(pkg, oracle_mod, nz, glbc)
    some = join(take(recover, slice(0, 60)), take(robin, slice(0, 12 if nz > 3 else 60)))
    k = len(some["mask"])
    fill = take(stable, np.resize(np.arange(len(stable["mask"])), 8000))

    with pkg.ColumnSolver() as s:
        def step(order, nfill):
            cols = join(take(some, order), take(fill, slice(0, nfill)))
            return np.asarray(s.thermo_step(p, zeta, cols)[0])[:len(order)]

        alone = np.stack([step([j], 200)[0] for j in range(k)])
        order = np.random.default_rng(nz).permutation(k)
        assert np.array_equal(step(order, 7000), alone[order])
        copies = 1 + 304 // k
        many = np.random.default_rng(nz).permutation(np.tile(np.arange(k), copies))
        assert len(many) > 304
        fill = take(stable, np.resize(np.arange(len(stable["mask"])), 100 * len(many) + 100))
        got = step(many, 100 * len(many) + 100)
        first = got[[int(np.flatnonzero(many == j)[0]) for j in range(k)]]
        assert np.array_equal(got, first[many])
