"""The scalar CSR solve where its persistent kernel is not launched: where the launch is refused (in ufe_solve_csr and in
the semi-implicit thickness step) and above the rows up to which it is the faster form, the kernels that need no
co-residency take the solve, with the same iterates to the bit."""
import pytest

import cuda_shim

SOLVES = """
def csr(s, m):
    rng = np.random.default_rng(m)
    ptr = np.arange(0, 3 * m + 1, 3)
    col = np.clip(np.arange(m)[:, None] + [-1, 0, 1], 0, m - 1)
    val = np.stack([rng.uniform(-1, 0, m), 4 + rng.random(m), rng.uniform(-1, 0, m)], axis=1)
    A = pkg.CSR(m, m, ptr, col.ravel(), val.ravel(), index_base=0)
    return pkg.VelocitySolver.solve_matrix_equation_CSR_PETSc(s, A, rng.standard_normal(m), np.zeros(m), 1e-10, 0.0)

def same(a, b):
    return a[1:] == b[1:] and np.array_equal(a[0], b[0])
"""

REFUSED = SOLVES + """
mesh, f, p = pkg.geometry.thickness_case()
p.choice_ice_integration_method = pkg.abi.DHI["semi-implicit"]
with pkg.VelocitySolver(mesh) as s:
    s.voronoi_upload()
    want = [csr(s, 1000), csr(s, 60_000)]
    h = s.calc_dHi_dt(p, f, 3.0)
    assert shim.shim_refused() == 0
    shim.shim_refuse_coop(1)
    got = [csr(s, 1000), csr(s, 60_000)]
    g = s.calc_dHi_dt(p, f, 3.0)
    assert shim.shim_refused() == 3
assert all(same(a, b) for a, b in zip(want, got))
assert h["stats"]["n_Axb_its"] == g["stats"]["n_Axb_its"] > 0
for k in ("Hi_tplusdt", "dHi_dt", "divQ", "AMB"):
    assert np.array_equal(h[k], g[k])
"""

ROWS = SOLVES + """
with pkg.ColumnSolver() as s:
    for m, coop in ((1 << 21, 1), ((1 << 21) + 1, 0)):
        n = shim.shim_coop()
        got = csr(s, m)
        assert shim.shim_coop() - n == coop
        shim.shim_refuse_coop(1)
        assert same(csr(s, m), got) and got[2] == 0
        shim.shim_refuse_coop(0)
"""


@pytest.mark.gpu
def test_rows_up_to_which_the_solve_is_persistent(gpu_lib, tmp_path):
    cuda_shim.run(tmp_path, ROWS)


@pytest.mark.gpu
def test_refused_cooperative_launch(gpu_lib, tmp_path):
    cuda_shim.run(tmp_path, REFUSED)
