"""The scalar CSR solve where its persistent kernel is not launched: where the launch is refused (in ufe_solve_csr and in
the semi-implicit thickness step), above the rows up to which it is the faster form, and while a velocity solve of
another thread runs, the kernels that need no co-residency take the solve, with the same iterates to the bit."""
import threading

import numpy as np
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

BESIDE = SOLVES + """
import threading
during, stats = [], {}
mesh, ice, p = pkg.geometry.small_dome()
p.visc_it_nit, p.visc_it_norm_dUV_tol = 2000, 0.0
with pkg.VelocitySolver(mesh) as v, pkg.ColumnSolver() as s:
    v.ice_upload(ice)
    want = csr(s, 1000)
    p.visc_it_nit = 2
    v.solve_resident(p, diva=False)
    p.visc_it_nit = 2000
    started, done = threading.Event(), threading.Event()
    def work():
        started.set()
        stats.update(v.solve_resident(p, diva=False))
        done.set()
    t = threading.Thread(target=work)
    t.start()
    started.wait()
    while not done.is_set():       # calls that began and ended while the solve ran
        n = shim.shim_coop()
        got = csr(s, 1000)
        if not done.is_set():
            during.append((shim.shim_coop() - n, same(got, want)))
    t.join()
    assert len(during) > 8 and all(ok for _, ok in during), (during, stats)
    assert not any(n for n, _ in during[3:]), during       # the first ones may have come before the solve
    n = shim.shim_coop()
    assert same(csr(s, 1000), want) and shim.shim_coop() - n == 1
"""


@pytest.mark.gpu
def test_beside_a_velocity_solve(gpu_lib, tmp_path):
    cuda_shim.run(tmp_path, BESIDE, UFE_NO_GRAPH="1")   # a graph with loops may hold back other streams


@pytest.mark.gpu
def test_two_threads_of_solves(pkg, gpu_lib):
    """Thickness steps in two host threads beside velocity solves in a third: each answer is that of a thread alone."""
    def thickness(seed, out):
        mesh, f, p = pkg.geometry.thickness_case(seed=seed)
        p.choice_ice_integration_method = pkg.abi.DHI["semi-implicit"]
        with pkg.VelocitySolver(mesh) as s:
            s.voronoi_upload()
            for i in range(20):
                out.append(s.calc_dHi_dt(p, f, 1.0 + 0.1 * i)["Hi_tplusdt"])

    def velocity(seed, out):
        mesh, ice, p = pkg.geometry.small_dome(seed=seed)
        p.visc_it_nit = 5
        with pkg.VelocitySolver(mesh) as s:
            s.ice_upload(ice)
            for i in range(10):
                s.solve_resident(p, diva=False)
                out.append(np.concatenate(s.velocity_download()))

    jobs = [(thickness, 0), (thickness, 1), (velocity, 0)]
    alone, both = [[] for _ in jobs], [[] for _ in jobs]
    for (f, seed), out in zip(jobs, alone):
        f(seed, out)
    threads = [threading.Thread(target=f, args=(seed, out)) for (f, seed), out in zip(jobs, both)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(alone, both):
        assert len(a) == len(b) > 0 and all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.gpu
def test_refused_cooperative_launch(gpu_lib, tmp_path):
    cuda_shim.run(tmp_path, REFUSED)
