"""Unused buffers that the library keeps between calls are there for its other allocations: a limit on the device memory
that a call can have (a library in front of the CUDA runtime refuses what goes past it) leaves room for the call only
when the kept buffers are given back.  The contexts of a process keep 1 GiB of them together.  A mesh's thickness steps
find their buffers there, and a network that only predicts has no gradient buffers."""
import pytest

import cuda_shim

KEEP = """
def keep(s, mb):        # leaves about mb of unused buffers with the context: a product's operand and result
    import scipy.sparse as sp
    n, cols = 100_000, max(1, int(mb * 1e6 / 2 / 8 / 100_000))
    A = pkg.CSR.from_scipy(sp.identity(n, format="csr"))
    x = np.asfortranarray(np.random.default_rng(0).random((n, cols)))
    y = pkg.VelocitySolver.multiply_CSR_matrix_with_vector_2D(s, A, x)
    assert np.array_equal(x, y)

def step(s):            # 12 fields of 20,000 x 30: 58 MB that the context keeps
    zeta, cols = pkg.geometry.random_columns(20_000, 30, seed=1)
    return s.thermo_step(pkg.abi.default_thermo_params(dt=1.0), zeta, cols)[0]

MB = 1 << 20
"""

OWN_AND_OTHERS = KEEP + """
with pkg.ColumnSolver() as alone:
    want = step(alone)
a, b, c = pkg.ColumnSolver(), pkg.ColumnSolver(), pkg.ColumnSolver()
keep(a, 200)
shim.shim_cap(shim.shim_held() + 20 * MB)
assert np.array_equal(step(a), want)       # its own buffers
shim.shim_cap((1 << 63))
keep(a, 200)
shim.shim_cap(shim.shim_held() + 20 * MB)
assert np.array_equal(step(b), want)       # another context's
shim.shim_cap((1 << 63))
keep(a, 200)
shim.shim_cap(shim.shim_held() + 20 * MB)
keep(c, 150)                               # temporary buffers from another context's
"""

TOGETHER = KEEP + """
some = [pkg.ColumnSolver() for _ in range(5)]
base = shim.shim_held()
for s in some:
    keep(s, 400)
assert shim.shim_held() - base <= 1025 * MB, (shim.shim_held() - base) / MB
n = shim.shim_mallocs()
keep(some[0], 400)                         # kept, not allocated again
assert shim.shim_mallocs() == n
for s in some:
    s.close()
assert shim.shim_held() < base
"""

CSR_SOLVE = KEEP + """
import scipy.sparse as sp
def solve(s, m):        # 112 bytes of work vectors a row beside the system itself
    rng = np.random.default_rng(m)
    A = pkg.CSR.from_scipy(sp.diags([rng.uniform(-1, 0, m - 1), 3 + rng.random(m), rng.uniform(-1, 0, m - 1)],
                                    [-1, 0, 1], format="csr"))
    return pkg.VelocitySolver.solve_matrix_equation_CSR_PETSc(s, A, rng.random(m), np.zeros(m), 1e-10, 0.0)

a = pkg.ColumnSolver()
base = shim.shim_held()
want = solve(a, 1_000_000)
assert want[2] == 0
n = shim.shim_mallocs()
x, its, st = solve(a, 1_000_000)
assert shim.shim_mallocs() == n and its == want[1] and np.array_equal(x, want[0])
small = solve(a, 400_000)   # in the larger call's buffers
with pkg.ColumnSolver() as fresh:
    got = solve(fresh, 400_000)
assert got[1] == small[1] and np.array_equal(got[0], small[0])
shim.shim_cap(base + 80 * MB)
step(a)
assert shim.shim_held() <= base + 80 * MB
"""

FIRST_STEP = KEEP + """
mesh, f, p = pkg.geometry.thickness_case(res=8e3)
for method in ("explicit", "semi-implicit"):
    p.choice_ice_integration_method = pkg.abi.DHI[method]
    with pkg.VelocitySolver(mesh) as s:
        s.voronoi_upload()
        n = shim.shim_mallocs()
        first = s.calc_dHi_dt(p, f, 3.0)["Hi_tplusdt"]
        assert shim.shim_mallocs() == n, method        # all buffers came with the mesh
        try:
            s.calc_dHi_dt(p, dict(f, Hi=None), 3.0)
            assert False, "a missing field was accepted"
        except pkg.UfeError:
            pass
        assert np.array_equal(s.calc_dHi_dt(p, f, 3.0)["Hi_tplusdt"], first)
        assert shim.shim_mallocs() == n, method        # and outlive a refused call
"""

NETWORK = KEEP + """
n = 60_000
i = np.arange(n)
nbr = np.stack([(i - 1) % n, (i + 1) % n, np.full(n, -1)], axis=1).astype(np.int32)
rng = np.random.default_rng(0)
x, y = rng.standard_normal((n, 16)).astype(np.float32), rng.standard_normal((n, 3)).astype(np.float32)
w = np.full(n, 1 / n, np.float32)
with pkg.ColumnSolver() as s:
    base = shim.shim_held()
    net = pkg.LearnedStart(s, seed=0)
    assert shim.shim_held() - base < 10 * MB       # weights and the sums' scalars
    net.forward(nbr[:100] % 100, x[:100])
    small = net.loss_grad(nbr[:100] % 100, x[:100], y[:100], w[:100])
    big = net.loss_grad(nbr, x, y, w)
    again = net.loss_grad(nbr[:100] % 100, x[:100], y[:100], w[:100])
    assert small[0] == again[0] and np.array_equal(small[1], again[1])
    other = pkg.LearnedStart(s, seed=0).loss_grad(nbr, x, y, w)
    assert big[0] == other[0] and np.array_equal(big[1], other[1])
"""


@pytest.mark.gpu
@pytest.mark.parametrize("script", [OWN_AND_OTHERS, TOGETHER, CSR_SOLVE, FIRST_STEP, NETWORK],
                         ids=["own_and_others", "together", "csr_solve", "first_step", "network"])
def test_kept_buffers_are_given_back(gpu_lib, tmp_path, script):
    cuda_shim.run(tmp_path, script)
