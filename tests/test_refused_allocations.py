"""A call whose n-th device allocation is refused ends with an error and leaves nothing half-built: the same call on the
same context, with memory again, gives what it gives on a fresh one.  Every n up to the call's last allocation."""
import pytest

import cuda_shim

SETUP = """
def every_refusal(name, make, call, at_least):
    with make() as s:
        want = call(s)
    failed = 0
    for n in range(400):
        with make() as s:
            shim.shim_fail_from(n)
            try:
                call(s)
                done = True
            except (pkg.UfeError, RuntimeError):
                done = False
                failed += 1
            shim.shim_fail_from(1 << 30)
            got = call(s)
            assert all(np.array_equal(np.asarray(a), np.asarray(b)) for a, b in zip(got, want)), (name, n)
        if done:
            break
    assert done and failed >= at_least, (name, failed)
"""

VELOCITY = SETUP + """
mesh, ice, p = pkg.geometry.small_dome()
p.visc_it_nit = 2
for precision in (pkg.abi.PREC_FP64, pkg.abi.PREC_FP32_PAIR):
    p.precision = precision
    def solve(s):
        s.ice_upload(ice)
        s.solve_resident(p, diva=True)
        return s.velocity_download()
    every_refusal("velocity", lambda: pkg.VelocitySolver(mesh), solve, 60)
mesh, ice, p = pkg.geometry.icestream_case(res=60e3)[:3]
p.visc_it_nit = 1
def stream(s):
    s.ice_upload(ice)
    s.solve_resident(p, diva=False)
    return s.velocity_download()
every_refusal("icestream", lambda: pkg.VelocitySolver(mesh), stream, 60)
"""

THICKNESS = SETUP + """
mesh, f, p = pkg.geometry.thickness_case(res=60e3)
p.choice_ice_integration_method = pkg.abi.DHI["semi-implicit"]
geo = pkg.mesh.voronoi_geometry(mesh)
def step(s):
    s.voronoi_upload(*geo)
    r = s.calc_dHi_dt(p, f, 1.0)
    return r["Hi_tplusdt"], r["divQ"]
every_refusal("thickness", lambda: pkg.VelocitySolver(mesh), step, 30)
with pkg.VelocitySolver(mesh) as s:        # refused areas, then a step without a new upload
    s.voronoi_upload(*geo)
    try:
        s.voronoi_upload(-geo[0], geo[1])
        assert False
    except pkg.UfeError:
        pass
    try:
        s.calc_dHi_dt(p, f, 1.0)
        assert False
    except pkg.UfeError as e:
        assert e.code == pkg.abi.UFE_ERR_INVALID
"""

COLUMNS = SETUP + """
pc = pkg.abi.default_thermo_params(dt=1.0)
small, large = (pkg.geometry.random_columns(n, nz, seed=nz) for n, nz in ((100, 5), (400, 12)))
def grown():           # a context that has stepped fewer columns before
    s = pkg.ColumnSolver()
    s.thermo_step(pc, *small)
    return s
every_refusal("columns", grown, lambda s: [s.thermo_step(pc, *large)[0], s.thermo_step(pc, *small)[0]], 4)
every_refusal("columns", pkg.ColumnSolver, lambda s: [s.thermo_step(pc, *large)[0]], 5)
mesh, fields, p = pkg.geometry.small_thermo(seed=3)
def heat(s):
    s.heat_upload(fields)
    s.heat_step_resident(p, 2)
    return [s.heat_download()]
every_refusal("heat", lambda: pkg.VelocitySolver(mesh), heat, 15)
"""

NETWORK = SETUP + """
def graph(n):
    i = np.arange(n)
    nbr = np.stack([(i - 1) % n, (i + 1) % n, np.full(n, -1)], axis=1).astype(np.int32)
    rng = np.random.default_rng(n)
    return (nbr, rng.standard_normal((n, 16)).astype(np.float32), rng.standard_normal((n, 3)).astype(np.float32),
            np.full(n, 1 / n, np.float32))
small, large = graph(100), graph(600)
class Net:
    def __enter__(self):
        self.s = pkg.ColumnSolver()
        self.net = pkg.LearnedStart(self.s, seed=0)
        self.net.loss_grad(*small)
        return self.net
    def __exit__(self, *a):
        self.net.close()
        self.s.close()
every_refusal("network", Net, lambda n: [*n.loss_grad(*large), *n.loss_grad(*small), n.forward(*large[:2])], 10)
"""


@pytest.mark.gpu
@pytest.mark.parametrize("script", [VELOCITY, THICKNESS, COLUMNS, NETWORK],
                         ids=["velocity", "thickness", "columns", "network"])
def test_refused_allocations_leave_nothing_half_built(gpu_lib, tmp_path, script):
    cuda_shim.run(tmp_path, script)
