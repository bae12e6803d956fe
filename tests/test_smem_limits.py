"""A kernel's dynamic shared-memory limit belongs to the function, and every context and instantiated graph launches it
with a size of its own: meshes, layer counts and column solves of different sizes in turn never lower it."""
import threading

import numpy as np
import pytest

import cuda_shim

TURNS = """
def solve(nV, nz, diva, precision):
    mesh, ice, p = pkg.geometry.dome_case(res_scale=(8492.0 / nV) ** 0.5, nz=nz)
    p.visc_it_nit, p.precision = 1, precision
    s = pkg.VelocitySolver(mesh)
    s.ice_upload(ice)
    return lambda: s.solve_resident(p, diva=diva)

def columns(nz):
    zeta, cols = pkg.geometry.random_columns(500, nz, seed=nz)
    p = pkg.abi.default_thermo_params(dt=1.0)
    s = pkg.ColumnSolver()
    return lambda: s.thermo_step(p, zeta, cols)

calls = [solve(2000, 12, True, pkg.abi.PREC_FP64), solve(400, 5, True, pkg.abi.PREC_FP64),
         solve(2000, 12, False, pkg.abi.PREC_FP32_PAIR), solve(400, 5, False, pkg.abi.PREC_FP32_PAIR),
         solve(2000, 12, False, pkg.abi.PREC_FP32_REFINE), solve(400, 5, False, pkg.abi.PREC_FP32_REFINE),
         columns(40), columns(12), columns(200), columns(34)]
for f in calls + calls:
    f()
assert shim.shim_lowered() == 0, shim.shim_lowered()
"""


@pytest.mark.gpu
@pytest.mark.parametrize("env", [{}, {"UFE_NO_GRAPH": "1"}])
def test_limits_are_never_lowered(gpu_lib, tmp_path, env):
    cuda_shim.run(tmp_path, TURNS, **env)


@pytest.mark.gpu
def test_two_threads_two_sizes(pkg, gpu_lib):
    """Two host threads, each with contexts of another size and layer count, whose solves build and launch their graphs
    in turn: the answers are those of a thread alone, to the bit."""
    def work(nV, nz, out, n=6):
        mesh, ice, p = pkg.geometry.dome_case(res_scale=(8492.0 / nV) ** 0.5, nz=nz)
        p.visc_it_nit = 2
        zeta, cols = pkg.geometry.random_columns(300, nz, seed=nz)
        pt = pkg.abi.default_thermo_params(dt=1.0)
        with pkg.VelocitySolver(mesh) as s, pkg.ColumnSolver() as c:
            s.ice_upload(ice)
            for i in range(n):
                p.visc_it_relax = 0.5 + 0.01 * i   # a graph of its own
                for diva in (True, False):
                    s.solve_resident(p, diva=diva)
                    out.append(np.concatenate(s.velocity_download()))
                out.append(np.asarray(c.thermo_step(pt, zeta, cols)[0]))

    sizes = [(1000, 12), (400, 40)]
    alone = [[], []]
    for q, out in zip(sizes, alone):
        work(*q, out)
    both = [[], []]
    threads = [threading.Thread(target=work, args=(*q, out)) for q, out in zip(sizes, both)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(alone, both):
        assert len(a) == len(b) and all(np.array_equal(x, y) for x, y in zip(a, b))
