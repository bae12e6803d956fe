"""A column step holds the fields and lists that its kernels read, and nothing else."""
import pytest

import cuda_shim

STEP = """
nV, nz = 20_000, 30
zeta, cols = pkg.geometry.random_columns(nV, nz, seed=1)
with pkg.ColumnSolver() as s:
    base = shim.shim_held()
    s.thermo_step(pkg.abi.default_thermo_params(dt=1.0), zeta, cols)
    fields = 8 * (12 * nV * nz + 6 * nV) + 4 * nV
    lists = 2 * 4 * nV
    assert shim.shim_held() - base <= fields + lists + (1 << 16), shim.shim_held() - base - fields - lists
"""


@pytest.mark.gpu
def test_a_column_step_holds_its_fields(gpu_lib, tmp_path):
    cuda_shim.run(tmp_path, STEP)
