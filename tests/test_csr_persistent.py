"""The persistent CSR solve against the kernels it replaces (UFE_NO_PERSIST=1): the same iterates to the bit, at the
sizes where its launch rule changes -- one virtual block, several per block (256 rows each, 152 blocks), several
sets of them, and more rows than virtual blocks x 256."""
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SIZES = [1, 255, 256, 257, 38912, 38913, 155648, 155649, 311296, 311297]

SCRIPT = """
import sys
import numpy as np
sys.path.insert(0, {root!r})
import __graft_entry__
pkg = __graft_entry__.load_package()
out = {{}}
with pkg.ColumnSolver() as s:
    for m in {sizes!r}:
        rng = np.random.default_rng(m)
        width = rng.integers(0, 9, m)                      # rows of 1 to 9 entries, the diagonal among them
        ptr = np.zeros(m + 1, np.int32)
        np.cumsum(width + 1, out=ptr[1:])
        row = np.repeat(np.arange(m), width + 1)
        col = np.clip(row + rng.integers(-700, 701, len(row)), 0, m - 1)
        col[ptr[1:] - 1] = np.arange(m)
        val = rng.uniform(-1.0, 0.0, len(row))
        val[ptr[1:] - 1] = 10.0 + rng.random(m)
        b = rng.standard_normal(m)
        A = pkg.CSR(m, m, ptr, col, val, index_base=0)
        x, its, status = pkg.VelocitySolver.solve_matrix_equation_CSR_PETSc(s, A, b, np.zeros(m), 1e-10, 0.0)
        out["x%d" % m] = x
        out["n%d" % m] = np.array([its, status])
        r = np.bincount(row, weights=val * x[col], minlength=m) - b
        out["r%d" % m] = np.array([np.abs(r).max()])
np.savez(sys.argv[1], **out)
"""


@pytest.mark.gpu
def test_persistent_csr_solve_is_the_kernels(gpu_lib, tmp_path):
    got = []
    for env in ({}, {"UFE_NO_PERSIST": "1"}):
        f = str(tmp_path / ("r%d.npz" % len(got)))
        subprocess.run([sys.executable, "-c", SCRIPT.format(root=ROOT, sizes=SIZES), f], check=True,
                       env=dict(os.environ, **env), timeout=300)
        got.append(np.load(f))
    for m in SIZES:
        assert np.array_equal(got[0]["x%d" % m], got[1]["x%d" % m]), m
        assert np.array_equal(got[0]["n%d" % m], got[1]["n%d" % m]), m
        # |D^-1 r| <= 1e-10 |D^-1 b| in the 2-norm, D within 10 .. 20, |b| < 6 sqrt(m)
        assert got[0]["r%d" % m][0] <= 1e-10 * 2 * 6 * np.sqrt(m) + 1e-12, m
