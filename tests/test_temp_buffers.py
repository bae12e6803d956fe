"""Calls that share a context's temporary buffers give, to the bit, what a context of their own gives: sizes that
grow, shrink and miss a block's size class (64 KB, four times), both index bases, and a refused call in between."""
import numpy as np
import pytest

# rows; 8 bytes a row: within one 64 KB block, at its edge, past it, larger, and back down
SIZES = [5, 8192, 8193, 40000, 7, 8192, 300000, 100, 40001]


def _system(m, base):
    rng = np.random.default_rng(m + base)
    col = np.stack([np.clip(np.arange(m) - 1, 0, m - 1), np.arange(m)], axis=1).ravel()
    val = np.stack([rng.uniform(-1.0, 0.0, m), rng.uniform(4.0, 5.0, m)], axis=1).ravel()
    ptr = np.arange(0, 2 * m + 1, 2)
    return ptr + base, col + base, val, rng.standard_normal(m)


def _calls(pkg, s, m, base):
    V = pkg.VelocitySolver
    ptr, col, val, b = _system(m, base)
    A = pkg.CSR(m, m, ptr, col, val, index_base=base)
    y = V.multiply_CSR_matrix_with_vector_1D(s, A, b)
    y3 = V.multiply_CSR_matrix_with_vector_2D(s, A, np.stack([b, 2 * b, -b], axis=1))
    x, its, status = V.solve_matrix_equation_CSR_PETSc(s, A, b, np.zeros(m), 1e-10, 0.0)
    assert np.array_equal(y3[:, 0], y) and np.array_equal(y3[:, 2], -y)
    # each product and the sum are rounded once
    lo = val[0::2] * b[col[0::2] - base] + val[1::2] * b[col[1::2] - base]
    assert np.all(np.abs(y - lo) <= 4 * 2.0 ** -53 * (np.abs(val[0::2]) + 5) * np.abs(b).max())
    return [y, y3, x, np.array([its, status])]


@pytest.mark.gpu
@pytest.mark.parametrize("base", [0, 1])
def test_shared_buffers(pkg, gpu_lib, base):
    with pkg.ColumnSolver() as shared:
        for m in SIZES:
            with pkg.ColumnSolver() as own:
                want = _calls(pkg, own, m, base)
            for _ in range(2):
                got = _calls(pkg, shared, m, base)
                for a, b in zip(want, got):
                    assert np.array_equal(a, b), m
            ptr, col, val, b = _system(m, base)
            for bad in (m + base, base - 1):
                wrong = col.copy()
                wrong[-1] = bad
                with pytest.raises(Exception):
                    pkg.VelocitySolver.multiply_CSR_matrix_with_vector_1D(
                        shared, pkg.CSR(m, m, ptr, wrong, val, index_base=base), b)
