"""The network's kernels at the edges of their 128-node tiles and of the resident grid (304 CTAs of one tile each: at
38,913 nodes the first CTA gets a second tile), against the oracle with the same BF16 roundings."""
import numpy as np
import pytest

from test_gnn import _net_case, _rel


@pytest.mark.gpu
@pytest.mark.parametrize("n", [100, 127, 128, 129, 257, 38912, 38913])
def test_network_at_tile_edges(pkg, gpu_lib, n):
    """BF16 operands differ between the two only where an FP32 sum of at most 128 terms (error 1e-5) crosses a rounding
    boundary of BF16 (2^-9): one operand in 200, by 4e-3 of its size -- about 3e-4 of a sum, and at most ten such
    sums in sequence."""
    import gnn_oracle as G
    nbr, x, p, tgt, w = _net_case(G, n=n, seed=n)
    x, tgt, w = x.astype(np.float32), tgt.astype(np.float32), w.astype(np.float32)
    with pkg.ColumnSolver() as s:
        net = pkg.LearnedStart(s)
        net.set_params(p.astype(np.float32))
        pf = net.get_params().astype(np.float64)
        y = net.forward(nbr, x)
        loss, g = net.loss_grad(nbr, x, tgt, w)
        again = net.forward(nbr, x)
    y_ref, _ = G.forward(pf, nbr, x, bf=True)
    loss_ref, g_ref = G.loss_grad(pf, nbr, x.astype(np.float64), tgt, w, bf=True)
    assert np.array_equal(y, again)
    assert _rel(y, y_ref) < 3e-3
    assert abs(loss - loss_ref) <= 3e-3 * loss_ref
    assert _rel(g, g_ref) < 5e-3
