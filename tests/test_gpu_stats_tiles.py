"""Horizontal statistics at the edges of the kernel's partition: fewer columns
than chunks, chunks that are no multiple of the warps' unrolled columns, and
level counts around a multiple of 32; sums 1e-13 relative against numpy
(another order of the additions), maximum and minimum exact."""
import numpy as np
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(5, 3, 26), (64, 70, 27), (101, 96, 58), (128, 130, 25)], ids=str)
def test_statistics_partition_edges(n):
    import torch
    from pycles_b200.grid import Grid
    from pycles_b200.simulation import namelist_for
    from pycles_b200.statistics import HorizontalStatistics
    Gr = Grid(namelist_for("dry_cbl", *n, 50.0, 50.0, 50.0))
    rng = np.random.default_rng(5)
    a, b = 300.0 + rng.standard_normal(Gr.shape), rng.standard_normal(Gr.shape)
    mask = (rng.random(Gr.shape) < 0.4).astype(np.float64)
    g = Gr.dims.gw
    col = lambda x: x[g:-g, g:-g].reshape(-1, x.shape[2])
    st = HorizontalStatistics(Gr)
    A, B, M = (torch.as_tensor(x.ravel(), device="cuda") for x in (a, b, mask))
    want = {
        "mean": (st.HorizontalMean(Gr, A), col(a).mean(0)),
        "squares": (st.HorizontalMeanofSquares(Gr, A, A), (col(a) ** 2).mean(0)),
        "cross": (st.HorizontalMeanofSquares(Gr, A, B), (col(a) * col(b)).mean(0)),
        "conditional": (st.HorizontalMeanConditional(Gr, A, M),
                        (col(a) * col(mask)).sum(0) / np.maximum(col(mask).sum(0), 1.0)),
    }
    for k, (x, y) in want.items():
        # the cross term cancels: its error is that of terms of size |a b|
        scale = 1e-13 if k != "cross" else 1e-13 * np.linalg.norm(np.abs(col(a) * col(b)).mean(0)) / np.linalg.norm(y)
        assert rel_l2(x.cpu().numpy(), y) < scale, k
    assert np.array_equal(st.HorizontalMaximum(Gr, B).cpu().numpy(), col(b).max(0))
    assert np.array_equal(st.HorizontalMinimum(Gr, B).cpu().numpy(), col(b).min(0))
