"""The residual of a batch's domains (lbm_batch_residuals) against the same sums
in NumPy, for domains of a few tiles and of more tiles than the summing block
has threads, and a retired one that keeps its last value."""
import numpy as np
import pytest

from thesis_gb300 import lattice
from thesis_gb300 import native as N
from thesis_gb300.batch import Batch, cavity_args

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(8, 8), (33, 40)], [(256, 32), (1040, 600), (24, 24)]])
def test_batch_residuals_match_numpy(sizes):
    lats = [lattice.cavity2d(n, m) for n, m in sizes]
    args = [cavity_args(n, 100.0, storage=N.STORE_F32) for n, _ in sizes]
    fields = lambda b: [np.stack(b.macro(d)[1:]).astype(np.float64) for d in range(len(sizes))]
    with Batch(lats, args) as b:
        b.init()
        b.step(20)
        b.residuals()
        old = fields(b)
        b.step(20)
        res, _ = b.residuals()
        new = fields(b)
        active = [1] * len(sizes)
        active[0] = 0
        b.set_active(active)
        b.step(10)
        later, _ = b.residuals()
    for lat, r, f0, f1 in zip(lats, res, old, new):
        fluid = lat.node_type == 1
        ref = np.sqrt(((f1 - f0)[:, fluid] ** 2).sum()) / np.sqrt((f1[:, fluid] ** 2).sum())
        # sums of at most 1.9e6 non-negative terms in FP64
        assert abs(r - ref) <= 1e-9 * ref
    assert later[0] == res[0] and np.all(later[1:] != res[1:])
