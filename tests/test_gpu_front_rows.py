"""Rows solved outside the multifrontal tree that a cluster of blocks sums
(front_rows in lu_front.cu): lengths at the edges of a block's and a cluster's
share, before the tree's right-hand sides and after them.  The blocks of a row
write their sums into the first one's shared memory, so the result must repeat
bit for bit however unevenly they start, and solve the system: backward error
<= 1e-13, the bound of the other LU paths."""
import numpy as np
import pytest
import scipy.sparse as sp

from test_gpu_lu import _backward_error
from xyce_gb300 import abi, engine

pytestmark = pytest.mark.gpu

CORE = 8400
# one entry over the limit (seven blocks of eight have nothing to add), one
# block's threads, all eight blocks' threads, and one to either side of each
LENGTHS = (65, 66, 127, 1023, 1024, 1025, 8191, 8192, 8193)


def _matrix(seed):
    """A banded core; rows of their own columns that name many core columns
    (solved after the tree); single-entry rows whose unknowns a few core rows
    name by the dozen or the thousand (solved before it)."""
    rng = np.random.default_rng(seed)
    after, before = len(LENGTHS) + 40, 8193
    n = CORE + after + before
    place = np.random.default_rng(1)
    rows, cols, vals = [], [], []

    def put(r, c, v):
        r, c, v = np.broadcast_arrays(r, c, v)
        rows.append(r.ravel())
        cols.append(c.ravel())
        vals.append(v.ravel())

    i = np.arange(CORE)
    put(i, i, rng.uniform(4.0, 5.0, CORE))
    put(i[1:], i[:-1], -rng.uniform(0.5, 1.0, CORE - 1))
    put(i[:-1], i[1:], -rng.uniform(0.5, 1.0, CORE - 1))
    for k in range(after):
        m = LENGTHS[k] if k < len(LENGTHS) else 65
        put(CORE + k, np.sort(place.choice(CORE, m, replace=False)), rng.uniform(-1.0, 1.0, m))
        put(CORE + k, CORE + k, rng.uniform(2.0, 3.0))
    b0 = CORE + after
    put(b0 + np.arange(before), b0 + np.arange(before), rng.uniform(1.0, 2.0, before))
    for k, m in enumerate(LENGTHS):
        put(900 * k + 7, b0 + np.sort(place.choice(before, m, replace=False)), rng.uniform(-1.0, 1.0, m))
    A = sp.coo_matrix((np.concatenate(vals), (np.concatenate(rows), np.concatenate(cols))), (n, n)).tocsr()
    A.sort_indices()
    return A


@pytest.mark.parametrize("precision,n_refine", [(abi.LU_FP64, 0), (abi.LU_FP32, 3)])
def test_long_rows_outside_the_tree(precision, n_refine, gpu_ctx):
    import torch
    A0, A = _matrix(2), _matrix(3)
    lu = engine.LU(gpu_ctx, A0.indptr, A0.indices, A0.data, precision)
    vals = torch.from_numpy(A.data.copy()).cuda()
    b = torch.from_numpy(np.random.default_rng(4).standard_normal(A.shape[0])).cuda()
    x = torch.zeros_like(b)
    torch.cuda.synchronize()
    first = None
    for _ in range(50):
        lu.refactor_solve(vals.data_ptr(), b.data_ptr(), x.data_ptr(), n_refine)
        assert lu.status() == (0, -1)
        got = x.cpu().numpy()
        if first is None:
            first = got
            assert _backward_error(A, got, b.cpu().numpy()) <= 1e-13
        assert np.array_equal(got, first)
    lu.close()
