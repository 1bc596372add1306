"""The entry-by-entry factor of small matrices in shared memory
(lu_entries.cuh): refactor and solve apart and together give the same bits
and meet the backward-error bound of the other LU paths (1e-13; FP32 factors
after three refinements), on one row, rows too long for a thread, levels
wider and narrower than the block, and matrices whose pivots are bad."""
import numpy as np
import pytest
import scipy.sparse as sp

from helpers import circuit_jacobian
from test_gpu_lu import _backward_error
from xyce_gb300 import abi, engine, netlists

pytestmark = pytest.mark.gpu


def _arrow(n, seed):
    rng = np.random.default_rng(seed)
    A = sp.lil_matrix((n, n))
    A.setdiag(rng.uniform(4.0, 5.0, n))
    A[n - 1, :n - 1] = rng.uniform(-1, 1, n - 1)
    A[:n - 1, n - 1] = rng.uniform(-1, 1, n - 1).reshape(-1, 1)
    A[n - 1, n - 1] = float(n)
    return A.tocsr()


def _blocks(k, m, seed):
    rng = np.random.default_rng(seed)
    return sp.block_diag([rng.uniform(-1, 1, (m, m)) + 2 * m * np.eye(m) for _ in range(k)]).tocsr()


CASES = {
    "one": lambda: sp.csr_matrix(np.array([[2.0]])),
    "three": lambda: sp.csr_matrix(np.array([[2.0, 1.0, 0.0], [1.0, 3.0, 0.5], [0.0, 0.5, 1.0]])),
    "arrow_14": lambda: _arrow(14, 1),     # a row one longer than a thread sums
    "arrow_900": lambda: _arrow(900, 2),
    "blocks_60x8": lambda: _blocks(60, 8, 3),
    "inverter_chain_300": lambda: circuit_jacobian(netlists.inverter_chain(300), seed=5),
    "ring_oscillator_501": lambda: circuit_jacobian(netlists.ring_oscillator(501, seed=4), seed=5),
}


@pytest.mark.parametrize("precision,n_refine", [(abi.LU_FP64, 0), (abi.LU_FP32, 3)])
@pytest.mark.parametrize("case", sorted(CASES))
def test_refactor_and_solve(case, precision, n_refine, gpu_ctx, oracle_lib):
    import torch
    A = CASES[case]()
    A.sort_indices()
    n = A.shape[0]
    b = torch.from_numpy(np.random.default_rng(6).standard_normal(n)).cuda()
    vals = torch.from_numpy(A.data.copy()).cuda()
    xs = []
    for fused in (True, False, True):
        lu = engine.LU(gpu_ctx, A.indptr, A.indices, A.data, precision)
        x = torch.zeros_like(b)
        if fused:
            lu.refactor_solve(vals.data_ptr(), b.data_ptr(), x.data_ptr(), n_refine)
        else:
            lu.refactor(vals.data_ptr())
            lu.solve(b.data_ptr(), x.data_ptr(), n_refine)
        assert lu.status() == (0, -1)
        xs.append(x.cpu().numpy())
        lu.refactor(torch.zeros_like(vals).data_ptr())
        assert lu.status() == (1, 0)
        lu.close()
    assert np.array_equal(xs[0], xs[1]) and np.array_equal(xs[0], xs[2])
    assert _backward_error(A, xs[0], b.cpu().numpy()) <= 1e-13
