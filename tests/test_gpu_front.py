"""The multifrontal LU (lu_front.cu) through the C ABI, on matrices of at
least 8,192 rows and on smaller ones: backward error |b - A x| / (|A| |x| + |b|) <= 1e-13 in FP64
and after three refinements of FP32 factors, as for the other LU paths; the
same solution as the grid path to the error both may have; run-to-run bits;
pivots and singular values reported."""
import numpy as np
import pytest
import scipy.sparse as sp

from helpers import circuit_jacobian
from test_gpu_lu import _backward_error, _solve
from xyce_gb300 import abi, engine, netlists

pytestmark = pytest.mark.gpu

CASES = {
    # just above the line; one wide tree; a long thin one; near-banded logic;
    # a chain whose supply row names every stage
    "power_grid_72x72": lambda: netlists.power_grid(72, 72, 1600, seed=1),
    "power_grid_150x140": lambda: netlists.power_grid(150, 140, 5000, seed=2),
    "power_grid_600x15": lambda: netlists.power_grid(600, 15, 900, seed=3),
    "random_logic_17000": lambda: netlists.random_logic(17000, seed=4),
    "inverter_chain_8300": lambda: netlists.inverter_chain(8300),
}
_JACOBIANS = {}


def _jacobian(case, seed):
    if (case, seed) not in _JACOBIANS:
        _JACOBIANS[case, seed] = circuit_jacobian(CASES[case](), seed=seed, pdt=1e12)
    return _JACOBIANS[case, seed]


@pytest.mark.parametrize("precision,n_refine", [(abi.LU_FP64, 0), (abi.LU_FP32, 3)])
@pytest.mark.parametrize("case", sorted(CASES))
def test_refactor_and_solve(case, precision, n_refine, gpu_ctx, oracle_lib, monkeypatch):
    A0, A = _jacobian(case, 4), _jacobian(case, 5)
    assert A.shape[0] >= 8192
    b = np.random.default_rng(7).standard_normal(A.shape[0])
    x, st, info = _solve(gpu_ctx, A0, A, b, precision, n_refine)
    again = _solve(gpu_ctx, A0, A, b, precision, n_refine)[0]
    assert st == 0 and info.solve_chain == 0
    assert np.array_equal(x, again)
    assert _backward_error(A, x, b) <= 1e-13
    monkeypatch.setenv("XG_LU_NO_FRONT", "1")
    other, st, _ = _solve(gpu_ctx, A0, A, b, precision, n_refine)
    assert st == 0 and _backward_error(A, other, b) <= 1e-13
    # both solve systems within 1e-13 of this one (the bound above), so they
    # differ by at most 2e-13 of the condition number, at most 1e6 here
    assert np.abs(x - other).max() <= 2e-7 * np.abs(other).max()


@pytest.mark.parametrize("precision", [abi.LU_FP64, abi.LU_FP32])
def test_bad_pivots_are_reported_and_do_not_stick(precision, gpu_ctx, oracle_lib):
    import torch
    A = _jacobian("power_grid_72x72", 5)
    lu = engine.LU(gpu_ctx, A.indptr, A.indices, A.data, precision)
    vals = torch.from_numpy(A.data.copy()).cuda()
    b = torch.from_numpy(np.random.default_rng(8).standard_normal(A.shape[0])).cuda()
    x = torch.zeros_like(b)
    for bad in (0.0, float("inf"), float("nan")):
        lu.refactor(torch.full_like(vals, bad).data_ptr())
        status, row = lu.status()
        assert status == 1 and row == 0
        lu.solve(b.data_ptr(), x.data_ptr(), 0)  # ends, whatever it gives
        lu.refactor_solve(vals.data_ptr(), b.data_ptr(), x.data_ptr(), 3 if precision == abi.LU_FP32 else 0)
        assert lu.status() == (0, -1)
        assert _backward_error(A, x.cpu().numpy(), b.cpu().numpy()) <= 1e-13
    lu.close()


def test_waits_that_run_out_report_timeout(gpu_ctx, oracle_lib):
    """With the limit lowered to one poll the solve's waits for children give
    up; the launch ends and says so, and the default limit works again."""
    import torch
    A = _jacobian("power_grid_150x140", 5)
    lu = engine.LU(gpu_ctx, A.indptr, A.indices, A.data, abi.LU_FP64)
    vals = torch.from_numpy(A.data.copy()).cuda()
    b = torch.from_numpy(np.random.default_rng(9).standard_normal(A.shape[0])).cuda()
    x = torch.zeros_like(b)
    lu.set_wait_limit(1)
    lu.refactor_solve(vals.data_ptr(), b.data_ptr(), x.data_ptr())
    assert lu.status()[0] & 2
    lu.set_wait_limit(1 << 20)
    lu.refactor_solve(vals.data_ptr(), b.data_ptr(), x.data_ptr())
    assert lu.status() == (0, -1)
    assert _backward_error(A, x.cpu().numpy(), b.cpu().numpy()) <= 1e-13
    lu.close()


def test_pivots_that_grow_keep_the_grid_path(gpu_ctx):
    """A chain of tiny pivots: eliminated in the tree's order its multipliers
    exceed the pivoting bound, so the analysed (pivoted) order is used."""
    n = 9000
    rng = np.random.default_rng(10)
    d = np.where(np.arange(n) % 2 == 0, 1e-9, 1.0)
    A = sp.diags([rng.uniform(1, 2, n - 1), d, rng.uniform(1, 2, n - 1)], [-1, 0, 1]).tocsr()
    A.sort_indices()
    b = rng.standard_normal(n)
    x, st, _ = _solve(gpu_ctx, A, A, b, abi.LU_FP64, 0)
    assert st == 0 and _backward_error(A, x, b) <= 1e-13


SMALLER = {
    # too large for the level path and without a solve chain
    "power_grid_20x20": lambda: netlists.power_grid(20, 20, 200, seed=1),
    "power_grid_30x28": lambda: netlists.power_grid(30, 28, 400, seed=2),
    "random_logic_2500": lambda: netlists.random_logic(2500, seed=4),
    "inverter_chain_1700": lambda: netlists.inverter_chain(1700),
    "inverter_chain_8000": lambda: netlists.inverter_chain(8000),
}


@pytest.mark.parametrize("precision,n_refine", [(abi.LU_FP64, 0), (abi.LU_FP32, 3)])
@pytest.mark.parametrize("case", sorted(SMALLER))
def test_smaller_matrices(case, precision, n_refine, gpu_ctx, oracle_lib, monkeypatch):
    """Matrices below 8,192 rows: whichever path the rule takes meets the
    same bound as the row-wise one it replaced."""
    nl = SMALLER[case]()
    A0, A = (circuit_jacobian(nl, seed=s, pdt=1e12) for s in (4, 5))
    b = np.random.default_rng(7).standard_normal(A.shape[0])
    x, st, info = _solve(gpu_ctx, A0, A, b, precision, n_refine)
    again = _solve(gpu_ctx, A0, A, b, precision, n_refine)[0]
    assert st == 0 and info.solve_chain == 0 and np.array_equal(x, again)
    assert _backward_error(A, x, b) <= 1e-13
    monkeypatch.setenv("XG_LU_NO_FRONT", "1")
    other, st, _ = _solve(gpu_ctx, A0, A, b, precision, n_refine)
    assert st == 0 and _backward_error(A, other, b) <= 1e-13
    assert np.abs(x - other).max() <= 2e-7 * np.abs(other).max()  # as above
