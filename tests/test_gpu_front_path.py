"""Which matrices the multifrontal path takes: those that test_gpu_front.py and
test_gpu_front_rows.py solve with it, and neither a matrix whose pivots grow in
the tree's order nor one with the path switched off."""
import numpy as np
import pytest
import scipy.sparse as sp

import test_gpu_front
import test_gpu_front_rows
from helpers import circuit_jacobian
from test_gpu_lu import _backward_error, _solve
from xyce_gb300 import abi, engine, netlists

pytestmark = pytest.mark.gpu

CIRCUITS = {**test_gpu_front.CASES, **test_gpu_front.SMALLER}


def _path(ctx, A, precision=abi.LU_FP64):
    lu = engine.LU(ctx, A.indptr, A.indices, A.data, precision)
    path = lu.path
    lu.close()
    return path


@pytest.mark.parametrize("precision", [abi.LU_FP64, abi.LU_FP32])
@pytest.mark.parametrize("case", sorted(CIRCUITS))
def test_circuits_take_fronts(case, precision, gpu_ctx, oracle_lib, monkeypatch):
    A = circuit_jacobian(CIRCUITS[case](), seed=4, pdt=1e12)
    # (1,704 rows of FP32 entries fit one SM's shared memory)
    level = case == "inverter_chain_1700" and precision == abi.LU_FP32
    assert _path(gpu_ctx, A, precision) == (abi.LU_PATH_LEVEL if level else abi.LU_PATH_FRONT)
    monkeypatch.setenv("XG_LU_NO_FRONT", "1")
    assert _path(gpu_ctx, A, precision) != abi.LU_PATH_FRONT


def test_long_rows_take_fronts(gpu_ctx):
    assert _path(gpu_ctx, test_gpu_front_rows._matrix(2)) == abi.LU_PATH_FRONT


def test_growing_pivots_do_not(gpu_ctx):
    """A mesh whose every other node has a tiny diagonal: its multipliers pass
    their bound in the tree's order, where the time model alone would take the
    tree (5.6 ms against 0.8); with ordinary ones it takes it."""
    m = 100
    line = sp.diags([-np.ones(m - 1), np.zeros(m), -np.ones(m - 1)], [-1, 0, 1])
    mesh = sp.kron(sp.eye(m), line) + sp.kron(line, sp.eye(m))
    node = np.arange(m * m)
    for tiny in (1e-9, 6.0):
        A = (mesh + sp.diags(np.where((node // m + node % m) % 2 == 0, tiny, 6.0))).tocsr()
        A.sort_indices()
        assert (_path(gpu_ctx, A) == abi.LU_PATH_FRONT) == (tiny > 1.0)
        b = np.random.default_rng(3).standard_normal(m * m)
        x, status, _ = _solve(gpu_ctx, A, A, b, abi.LU_FP64, 0)
        assert status == 0 and _backward_error(A, x, b) <= 1e-13


def test_small_matrices_go_level_by_level(gpu_ctx, oracle_lib):
    for nl in (netlists.inverter_chain(1000), netlists.ring_oscillator(101, seed=2)):
        assert _path(gpu_ctx, circuit_jacobian(nl, seed=5)) == abi.LU_PATH_LEVEL
