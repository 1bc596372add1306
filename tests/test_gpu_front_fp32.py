"""FP32 dense fronts and the row-wise factors they stand in for, after two FP64
refinements, on power grids near their operating point: forward error against
the solution that the right-hand side was made from.  The orders differ, so
single errors do by a few times; the tree may be 4 times the row-wise error
further off, above 1e-13, where FP64's own rounding ends (its factors leave up
to 4e-14 here)."""
import numpy as np
import pytest
import scipy.sparse as sp

from xyce_gb300 import abi, engine, netlists

pytestmark = pytest.mark.gpu

GRIDS = {(30, 30): 300, (50, 30): 500, (72, 72): 1728, (90, 90): 2700, (120, 70): 2800}


def _matrix(n, m, sinks, seed):
    """dQ/dx / h + dF/dx / 2 of a step of 1 ps near the grid's start."""
    from oracle.oracle import OracleCircuit
    nl = netlists.power_grid(n, m, sinks, seed=7)
    opt = abi.device_options(fma=1)
    params = {t: engine.setup_params(nl, t, opt) for t in range(abi.NUM_DEV_TYPES) if nl.count(t)}
    oc = OracleCircuit(nl, params, opt)
    guess = netlists.power_grid_nodeset(n, m, sinks)
    x = np.zeros(oc.n_unknowns + 1)
    x[:len(guess)] = guess
    x[:nl.n_nodes] += np.random.default_rng([seed, 3]).normal(0.0, 0.05, nl.n_nodes)
    zero = [np.zeros(k) for k in (oc.n_unknowns + 1, oc.n_state, oc.n_store)]
    out = oc.load(abi.load_flags(transient=1, newton_iter=0, pdt=1e12, time=1e-12), [x, zero[0], zero[0]],
                  [zero[1]] * 3, [zero[2]] * 3)
    A = sp.csr_matrix((1e12 * out["dQdx"] + 0.5 * out["dFdx"], (out["rows"], out["cols"])), (oc.n_unknowns,) * 2)
    oc.close()
    A.sort_indices()
    return A


def _error(ctx, A0, A, b, x, n_refine, path):
    import torch
    lu = engine.LU(ctx, A0.indptr, A0.indices, A0.data, abi.LU_FP32)
    assert (lu.path == abi.LU_PATH_FRONT) == path
    dev = [torch.from_numpy(a.copy()).cuda() for a in (A.data, b, x)]
    torch.cuda.synchronize()
    lu.refactor_solve(dev[0].data_ptr(), dev[1].data_ptr(), dev[2].data_ptr(), n_refine)
    assert lu.status() == (0, -1)
    got = dev[2].cpu().numpy()
    lu.close()
    return np.abs(got - x).max() / np.abs(x).max()


@pytest.mark.parametrize("grid", sorted(GRIDS))
def test_refined_fronts_are_as_close_as_rows(grid, gpu_ctx, oracle_lib, monkeypatch):
    A0 = _matrix(*grid, GRIDS[grid], 0)
    for seed in (1, 2, 3):
        A = _matrix(*grid, GRIDS[grid], seed)
        x = np.random.default_rng([seed, 4]).normal(0.0, 0.05, A.shape[0])
        b = np.add.reduceat(A.data.astype(np.longdouble) * x[A.indices], A.indptr[:-1]).astype(np.float64)
        monkeypatch.delenv("XG_LU_NO_FRONT", raising=False)
        tree = _error(gpu_ctx, A0, A, b, x, 2, True)
        monkeypatch.setenv("XG_LU_NO_FRONT", "1")
        rows = _error(gpu_ctx, A0, A, b, x, 2, False)
        assert tree <= max(4 * rows, 1e-13), (seed, tree, rows)
