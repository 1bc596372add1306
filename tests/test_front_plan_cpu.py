"""The multifrontal plan (lu_front.h, no GPU).  A test program
(front_plan_check.cpp, compiled here with the host analysis) checks that every
index the kernels follow lies in its buffer, that each unknown and each entry
of A is placed once, that the maps between fronts are inverse to each other,
and that the elimination and solves over the plan, done as the kernels do
them, give a backward error of rounding size."""
import os
import shutil
import subprocess

import numpy as np
import pytest
import scipy.sparse as sp

from helpers import circuit_jacobian
from xyce_gb300 import netlists

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "xyce_gb300", "csrc")
INCLUDE = os.path.join(HERE, "..", "include")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path_factory.mktemp("front") / "front_plan_check")
    r = subprocess.run([gxx, "-std=c++17", "-O2", "-I" + CSRC, "-I" + INCLUDE,
                        os.path.join(HERE, "front_plan_check.cpp"), os.path.join(CSRC, "lu_front_plan.cpp"),
                        os.path.join(CSRC, "lu_symbolic.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return exe


def _floating_source():
    """A resistor chain with a voltage source between two of its nodes: the
    source's branch row has no diagonal entry."""
    n = 400
    A = sp.lil_matrix((n + 1, n + 1))
    for i in range(n):
        A[i, i] = 3.0
        if i:
            A[i, i - 1] = A[i - 1, i] = -1.0
    A[n, 100], A[n, 250], A[100, n], A[250, n] = 1.0, -1.0, 1.0, -1.0
    return A.tocsr()


CASES = {
    "inverter_chain_300": lambda: circuit_jacobian(netlists.inverter_chain(300), seed=5),
    "power_grid_40x30": lambda: circuit_jacobian(netlists.power_grid(40, 30, 400, seed=1), seed=5),
    "random_logic_6000": lambda: circuit_jacobian(netlists.random_logic(6000, seed=2), seed=5),
    "random_mos_3000": lambda: circuit_jacobian(netlists.random_mos_netlist(3000, 1000, seed=2), seed=5),
    "floating_source": _floating_source,
    "two_parts": lambda: sp.block_diag([sp.diags([[-1.0] * 199, [3.0] * 200, [-1.0] * 199], [-1, 0, 1]),
                                        sp.diags([[-1.0] * 69, [3.0] * 70, [-1.0] * 69], [-1, 0, 1])]).tocsr(),
}


def _write(A, path):
    with open(path, "wb") as f:
        np.array([A.shape[0], A.nnz], np.int64).tofile(f)
        A.indptr.astype(np.int32).tofile(f)
        A.indices.astype(np.int32).tofile(f)
        A.data.astype(np.float64).tofile(f)


@pytest.mark.parametrize("case", sorted(CASES))
def test_plan_indices_and_elimination(checker, tmp_path, case):
    A = CASES[case]()
    A.sort_indices()
    path = str(tmp_path / "a.bin")
    _write(A, path)
    r = subprocess.run([checker, path], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    out = r.stdout.split()
    if case == "random_mos_3000":  # an expander: its fronts may outgrow the kernels
        assert out[0] == "ok" or r.stdout.startswith("no plan"), r.stdout
    else:
        assert out[0] == "ok", r.stdout
    if out[0] == "ok":
        assert float(out[1]) <= 1e-13, r.stdout


def test_unsorted_rows_are_left_to_the_other_path(checker, tmp_path):
    A = CASES["two_parts"]()
    A.sort_indices()
    A.indices[A.indptr[5]:A.indptr[6]] = A.indices[A.indptr[5]:A.indptr[6]][::-1].copy()
    path = str(tmp_path / "a.bin")
    _write(A, path)
    r = subprocess.run([checker, path], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("no plan"), r.stdout + r.stderr
