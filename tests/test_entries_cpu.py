"""The entry schedule of small factors (LuEntries, no GPU).  A test program
(entries_check.cpp, compiled here with the host analysis) checks that every
position lies in range, each entry and row is placed once, nothing is read
before it is final, and that the factor and solution are those of a row-wise
elimination, bit for bit (the same operations in the same order)."""
import os
import shutil
import subprocess

import numpy as np
import pytest
import scipy.sparse as sp

from helpers import circuit_jacobian
from test_front_plan_cpu import _write
from xyce_gb300 import netlists

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "xyce_gb300", "csrc")
INCLUDE = os.path.join(HERE, "..", "include")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path_factory.mktemp("entries") / "entries_check")
    r = subprocess.run([gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I" + CSRC, "-I" + INCLUDE,
                        os.path.join(HERE, "entries_check.cpp"), os.path.join(CSRC, "lu_symbolic.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return exe


CASES = {
    "one": lambda: sp.csr_matrix(np.array([[2.0]])),
    "two": lambda: sp.csr_matrix(np.array([[2.0, 1.0], [1.0, 3.0]])),
    "inverter_chain_24": lambda: circuit_jacobian(netlists.inverter_chain(24), seed=5),
    "inverter_chain_1000": lambda: circuit_jacobian(netlists.inverter_chain(1000), seed=5),
    "ring_oscillator_501": lambda: circuit_jacobian(netlists.ring_oscillator(501, seed=1), seed=5),
    "power_grid_20x20": lambda: circuit_jacobian(netlists.power_grid(20, 20, 60, seed=1), seed=5),
}


@pytest.mark.parametrize("ordering", [0, 1])
@pytest.mark.parametrize("case", sorted(CASES))
def test_schedule(checker, tmp_path, case, ordering):
    A = CASES[case]()
    A.sort_indices()
    path = str(tmp_path / "a.bin")
    _write(A, path)
    r = subprocess.run([checker, path, str(ordering)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
    assert float(r.stdout.split()[2]) == 0.0, r.stdout


def test_too_many_entries_for_sixteen_bits(checker, tmp_path):
    A = sp.random(400, 400, density=0.6, random_state=1, format="csr") + sp.eye(400) * 40.0
    A = A.tocsr()
    A.sort_indices()
    path = str(tmp_path / "a.bin")
    _write(A, path)
    r = subprocess.run([checker, path, "0"], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("no schedule"), r.stdout + r.stderr
