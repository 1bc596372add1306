"""The LU analysis tries the multifrontal path itself; whatever refuses it must
leave the row-wise paths.  lu_trial_check.cpp links the engine's own objects to
a CUDA runtime that runs nothing and fails the call it is told to (no GPU)."""
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

from helpers import circuit_jacobian
from xyce_gb300 import build, netlists

HERE = os.path.dirname(os.path.abspath(__file__))
OOM, CUDA = -3, -2


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not found")
    build.build_engine()
    tmp = tmp_path_factory.mktemp("trial")
    exe, path = str(tmp / "lu_trial_check"), str(tmp / "a.bin")
    objs = [os.path.join(build.BUILD, f"{f}.o") for f in ("lu_kernels", "lu_front", "lu_front_plan", "lu_symbolic")]
    cuda = build._cuda_home(build._nvcc())
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I" + build.CSRC, "-I" + os.path.join(build.REPO, "include"),
                        "-I" + os.path.join(cuda, "include"), os.path.join(HERE, "lu_trial_check.cpp")] + objs +
                       ["-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    # logic: fronts of 16 CTAs, and a supply row summed by a cluster
    A = circuit_jacobian(netlists.random_logic(17000, seed=4), seed=4, pdt=1e12)
    A.sort_indices()
    with open(path, "wb") as f:
        np.array([A.shape[0], A.nnz], np.int64).tofile(f)
        A.indptr.astype(np.int32).tofile(f)
        A.indices.astype(np.int32).tofile(f)
        A.data.astype(np.float64).tofile(f)

    def go(*args):
        r = subprocess.run([exe, path] + [str(a) for a in args], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
        m = re.fullmatch(r"rc (-?\d+) path (\w+) pending (\d+) status (-?\d+) allocations (\d+)\s*", r.stdout)
        return int(m[1]), m[2], int(m[3]), int(m[4]), int(m[5])

    return go


def test_granted_everything_the_tree_is_taken(run):
    assert run()[:4] == (0, "front", 0, 0)


@pytest.mark.parametrize("refusal", [("cluster", 8), ("cluster", 4), ("launch", 8), ("copies", 1), ("copies", 2),
                                     ("pivot",)])
def test_refused_the_rows_are(run, refusal):
    assert run(*refusal)[:4] == (0, "rows", 0, 0)


def test_memory_that_runs_out(run):
    """Whichever allocation fails: the rows when it was the tree's (the plan's
    arrays come one after another), out of memory when it was the matrix's."""
    got = [run("memory", k)[:4] for k in range(1, run()[4] + 1, 3)]
    rows = [g for g in got if g[0] == 0]
    assert len(rows) >= len(got) - 4 and set(rows) == {(0, "rows", 0, 0)}
    assert all(g[0] in (0, OOM, CUDA) for g in got)
