"""A kernel launch that fails inside a solve ends it with HMVM_ECUDA: the work
vectors and scalars stay with the plan between solves, so what the kernel did not
write would be an earlier solve's.  csrc/solve.cu is linked here with a CUDA
runtime that runs nothing and refuses the K-th launch."""
import os
import subprocess

import pytest

from hacapk_hmvm_b200 import _lib, build
from helpers import ROOT


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    d = tmp_path_factory.mktemp("solver")
    inc = os.path.join(ROOT, "include")
    subprocess.run([build._nvcc(), "-O1", "-std=c++17", *build.ARCH, "-ccbin", build._hostcxx(), "-I", inc, "-c",
                    "-o", str(d / "solve.o"), os.path.join(build.CSRC, "solve.cu")], check=True)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc()))), "include")
    subprocess.run([build._hostcxx(), "-std=c++17", "-I", inc, "-I", cuda, "-o", str(d / "probe"),
                    os.path.join(ROOT, "tests", "cxx", "solver_launch_probe.cpp"), str(d / "solve.o")], check=True)

    def run(solver, k):
        out = subprocess.run([str(d / "probe"), solver, str(k)], capture_output=True, text=True, check=True).stdout
        rc, steps, relres, launches = out.split()
        return int(rc), int(steps), float(relres), int(launches)

    return run


@pytest.mark.parametrize("solver", ["bicgstab", "gcrm"])
def test_any_failed_launch_ends_the_solve(probe, solver):
    launches = probe(solver, 0)[3]  # none refused: the scalars are all 1, so three steps are taken
    assert launches > 10
    for k in range(1, launches + 1):
        rc, _, _, seen = probe(solver, k)
        assert rc == _lib.HMVM_ECUDA, k
        assert seen == k  # nothing was launched after it
