"""The cell groups' reaction lists against the incidence walk they replace, on
the host (tests/layout/check_lists.cpp): every sum's terms and their order,
and every index the kernels use, at the edges of the chunks."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "fastchemistrysolver-openfoam-10_gb300", "csrc")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    exe = str(tmp_path_factory.mktemp("lists") / "check_lists")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-I" + CSRC,
                    os.path.join(ROOT, "tests", "layout", "check_lists.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("ns,nr", [(1, 0), (1, 1), (2, 15), (5, 16), (10, 27), (31, 64), (33, 65), (53, 325), (111, 256),
                                   (140, 643), (200, 1500), (255, 257)])
def test_lists_equal_the_incidence_walk(checker, ns, nr):
    for seed in range(3):
        r = subprocess.run([checker, str(ns), str(nr), str(seed)], capture_output=True, text=True)
        assert r.returncode == 0 and r.stdout == "ok\n", (ns, nr, seed, r.stdout)
