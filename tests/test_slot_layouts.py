"""The cell groups' slots as the kernels take them, checked on the host: every region
that the kernels write is inside the slot, overlaps no other and is aligned
(integrators with a Jacobian chunk's values, source terms, Jacobians)."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT
from test_layouts import CSRC, KNV, _disjoint


@pytest.fixture(scope="module")
def slots(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path_factory.mktemp("slots") / "print_slots")
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I" + CSRC, "-I" + os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "layout", "print_slots.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split("\n")
    rows = {kind: [list(map(int, ln.split()[1:])) for ln in out if ln.startswith(kind + " ")]
            for kind in ("step", "jac", "source")}
    assert all(rows.values())
    return rows


def check(regions, nbytes, what):
    assert _disjoint(regions, what) <= nbytes and nbytes % 16 == 0, what
    for name, off, _ in regions:
        assert off % 16 == 0, (what, name, off)


def test_integrator_slots(slots):
    for (ns, ntb, mixed, seulex, room, ld, offJ64, offLU64, offLU32, offVec, offVec32, offSp, offInvD, offScale, offPiv,
         offRx, offTb, offTable, offRed, nbytes) in slots["step"]:
        n = ns + 1
        m64, m32 = n * ld * 8, n * ld * 4
        assert ld >= n and ld % 2 == 1
        regions = [("J64", offJ64, m64), ("vectors", offVec, KNV * n * 8), ("species", offSp, 7 * ns * 8),
                   ("invD", offInvD, n * 8), ("piv", offPiv, n * 4), ("rates or chunk", offRx, room * 8),
                   ("third body", offTb, 2 * max(ntb, 1) * 8), ("reduction", offRed, 48 * 8)]
        if seulex:
            regions += [("LU64", offLU64, m64), ("table", offTable, 12 * n * 8)]
        else:
            assert offLU64 == offJ64
        if mixed:
            regions += [("x32, r32", offVec32, 2 * n * 4), ("scale", offScale, 2 * n * 8)]
            if seulex:  # inside the FP64 factors
                assert offLU64 <= offLU32 and offLU32 + m32 <= offLU64 + m64
            else:
                regions += [("LU32", offLU32, m32)]
        check(regions, nbytes, f"step ns={ns} nTB={ntb} mixed={mixed} seulex={seulex} room={room}")


def test_jacobian_slots(slots):
    for ns, ntb, values, ld, offJ64, offVec, offSp, offRx, offTb, offRed, nbytes in slots["jac"]:
        n = ns + 1
        check([("J64", offJ64, n * ld * 8), ("vectors", offVec, 2 * n * 8), ("species", offSp, 7 * ns * 8),
               ("chunk", offRx, values * 8), ("third body", offTb, 2 * max(ntb, 1) * 8), ("reduction", offRed, 48 * 8)],
              nbytes, f"jac ns={ns} nTB={ntb} values={values}")


def test_source_slots(slots):
    for ns, nr, ntb, offVec, offSp, offRx, offTb, offRed, nbytes in slots["source"]:
        n = ns + 1
        check([("vectors", offVec, 2 * n * 8), ("species", offSp, 5 * ns * 8), ("rates", offRx, max(nr, 1) * 8),
               ("third body", offTb, max(ntb, 1) * 8), ("reduction", offRed, 48 * 8)],
              nbytes, f"source ns={ns} nr={nr} nTB={ntb}")
