"""The inference kernel's shared memory on the host (tests/layout/check_infer_layout.cpp)
and, on the GPU, batches whose blocks take several tiles."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "fastchemistrysolver-openfoam-10_gb300", "csrc")


def test_staged_outputs_and_next_inputs_share_no_byte(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    exe = str(tmp_path / "check_infer_layout")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC,
                    os.path.join(ROOT, "tests", "layout", "check_infer_layout.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("n_in,n_out,n", [(13, 12, 41000), (13, 1, 100003), (65, 34, 65536), (130, 48, 80001),
                                          (56, 55, 65536), (130, 16, 100003), (65, 33, 65536)])
def test_every_row_of_several_tiles_per_block(n_in, n_out, n):
    """More than two resident blocks per SM times 128 rows: a block goes on to a
    second and a third tile while a warp that had more output columns still stores
    the tile before.  Every row has the bits of batches with one tile per block."""
    import __graft_entry__
    __graft_entry__.build()
    from fcs import _lib
    rng = np.random.default_rng(n_in * n_out)
    mlp = _lib.Mlp(n_in, n_out, width=256, depth=2, members=1, seed=3)
    mlp.set_normalization(rng.normal(0, 0.5, n_in), rng.uniform(0.5, 2.0, n_in), rng.normal(0, 1, n_out),
                          rng.uniform(0.1, 3.0, n_out))
    x = rng.normal(0, 1, (n, n_in)).astype(np.float32)
    parts = np.concatenate([mlp.forward(0, x[k:k + 19000]) for k in range(0, n, 19000)])
    for _ in range(3):
        np.testing.assert_array_equal(mlp.forward(0, x), parts)
    mlp.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n_in,n_out,shift", [(56, 55, 0), (13, 12, 128), (20, 64, 0)])
def test_forward_in_place(n_in, n_out, shift):
    """Device arrays that overlap: the result is that of separate arrays."""
    import __graft_entry__
    __graft_entry__.build()
    import torch
    from fcs import _lib
    n = 3000
    mlp = _lib.Mlp(n_in, n_out, width=256, depth=2, members=1, seed=4)
    x = np.random.default_rng(n_in).normal(0, 1, (n, n_in)).astype(np.float32)
    buf = torch.zeros(n * max(n_in, n_out) + shift, dtype=torch.float32, device="cuda")
    buf[:n * n_in] = torch.from_numpy(x.ravel()).cuda()
    torch.cuda.synchronize()
    at = buf.data_ptr()
    mlp._check(mlp.L.fcs_mlp_forward(mlp.h, 0, n, at, at + 4 * shift, _lib.PTR_DEVICE))
    y = buf[shift:shift + n * n_out].cpu().numpy().reshape(n, n_out)
    np.testing.assert_array_equal(y, mlp.forward(0, x))
    mlp.close()
