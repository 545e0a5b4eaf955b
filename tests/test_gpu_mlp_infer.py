"""The inference kernel of the surrogate at the edges of its tiles, against the
CPU oracle: row counts around the 128-row tile and beyond one tile per
resident block, inputs and outputs around their 64- and 128-column padding,
one hidden layer to eight.  Tolerances as in test_gpu_mlp.py."""
import numpy as np
import pytest

from mlp_oracle import MlpOracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,n_out,depth,n", [(1, 1, 1, 1), (64, 128, 2, 127), (65, 129, 1, 128), (56, 55, 4, 129),
                                                (128, 31, 8, 255), (129, 256, 3, 300), (256, 32, 2, 41000)])
def test_forward_at_tile_edges(n_in, n_out, depth, n):
    import __graft_entry__
    __graft_entry__.build()
    from fcs import _lib
    rng = np.random.default_rng(n_in + n)
    mlp = _lib.Mlp(n_in, n_out, width=256, depth=depth, members=1, seed=2)
    mlp.set_normalization(rng.normal(0, 0.5, n_in), rng.uniform(0.5, 2.0, n_in), rng.normal(0, 1, n_out),
                          rng.uniform(0.1, 3.0, n_out))
    x = rng.normal(0, 1, (n, n_in)).astype(np.float32)
    y = mlp.forward(0, x)
    some = np.unique(np.concatenate([np.arange(min(n, 200)), np.arange(max(0, n - 200), n)]))
    im, is_, om, os_ = mlp.get_normalization()
    ref, _, _ = MlpOracle(mlp.unflatten(mlp.get_params(0)), im, is_, om, os_).forward(x[some])
    scale = np.abs(ref).max()
    err = np.abs(y[some] - ref)
    assert err.max() <= 1e-2 * scale and err.mean() <= 2e-3 * scale, (err.max(), err.mean(), scale)
    # every row the same as when it is alone in the batch
    k = n - 1
    np.testing.assert_array_equal(mlp.forward(0, x[k:k + 1])[0], y[k])
    mlp.close()
