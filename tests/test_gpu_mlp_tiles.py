"""The network's tensor-core GEMMs at the edges of their 128 x 64 tiles, 64-wide
K blocks and gradient runs: gradients and predictions of both engines against
each other and the float64 oracle, on one handle whose workspaces grow and are
used again for smaller batches."""
import os
import sys

import numpy as np
import pytest

from fvs2d_gb300.mlp import MLP

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import mlp_oracle  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,width,depth,n_out", [(5, 16, 1, 1), (16, 64, 2, 16), (17, 80, 3, 17), (64, 144, 2, 64),
                                                    (8, 256, 2, 4), (3, 528, 1, 33)])
def test_tile_edges(n_in, width, depth, n_out):
    rng = np.random.default_rng(width)
    m = MLP(n_in, width, depth, n_out, seed=2)
    p = m.get_params() + (0.01 * rng.standard_normal(m.num_params())).astype(np.float32)
    m.set_params(p)
    for n in (1, 127, 129, 300, 64, 1025):
        x = rng.standard_normal((n, n_in)).astype(np.float32)
        y = (0.3 * rng.standard_normal((n, n_out))).astype(np.float32)
        ref_loss, ref_g = mlp_oracle.loss_grad(p, x.astype(np.float64), y.astype(np.float64), n_in, width, depth, n_out)
        got = {}
        for engine in ("tcgen05", "mma.sync"):
            m.set_engine(engine)
            loss, g = m.loss_grad(x, y)
            got[engine] = m.predict(x)
            # BF16 activations that fall the other way, one part in 256 each,
            # move the loss and a gradient by the bars of the gradient test
            assert abs(loss - ref_loss) <= 5e-5 * abs(ref_loss), (n, engine)
            assert np.linalg.norm(g - ref_g) <= 5e-4 * np.linalg.norm(ref_g), (n, engine)
        d = np.linalg.norm(got["tcgen05"] - got["mma.sync"])
        assert d <= 5e-4 * np.linalg.norm(got["mma.sync"]), n
    m.close()


@pytest.mark.parametrize("n_in,width,depth,n", [(8, 128, 2, 39100), (5, 112, 1, 38913), (17, 144, 2, 30001), (5, 256, 1, 65537)])
def test_wide_tiles(n_in, width, depth, n):
    """Predictions of enough rows for the hidden layers' 128-column tiles, whole
    and ragged in rows and columns: both engines against each other."""
    rng = np.random.default_rng(width)
    m = MLP(n_in, width, depth, 3, seed=2)
    x = rng.standard_normal((n, n_in)).astype(np.float32)
    got = {}
    for engine in ("tcgen05", "mma.sync"):
        m.set_engine(engine)
        got[engine] = m.predict(x)
    d = np.linalg.norm(got["tcgen05"] - got["mma.sync"], axis=1)
    # the bar of the tile test, and row by row with the margin of a BF16 rounding
    assert np.linalg.norm(d) <= 5e-4 * np.linalg.norm(got["mma.sync"])
    assert d.max() <= 2.0 ** -7 * np.linalg.norm(got["mma.sync"], axis=1).max()
    m.close()
