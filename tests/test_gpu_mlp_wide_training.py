"""Loss and gradients of batches large enough for the network's two-stage
GEMMs in training: 128-column hidden layers that also store their
pre-activations, the two-stage backward and the two-stage loss epilogue.  Rows
ragged (306 row tiles, the last of 60 rows), widths whole and ragged."""
import os
import sys

import numpy as np
import pytest

from fvs2d_gb300.mlp import MLP

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import mlp_oracle  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,width,n_out", [(8, 256, 4), (17, 144, 33)])
def test_loss_grad_of_large_batches(n_in, width, n_out):
    n, depth = 39_100, 2
    rng = np.random.default_rng(width)
    m = MLP(n_in, width, depth, n_out, seed=2)
    p = m.get_params() + (0.01 * rng.standard_normal(m.num_params())).astype(np.float32)
    m.set_params(p)
    x = rng.standard_normal((n, n_in)).astype(np.float32)
    y = (0.3 * rng.standard_normal((n, n_out))).astype(np.float32)
    ref_loss, ref = mlp_oracle.loss_grad(p, x.astype(np.float64), y.astype(np.float64), n_in, width, depth, n_out)
    got = {}
    for engine in ("tcgen05", "mma.sync"):
        m.set_engine(engine)
        loss, got[engine] = m.loss_grad(x, y)
        # the bars of the tile test
        assert abs(loss - ref_loss) <= 5e-5 * abs(ref_loss), (engine, loss, ref_loss)
        assert np.linalg.norm(got[engine] - ref) <= 5e-4 * np.linalg.norm(ref), engine
    m.close()
    # layer by layer, weights and biases: twice that bar between the engines
    at = 0
    for rows, cols in ((width, n_in), (width, width), (n_out, width)):
        for k in (rows * cols, rows):
            a, b = got["tcgen05"][at:at + k], got["mma.sync"][at:at + k]
            assert np.linalg.norm(a - b) <= 1e-3 * np.linalg.norm(b), (rows, cols, k)
            at += k
    assert at == len(ref)
