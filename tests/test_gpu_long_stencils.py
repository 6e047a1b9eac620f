"""GG-node stencils of several hundred cells (a fan of triangles around one
node; the LSQ setup takes at most 64): residuals against the oracle."""
import numpy as np
import pytest

import cases
from fvs2d_gb300 import PREC_FP64, PREC_FP64_STRICT, Solver, meshgen
from oracle_lib import Oracle
from test_gpu_parity import rel

pytestmark = pytest.mark.gpu


def fan(n):
    t = 2.0 * np.pi * np.arange(n) / n
    xy = np.concatenate([[[0.0, 0.0]], np.stack([np.cos(t), np.sin(t)], 1)])
    i = np.arange(n)
    tri = np.stack([np.ones(n), i + 2, (i + 1) % n + 2], 1).astype(np.int32)
    return meshgen.Mesh(xy, tri, np.zeros((0, 4), np.int32), ["freestream"], [(i + 1).astype(np.int32)], name=f"fan_{n}")


@pytest.mark.parametrize("n", [254, 255, 256, 257, 300])
def test_fan(n):
    mesh = fan(n)
    _, opt = cases.dirichlet_vortex(dt=0.01, grad_method=2)
    orc = Oracle(mesh, opt)
    orc.initialize_solution()
    rng = np.random.default_rng(n)
    u0 = orc.cvar * (1.0 + 0.01 * rng.standard_normal(orc.cvar.shape))
    orc.cvar = u0
    ref = orc.compute_residual()[0]
    # FP64: sums of up to 3 x 300 terms, rounded in another way (900 x 1.1e-16),
    # of values 100 times the differences that are left (a perturbation of 1 %)
    for prec, tol in ((PREC_FP64_STRICT, 0.0), (PREC_FP64, 1e-11)):
        with Solver(mesh, opt.replace(precision=prec)) as s:
            s.cvar = u0
            assert rel(s.compute_residual()[0], ref) <= tol, prec
