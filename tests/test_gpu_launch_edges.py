"""Cell and edge counts around the block sizes of the step kernels (64, 128
and 256 threads) and the groups of 32 cells of the interleaved stencils, with
stencils of 3, 12 and 18 entries and the limiter: state and norms of a small
Dirichlet box against the oracle (the boundary values' exp and pow differ from
its in the last bits, the norms' block sums are in another order)."""
import numpy as np
import pytest

import cases
from fvs2d_gb300 import PREC_FP64, PREC_FP64_DF, PREC_FP64_STRICT, PREC_MIXED, Solver, meshgen
from oracle_lib import Oracle
from test_gpu_parity import rel

pytestmark = pytest.mark.gpu

# 2 * nx * ny cells: 64, 66, 126, 128, 130, 256 and 258
SHAPES = [(8, 4), (11, 3), (9, 7), (8, 8), (13, 5), (16, 8), (43, 3)]
SCHEMES = {"ggcell": dict(grad_method=1), "ggnode": dict(grad_method=2),
           "lsq_nn_limited": dict(grad_method=3, lsq_stencil="nn", limiter=1)}
TOL = {PREC_FP64_STRICT: 1e-13, PREC_FP64: 1e-12, PREC_FP64_DF: 1e-12, PREC_MIXED: 2e-6}


@pytest.mark.parametrize("prec", sorted(TOL))
@pytest.mark.parametrize("scheme", sorted(SCHEMES))
@pytest.mark.parametrize("nx,ny", SHAPES)
def test_block_edges(nx, ny, scheme, prec):
    mesh = meshgen.dirichlet_square(nx, ny, jitter=0.1)
    _, opt = cases.dirichlet_vortex(dt=0.01, **SCHEMES[scheme])
    orc = Oracle(mesh, opt)
    orc.initialize_solution()
    u0 = orc.cvar
    n_ref = orc.time_integration(0.0, 3)
    with Solver(mesh, opt.replace(precision=prec)) as s:
        s.cvar = u0
        n = s.time_integration(0.0, 3)
        u = s.cvar
    tol = 1e-4 if prec == PREC_MIXED and "limited" in scheme else 3 * TOL[prec]
    assert rel(u, orc.cvar) <= tol, rel(u, orc.cvar)
    assert np.allclose(n, n_ref, rtol={PREC_MIXED: 1e-3, PREC_FP64_DF: 1e-9}.get(prec, 1e-10), atol=0)
