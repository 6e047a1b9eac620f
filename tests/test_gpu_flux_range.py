"""The Roe flux's range: densities and pressures far from 1, and of two cells
both negative, give the finite residual that the source form gives."""
import numpy as np
import pytest

import cases
from fvs2d_gb300 import PREC_FP64, PREC_FP64_DF, Solver
from oracle_lib import Oracle
from test_gpu_parity import rel

pytestmark = pytest.mark.gpu


# the double-float mode's range is FP32's
@pytest.mark.parametrize("prec,scale", [(PREC_FP64, s) for s in (-1.0, 1e-200, 1e-154, 1e154, 1e200, -1e-200, -1e200)]
                         + [(PREC_FP64_DF, -1.0)])
def test_scaled_states(prec, scale):
    mesh, opt = cases.periodic_vortex(9, jitter=0.2, vortex=False, reconst=1)
    r = np.random.default_rng(7)
    n = mesh.ncells
    rho, p = r.uniform(0.5, 2.0, n), r.uniform(0.5, 2.0, n)
    u, v = r.uniform(-1.5, 1.5, (2, n))
    state = scale * np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)], 1)
    orc = Oracle(mesh, opt)
    orc.cvar = state
    ref, ws = orc.compute_residual(0.0)
    assert np.isfinite(ref).all() and np.isfinite(ws).all()
    with Solver(mesh, opt.replace(precision=prec)) as s:
        s.cvar = state
        got, w = s.compute_residual(0.0)
    # the bar of the flux test, per component
    for k in range(4):
        assert rel(got[:, k], ref[:, k]) <= 1e-12, k
    assert rel(w, ws) <= 1e-12
