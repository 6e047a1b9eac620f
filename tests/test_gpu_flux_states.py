"""The FP64 and double-float Roe fluxes from near rest to Mach 3, across the
range where the entropy fix acts on either acoustic wave, with density and
pressure ratios of neighbours up to about 20: residuals of random cell states
on a periodic mesh against the oracle, first order and reconstructed."""
import numpy as np
import pytest

import cases
from fvs2d_gb300 import PREC_FP64, PREC_FP64_DF, Solver
from oracle_lib import Oracle
from test_gpu_parity import rel

pytestmark = pytest.mark.gpu


def states(n, mach, seed):
    r = np.random.default_rng(seed)
    rho, p = np.exp(r.uniform(-1.5, 1.5, n)), np.exp(r.uniform(-1.5, 1.5, n))
    q, th = mach * np.sqrt(1.4 * p / rho) * r.uniform(0.5, 1.0, n), r.uniform(0, 2 * np.pi, n)
    u, v = q * np.cos(th), q * np.sin(th)
    return np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)], 1)


@pytest.mark.parametrize("prec", [PREC_FP64, PREC_FP64_DF])
@pytest.mark.parametrize("mach", [1e-3, 0.3, 1.0, 1.3, 3.0])
@pytest.mark.parametrize("smooth", [False, True])
def test_flux_over_states(mach, smooth, prec):
    # first order: the flux of the cell states as drawn; reconstructed: close
    # to one state, so that no face value leaves the physical range
    mesh, opt = cases.periodic_vortex(13, jitter=0.2, vortex=False, reconst=2 if smooth else 1)
    u = states(mesh.ncells, mach, 3)
    if smooth:
        u = states(1, mach, 5) * (1.0 + 0.01 * (u / np.abs(u).max(0)))
    orc = Oracle(mesh, opt)
    orc.cvar = u
    r_ref, w_ref = orc.compute_residual(0.0)
    assert np.isfinite(r_ref).all()
    with Solver(mesh, opt.replace(precision=prec)) as s:
        s.cvar = u
        r, w = s.compute_residual(0.0)
    # per component: the energy flux would hide the others; a reconstructed
    # residual cancels fluxes about 100 times its size
    tol = 1e-12 * (100 if smooth else 1)
    for k in range(4):
        assert rel(r[:, k], r_ref[:, k]) <= tol, (k, rel(r[:, k], r_ref[:, k]))
    assert rel(w, w_ref) <= 1e-12
