"""Rounding of the rearranged Roe fluxes: root mean square error of first-order
residuals and wave-speed sums against extended precision.

The states keep the conversion to primitives exact (density 1, velocities and
pressure multiples of 2^-12, gamma 3/2), so that what is measured is the flux
and its sum over the faces.  Bars, in units of pressure times the mean face
length for the momentum and relative for the wave speed:

FP64: the momentum no further off than the strict mode's, which takes the
source's order (an emulation of both gives 0.71 to 0.83 of it; 1.12 to 1.29
when the momentum flux is turned back from the face's frame as a whole).

Double-float, log2: emulated with the correctly rounded roots and divisions
and the momentum summed in x and y -48.1 (Mach 0.01) and -47.9 (0.5) for the
momentum, -49.0 and -49.1 for the wave speed; turned back from the face's frame
with a reciprocal root of 2^-44, 0.5 and 1.1 to 0.9 more.  Half way."""
import numpy as np
import pytest

import cases
from fvs2d_gb300 import PREC_FP64, PREC_FP64_DF, PREC_FP64_STRICT, Solver

pytestmark = pytest.mark.gpu

GAMMA = 1.5
X = np.longdouble


def roe(pl, pr, nx, ny):
    """Twice the flux and wave speed per unit length, src/flux_invscid.f90:37-136."""
    (rl, ul, vl, ql), (rr, ur, vr, qr) = pl, pr
    g1 = X(GAMMA) - 1
    unl, unr, utl, utr = ul * nx + vl * ny, ur * nx + vr * ny, vl * nx - ul * ny, vr * nx - ur * ny
    hl, hr = X(GAMMA) / g1 * ql / rl + (ul * ul + vl * vl) / 2, X(GAMMA) / g1 * qr / rr + (ur * ur + vr * vr) / 2
    rt = np.sqrt(rr / rl)
    rho, u, v, h = rt * rl, (ul + rt * ur) / (1 + rt), (vl + rt * vr) / (1 + rt), (hl + rt * hr) / (1 + rt)
    q2 = (u * u + v * v) / 2
    a = np.sqrt(g1 * (h - q2))
    un, ut = u * nx + v * ny, v * nx - u * ny
    dp, dun = qr - ql, unr - unl
    fix = lambda w: np.where(w < 0.2, (w * w * 5 + X(1) / 5) / 2, w)  # noqa: E731
    w0, w3 = fix(abs(un - a)) * (dp - rho * a * dun) / (2 * a * a), fix(abs(un + a)) * (dp + rho * a * dun) / (2 * a * a)
    w1, w2 = abs(un) * rho * (utr - utl), abs(un) * (rr - rl - dp / (a * a))
    s = w0 + w3
    sd, dw = s + w2, (w3 - w0) * a
    ml, mr = rl * unl, rr * unr
    return np.stack([ml + mr - sd, ml * ul + mr * ur + (ql + qr) * nx - (u * sd + dw * nx - w1 * ny),
                     ml * vl + mr * vr + (ql + qr) * ny - (v * sd + dw * ny + w1 * nx),
                     ml * hl + mr * hr - (h * s + un * dw + w1 * ut + w2 * q2)], 1), abs(un) + a


def errors(mach, precs):
    mesh, opt = cases.periodic_vortex(64, jitter=0.2, vortex=False, reconst=1, gamma=GAMMA)
    rng = np.random.default_rng(1)
    n = mesh.ncells
    q = mach * GAMMA ** 0.5
    grid = lambda x: np.round(4096 * x) / 4096  # noqa: E731
    prim = np.stack([np.ones(n), grid(q * np.cos(0.7) + 0.05 * rng.uniform(-1, 1, n)),
                     grid(q * np.sin(0.7) + 0.05 * rng.uniform(-1, 1, n)), grid(1 + 0.05 * rng.uniform(-1, 1, n))])
    rho, u, v, p = prim
    state = np.stack([rho, rho * u, rho * v, 2.0 * p + 0.5 * rho * (u * u + v * v)], 1)
    exact, out = None, {}
    for prec in precs:
        with Solver(mesh, opt.replace(precision=prec)) as s:
            if exact is None:
                geo, ec = s.export("edge_geom").reshape(-1, 7), s.export("edge_cells").reshape(-1, 2) - 1
                vol, area = s.export("cell_vol"), geo[:, 2]
                assert ec.min() == 0 and ec.max() == n - 1
                f, w = roe(prim[:, ec[:, 0]].astype(X), prim[:, ec[:, 1]].astype(X), geo[:, 3].astype(X), geo[:, 4].astype(X))
                exact, ws = np.zeros((n, 4), X), np.zeros(n, X)
                half = area.astype(X) / 2
                for side, sign in ((0, -1), (1, 1)):
                    np.add.at(exact, ec[:, side], sign * f * half[:, None])
                    np.add.at(ws, ec[:, side], w * half)
                exact /= vol.astype(X)[:, None]
            s.cvar = state
            r, wsum = s.compute_residual(0.0)
        d = ((r - exact) * vol[:, None]).astype(np.float64)[:, 1:3] / area.mean()
        out[prec] = np.sqrt((d * d).mean()), np.sqrt((((wsum - ws) / ws).astype(np.float64) ** 2).mean())
    return out


@pytest.mark.parametrize("mach", [0.01, 0.5, 1.0, 3.0])
def test_fp64_momentum(mach):
    e = errors(mach, (PREC_FP64_STRICT, PREC_FP64))
    assert e[PREC_FP64_STRICT][0] < 1e-14  # the extended-precision residual is the strict mode's
    assert e[PREC_FP64][0] <= e[PREC_FP64_STRICT][0], (e, e[PREC_FP64][0] / e[PREC_FP64_STRICT][0])


@pytest.mark.parametrize("mach,momentum,wave", [(0.01, -47.85, -48.5), (0.5, -47.65, -48.6)])
def test_double_float(mach, momentum, wave):
    m, w = errors(mach, (PREC_FP64_DF,))[PREC_FP64_DF]
    assert np.log2(m) <= momentum and np.log2(w) <= wave, (np.log2(m), np.log2(w))
