"""The autotuner leaves the batch's state and primitives as it found them:
steps after it give, bit for bit, those of a batch that was not tuned."""
import numpy as np
import pytest

import cases
from fvs2d_gb300 import PREC_MIXED
from fvs2d_gb300.batch import Batch

pytestmark = pytest.mark.gpu


def test_steps_after_autotune():
    meshes, opts = [], []
    for nw, nr, mach in ((96, 40, 0.5), (128, 60, 0.7), (64, 30, 0.8)):
        m, o = cases.airfoil(nw=nw, nr=nr, mach_inf=mach, reconst=1, precision=PREC_MIXED)
        meshes.append(m)
        opts.append(o)
    got = []
    for tunes in (0, 1, 1, 1, 1):
        with Batch(meshes, opts) as b:
            b.initialize_solution()
            b.steps(20)
            for _ in range(tunes):
                b.autotune(3)
            b.steps(50)
            got.append([b.get_state(c) for c in range(b.ncases)])
    for g in got[1:]:
        for x, y in zip(g, got[0]):
            assert np.array_equal(x, y)
