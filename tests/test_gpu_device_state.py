"""fvs_set_state, and the batch's, are complete when they return: the array that
fvs_device_state gives out is read at once on a stream that knows nothing of
the handle's, and by the next calls."""
import ctypes as C

import numpy as np
import pytest

import cases
from fvs2d_gb300 import PREC_MIXED, Solver, meshgen

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


class DeviceArray:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n, 4), "typestr": "<f8", "data": (ptr, False), "version": 3}


@pytest.mark.parametrize("prec", [0, PREC_MIXED])
def test_state_read_on_another_stream(prec):
    mesh = meshgen.periodic_square(512, 400, jitter=0.2)
    opt = cases.periodic_vortex(4)[1].replace(precision=prec)
    with Solver(mesh, opt) as s:
        ptr = C.c_void_p()
        s._check(s._lib.fvs_device_state(s._h, C.byref(ptr)))
        u = torch.as_tensor(DeviceArray(ptr.value, s.ncells), device="cuda")
        side = torch.cuda.Stream()
        r = np.random.default_rng(1)
        for _ in range(5):
            state = 1.0 + r.random((s.ncells, 4))
            s.cvar = state
            with torch.cuda.stream(side):
                seen = u.clone()
            side.synchronize()
            # the RCM order permutes whole cells
            got = seen.cpu().numpy()
            assert np.array_equal(got[np.lexsort(got.T)], state[np.lexsort(state.T)])
            assert np.array_equal(s.cvar, state)
