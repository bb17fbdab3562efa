"""The adjoint state of a context across failed calls and changed recorders."""
import ctypes as C

import numpy as np
import pytest

from openswpc_b200._lib import check, fptr
from openswpc_b200.swpc3d import Swpc3D
from tests.models import small3d

pytestmark = pytest.mark.gpu

NOMEM = 5


def _gradient(g, p, obs):
    J = C.c_double()
    check(g.ctx, g.lib.swpc_gradient(g.ctx, fptr(obs), 4, C.byref(J)))
    out = []
    for w in range(8):
        a = np.zeros((p.ny + 6, p.nx + 6, p.nz + 6), np.float64)
        check(g.ctx, g.lib.swpc_gradient_fetch(g.ctx, w, a.ctypes.data_as(C.POINTER(C.c_double)), p.nz + 6, p.nx + 6))
        out.append(a)
    return J.value, out


def _same(a, b):
    assert a[0] == b[0]
    assert max(np.abs(x).max() for x in a[1]) > 0
    for x, y in zip(a[1], b[1]):
        assert np.array_equal(x.view(np.uint64), y.view(np.uint64))


def test_gradient_after_the_adjoint_state_found_no_room():
    """Calls that find no room for one of the adjoint's blocks report it, leave
    nothing allocated, and the gradient after them equals a fresh context's."""
    import torch
    p = small3d(nx=128, ny=128, nz=64, na=12, nt=16)
    g = Swpc3D(p)
    obs = np.zeros_like(g.waveforms())
    held = g.lib.swpc_device_bytes(g.ctx)
    # 413 MiB in blocks of 148 (state), 49 + 49 (bases), 1, 34 (auxiliaries), 88 (totals) and 44 MiB (sums)
    for left in (64, 170, 220, 265, 320, 390):
        free, _ = torch.cuda.mem_get_info(0)
        filler = torch.empty(free - (left << 20), dtype=torch.uint8, device="cuda:0")
        for _ in range(2):
            assert g.lib.swpc_adj_reset(g.ctx) == NOMEM, left
            assert g.lib.swpc_device_bytes(g.ctx) == held
        del filler
        torch.cuda.empty_cache()
    got = _gradient(g, p, obs)
    fresh = Swpc3D(p)
    _same(got, _gradient(fresh, p, obs))
    g.close()
    fresh.close()
