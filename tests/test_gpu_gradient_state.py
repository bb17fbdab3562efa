"""The adjoint state of a context across failed calls and changed recorders."""
import ctypes as C

import numpy as np
import pytest

from openswpc_b200._lib import WAV_V, check, fptr, iptr
from openswpc_b200.params import Station
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


def test_gradient_after_the_recorder_was_set_up_again():
    """A recorder set up again with more samples than the gradient before had:
    misfit and gradients equal those of a fresh context with that recorder."""
    p = small3d(nx=40, ny=36, nz=32, na=8, nt=24)
    g = Swpc3D(p)
    rng = np.random.default_rng(4)

    def recorder(r, nst, ntdec_w):
        q = np.random.default_rng(nst)
        pos = [q.integers(p.na + 2, n - p.na - 2, nst).astype(np.int32) for n in (p.nx, p.ny, p.nz)]
        check(r.ctx, r.lib.swpc_wav_setup(r.ctx, nst, *(iptr(a) for a in pos), ntdec_w, WAV_V, r.M0, r.UC))

    for nst, ntdec_w in ((2, 8), (40, 8), (40, 1), (2, 8)):
        obs = rng.standard_normal((nst, 3, (p.nt - 1) // ntdec_w + 1)).astype(np.float32)
        recorder(g, nst, ntdec_w)
        got = _gradient(g, p, obs)
        fresh = Swpc3D(p)
        recorder(fresh, nst, ntdec_w)
        _same(got, _gradient(fresh, p, obs))
        fresh.close()
    g.close()


def test_device_gradient_of_converted_models():
    """float64 and transposed CUDA models, which torch converts on its own
    stream before the library reads them, give the bits of contiguous float32
    ones (256 x 256 x 128 cells: the conversion outlasts the host's way to
    the kernel)."""
    import torch
    from openswpc_b200.adjoint import Misfit3D
    p = small3d(nx=256, ny=256, nz=128, na=12, nt=12, stations=[Station(1.0, 0.5, 6.0, "st", "dep")])
    shape = (p.ny + 6, p.nx + 6, p.nz + 6)
    q = np.full(shape, 200.0, np.float32)
    vs = np.full(shape, 3.0, np.float32)
    vs *= 1 + 0.05 * np.random.default_rng(2).random(shape, np.float32)
    vp, rho = vs * np.float32(1.75), np.full(shape, 2.7, np.float32)
    prob = Misfit3D(p, vp, vs, rho, q, q, np.ones((1, 3, p.nt), np.float32), ckpt=4)
    f32 = [torch.from_numpy(a).cuda() for a in (vp, vs, rho)]
    ref = prob.gradient(*f32)
    assert all(float(g.abs().max()) > 0 for g in ref[1:])
    for model in ([t.double() for t in f32], [t.permute(2, 1, 0).contiguous().permute(2, 1, 0) for t in f32]):
        got = prob.gradient(*model)
        assert got[0] == ref[0]
        for a, b in zip(got[1:], ref[1:]):
            assert torch.equal(a.view(torch.int64), b.view(torch.int64))
    prob.close()
