"""Field transfers between host boxes and the device columns."""
import numpy as np
import pytest

from openswpc_b200 import _lib
from openswpc_b200._lib import check, fptr
from tests.models import small2d, small3d

pytestmark = pytest.mark.gpu


def _run(kind, dims):
    if kind == "3d":
        from openswpc_b200.swpc3d import Swpc3D

        return Swpc3D(small3d(nx=dims[1], ny=dims[2], nz=dims[0], na=4, nt=2), medium_on_device=True)
    from openswpc_b200.swpc2d import Swpc2D

    return Swpc2D(small2d(kind, nx=dims[1], nz=dims[0], na=4, nt=2), kind)


# the smallest box, odd sizes, rows of whole warps, and a box of several staging chunks
@pytest.mark.parametrize("kind,dims", [("3d", (13, 21, 22)), ("3d", (67, 43, 31)), ("3d", (58, 26, 26)),
                                       ("3d", (250, 282, 270)), ("psv", (33, 57, 1)), ("sh", (250, 519, 1))])
def test_download_box(kind, dims):
    """A box without padding (packed on the device) and one with padding (row
    by row) hold the uploaded field; the padding keeps its values."""
    run = _run(kind, dims)
    shape = ((dims[2] + 6,) if kind == "3d" else ()) + (dims[1] + 6, dims[0] + 6)
    field = _lib.F_VY if kind == "sh" else _lib.F_VX
    a = np.random.default_rng(3).standard_normal(shape).astype(np.float32)
    run.upload(field, a)
    b = run.download(field)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    pad = np.full(shape[:-2] + (shape[-2] + 2, shape[-1] + 3), -7.0, np.float32)
    check(run.ctx, run.lib.swpc_download_field(run.ctx, field, fptr(pad), shape[-1] + 3, shape[-2] + 2))
    assert np.array_equal(pad[..., :-2, :-3].view(np.uint32), a.view(np.uint32))
    assert np.all(pad[..., -3:] == -7.0)
    assert np.all(pad[..., -2:, :] == -7.0)
    run.close()


# page-locked boxes on both sides of the row length and of the size at which a 3D download is packed, and 2D ones
@pytest.mark.parametrize("kind,dims", [("3d", (250, 109, 101)), ("3d", (250, 102, 101)), ("3d", (121, 27, 25)),
                                       ("3d", (122, 27, 25)), ("3d", (29, 31, 26)), ("psv", (33, 57, 1)),
                                       ("sh", (250, 519, 1))])
def test_download_into_page_locked_memory(kind, dims):
    import torch
    run = _run(kind, dims)
    shape = ((dims[2] + 6,) if kind == "3d" else ()) + (dims[1] + 6, dims[0] + 6)
    field = _lib.F_VY if kind == "sh" else _lib.F_VX
    a = np.random.default_rng(4).standard_normal(shape).astype(np.float32)
    run.upload(field, a)
    b = torch.full(shape, -7.0).pin_memory().numpy()
    check(run.ctx, run.lib.swpc_download_field(run.ctx, field, fptr(b), shape[-1], shape[-2]))
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    run.close()
