"""Point sources, recorder and step counter inside the staged launches against
the launches of their own (flat and tile-walking kernels), bitwise."""
import numpy as np
import pytest

from openswpc_b200 import _lib
from openswpc_b200._lib import check
from openswpc_b200.params import Source, Station
from openswpc_b200.swpc2d import Batch2D, Swpc2D
from openswpc_b200.swpc3d import Swpc3D
from tests.models import small2d, small3d

pytestmark = pytest.mark.gpu


def _sources(p, n, seed, force):
    """Seeded sources over the whole grid, several in the same cell and some at its edges."""
    g = np.random.default_rng(seed)
    out = []
    for q in range(n):
        if q % 3 == 2:
            x, y, z = out[-1].x, out[-1].y, out[-1].z
        else:
            i = 1 if q % 7 == 3 else int(g.integers(2, p.nx))
            j = p.ny if q % 7 == 4 else int(g.integers(2, max(p.ny, 3)))
            k = int(g.integers(5, p.nz))
            x, z = p.xbeg + (i - 0.5) * p.dx, p.zbeg + (k - 0.5) * p.dz
            y = p.ybeg + (j - 0.5) * p.dy if p.ny > 1 else 0.0
        m = g.uniform(-1, 1, 6)
        out.append(Source(x, y, z, 0.0, 0.3, mo=1e15, mxx=m[0], myy=m[1], mzz=m[2], myz=m[3], mxz=m[4], mxy=m[5],
                          fx=m[0] * force, fy=m[1] * force, fz=m[2] * force))
    return out


def _same(a, b):
    return np.array_equal(np.ascontiguousarray(a, np.float32).view(np.uint32),
                          np.ascontiguousarray(b, np.float32).view(np.uint32))


# one and several steps per graph with a remainder; one and several recorder CTAs (64 stations each); grids whose
# tiles are partial in k, i and j
@pytest.mark.parametrize("mode", ["glut", "force", "green"])
@pytest.mark.parametrize("dims,nsrc,nst,nt", [((21, 23, 13), 1, 1, 9), ((40, 36, 33), 40, 65, 23),
                                              ((33, 29, 64), 7, 64, 10)])
def test_step3d(mode, dims, nsrc, nst, nt):
    p = small3d(nx=dims[0], ny=dims[1], nz=dims[2], na=4, nt=nt, sw_wav_u=True, sw_wav_strain=True,
                bf_mode=mode == "force", green_mode=mode == "green", green_trise=0.5)
    g = np.random.default_rng(5)
    p.stations = [Station(p.xbeg + (int(g.integers(2, p.nx)) - 0.5) * p.dx,
                          p.ybeg + (int(g.integers(2, p.ny)) - 0.5) * p.dy, 0.5, f"s{n}", "fsb") for n in range(nst)]
    p.sources = _sources(p, nsrc, 11, 1.0)
    runs = []
    for flat in (False, True):
        r = Swpc3D(p, medium_on_device=True)
        if mode == "green":
            r.record(what=_lib.WAV_V | _lib.WAV_U | _lib.WAV_STRAIN)
        if flat:
            check(r.ctx, r.lib.swpc_set_launch(r.ctx, 0, 2, 2, 1))
            check(r.ctx, r.lib.swpc_set_launch(r.ctx, 1, 4, 2, 2))
        r.run(1, nt)
        runs.append([r.waveforms(w) for w in (_lib.WAV_V, _lib.WAV_U, _lib.WAV_STRAIN)] +
                    [r.download(f) for f in range(9)])
        r.close()
    assert np.abs(runs[0][3]).max() > 0
    for a, b in zip(*runs):
        assert _same(a, b)


@pytest.mark.parametrize("kind", ["psv", "sh"])
@pytest.mark.parametrize("dims,nsrc,nst,nt", [((19, 14), 1, 1, 9), ((120, 61), 30, 65, 23), ((48, 33), 5, 64, 10)])
def test_step2d(kind, dims, nsrc, nst, nt):
    """A single run and a batch with a second model, staged and tile-walking."""
    def params(seed):
        p = small2d(kind, nx=dims[0] + seed, nz=dims[1], na=4, nt=nt)
        g = np.random.default_rng(seed)
        p.stations = [Station(p.xbeg + (int(g.integers(2, p.nx)) - 0.5) * p.dx, 0.0, 0.3, f"s{n}", "fsb")
                      for n in range(nst)]
        p.sources = _sources(p, nsrc, seed, 0.0)
        return p

    def out(r):
        return [r.waveforms(w) for w in (_lib.WAV_V, _lib.WAV_U)] + [r.download(f) for f in r.field_ids.values()]

    single = []
    for flat in (False, True):
        r = Swpc2D(params(1), kind)
        if flat:
            check(r.ctx, r.lib.swpc_set_launch(r.ctx, 0, 1, 1, 1))
            check(r.ctx, r.lib.swpc_set_launch(r.ctx, 1, 1, 1, 1))
        r.run(1, nt)
        single.append(out(r))
    assert max(np.abs(f).max() for f in single[0][2:]) > 0
    for a, b in zip(*single):
        assert _same(a, b)
    for staged in (8, 0):
        runs = [Swpc2D(params(s), kind) for s in (1, 2)]
        b = Batch2D(runs)
        b.set_staged(staged, staged)
        b.run(1, nt)
        for x, y in zip(out(runs[0]), single[0]):
            assert _same(x, y)
        b.close()


@pytest.mark.parametrize("what", ["green_store", "medium"])
def test_setup_between_runs(what):
    """A setup change between two runs of whole step graphs reaches the second one."""
    p = small3d(nx=33, ny=29, nz=30, na=4, nt=40)
    out = []
    for graphs in (True, False):
        r = Swpc3D(p, medium_on_device=True)

        def steps(it0):
            if graphs:
                r.run(it0, 20)
            else:
                for it in range(it0, it0 + 20):
                    r.step(it)
        steps(1)
        if what == "green_store":
            r.green_store_setup([10, 20], [9, 21], [8, 12])
        else:
            xi = np.full((p.ny + 6, p.nx + 6, p.nz + 6), 0.05, np.float32)
            r.medium.__init__(r.lib, r.ctx, p, xi)
        steps(21)
        out.append([r.waveforms(), r.download(_lib.F_VZ)] + ([r.green_functions()] if what == "green_store" else []))
        r.close()
    for a, b in zip(*out):
        assert np.abs(b).max() > 0 and _same(a, b)


def _column(p, ks, i, j=None):
    """One source per entry of ks, all in the column (i, j)."""
    out = []
    for n, k in enumerate(ks):
        m = np.random.default_rng(n).uniform(-1, 1, 6)
        y = p.ybeg + (j - 0.5) * p.dy if j else 0.0
        out.append(Source(p.xbeg + (i - 0.5) * p.dx, y, p.zbeg + (k - 0.5) * p.dz, 0.0, 0.3, mo=1e15, mxx=m[0],
                          myy=m[1], mzz=m[2], myz=m[3], mxz=m[4], mxy=m[5]))
    return out


# a fault from bottom to top, one whose subfaults share cells, and one with a cell of many sources between single ones
@pytest.mark.parametrize("ks", [list(range(90, 6, -3)), list(range(8, 60)) * 2, [70, 9] + [30] * 9 + [31, 12]])
def test_long_source_columns(ks):
    """Columns with many sources, in any order of depth, give the bits of the
    injection launch."""
    p = small3d(nx=33, ny=29, nz=96, na=4, nt=12)
    p.sources = _column(p, ks, 17, 15)
    q = small2d("psv", nx=64, nz=96, na=4, nt=12)
    q.sources = _column(q, ks, 30)
    out = []
    for flat in (False, True):
        r, s = Swpc3D(p, medium_on_device=True), Swpc2D(q, "psv")
        if flat:
            for g, a, b in ((r, (2, 2, 1), (4, 2, 2)), (s, (1, 1, 1), (1, 1, 1))):
                check(g.ctx, g.lib.swpc_set_launch(g.ctx, 0, *a))
                check(g.ctx, g.lib.swpc_set_launch(g.ctx, 1, *b))
        r.run(1, p.nt)
        s.run(1, q.nt)
        out.append([r.waveforms(), s.waveforms()] + [r.download(f) for f in range(9)] +
                   [s.download(f) for f in s.field_ids.values()])
        r.close()
        s.close()
    assert np.abs(out[0][2]).max() > 0
    for a, b in zip(*out):
        assert _same(a, b)


def test_a_long_source_column_does_not_hold_the_step_back():
    """Forty subfaults in one column cost no more than the same forty spread
    over the grid, to a quarter of the step (walking the column's entries one
    after another took the whole step again)."""
    p = small3d(nx=96, ny=96, nz=160, na=8, nt=400)
    spread = [s for n in range(40) for s in _column(p, [10 + 3 * n], 20 + 7 * n % 56, 20 + 11 * n % 56)]
    best = []
    for sources in (spread, _column(p, [10 + 3 * n for n in range(40)], 30, 30)):
        p.sources = sources
        r = Swpc3D(p, medium_on_device=True)
        r.run(1, 40)
        best.append(min(r.time_steps(41 + 40 * n, 40) for n in range(7)))
        r.close()
    assert best[1] <= 1.25 * best[0], best


# every staged tile a single FP32 run takes by default (four planes on larger grids, two on small ones), and mixed
@pytest.mark.parametrize("nm", [3, 2, 1, 0])
@pytest.mark.parametrize("mode", ["glut", "force", "green"])
@pytest.mark.parametrize("sbj,vbj", [(4, 4), (2, 2), (4, 2)])
def test_staged_tiles_against_the_flat_kernels(sbj, vbj, mode, nm):
    """Stress and velocity tiles of four and of two planes, with the sources
    inside the launches and any number of memory variables, give the bits of
    the one-cell kernels; tiles partial in k, i and j."""
    p = small3d(nx=42, ny=39, nz=45, na=6, nt=14, nm=nm, sw_wav_u=True, bf_mode=mode == "force",
                green_mode=mode == "green", green_trise=0.3)
    p.sources = _sources(p, 30, 11, 1.0)
    out = []
    for flat in (False, True):
        r = Swpc3D(p, medium_on_device=True)
        if mode == "green":
            r.record(what=_lib.WAV_V | _lib.WAV_U)
        for kernel, bj in ((0, 1), (1, 1)) if flat else ((5, sbj), (6, vbj)):
            check(r.ctx, r.lib.swpc_set_launch(r.ctx, kernel, *((2, 2, 1) if flat else (1, 4, bj))))
        r.run(1, p.nt)
        out.append([r.waveforms(w) for w in (_lib.WAV_V, _lib.WAV_U)] + [r.download(f) for f in range(9)] +
                   [r.download(_lib.F_R + 3 * c + m) for c in range(6) for m in range(nm)] +
                   [r.download(_lib.F_AUX + q) for q in range(18)])
        r.close()
    assert np.abs(out[0][2]).max() > 0
    for a, b in zip(*out):
        assert _same(a, b)
