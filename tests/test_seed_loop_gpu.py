"""The device seed loop against the host's rounds (tail_max_ready = 0): the
halo table and the counters that do not depend on the schedule are equal bit
for bit, whatever the order in which ready seeds run.  Boxes where the loop's
parts change: windows that cover the whole axis or wrap, block sides of one
cell (odd grids: windows too large to stage), the list's minimum-image form
below 16 cells, a preselect cube narrower than the list (ncut 1), a particle
filed under a foreign cell, seeds whose records exceed a CTA's list."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from psod_b200 import synth  # noqa: E402
from psod_b200.sod import SphericalOverdensity  # noqa: E402


def host(b):
    return b.pos.cpu().numpy(), b.ids.cpu().numpy()


def lone_last(pos, nx):
    """One particle in the last cell, next to a dense clump: filed under the
    cell before it."""
    p = pos.copy()
    last = np.all(p >= 1 - 1 / nx, axis=1)
    p[last] -= np.float32(1.5 / nx)
    p[0] = 1 - 0.4 / nx
    rng = np.random.default_rng(5)
    k = len(p) // 20
    p[1 : 1 + k] = (1 - 1.2 / nx) + (rng.random((k, 3)) - 0.5) * 0.3 / nx
    return np.minimum(p, np.float32(1 - 2**-24)).astype(np.float32)


def tables(nx, pos, ids, loop, **kw):
    with SphericalOverdensity(nx, **kw) as s:
        if not loop:
            s.set_tuning(tail_max_ready=0)
        s.load(pos, ids)
        s.cic()
        s.tri_cic()
        st = s.spherover()
        t = s.halos()
    assert loop or st["tail_rounds"] == 0
    return t, st


CASES = [
    # nx, largest halo, options
    (8, 300, dict(ncut=2)),
    (9, 300, dict(ncut=3)),
    (12, 500, dict(ncut=3)),
    (16, 800, dict(ncut=1)),
    (21, 800, dict(ncut=5)),
    (24, 1500, dict(ncut=7)),
    (33, 1500, dict(ncut=3)),
    (48, 8000, dict(ncut=5)),
    (64, 20000, dict(ncut=4, delta_extra=(500.0, 178.0))),
]


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("quirk", [False, True])
@pytest.mark.parametrize("nx,nmax,kw", CASES)
def test_loop_matches_host_rounds(nx, nmax, kw, quirk, mode):
    pos, ids = host(synth.make_box(nx, nmax_halo=nmax, seed=100 + nx))
    if quirk:
        pos = lone_last(pos, nx)
    kw = dict(mode=mode, nmin=10, nbins=8, **kw)
    a = tables(nx, pos, ids, True, **kw)
    assert a[1]["tail_rounds"] > 0
    same(a, tables(nx, pos, ids, False, **kw))


@pytest.mark.parametrize("nx,share", [(64, 10), (96, 20)])
def test_heavy_clusters(nx, share):
    """Two clusters of a large part of the box: long chains of seeds, balls and
    lists of every form."""
    pos, ids = host(synth.make_box(nx, nmax_halo=3000, n_clusters=2, cluster_size=nx**3 // share, seed=nx))
    kw = dict(mode=1, nmin=10, nbins=8, ncut=7)
    same(tables(nx, pos, ids, True, **kw), tables(nx, pos, ids, False, **kw))


@pytest.mark.parametrize("count,radius", [(5000, 2.0), (12000, 2.9), (30000, 2.9)])
def test_lists_beyond_shared_memory(count, radius):
    """Overlapping balls with more records within two cells of a seed than a
    CTA's list holds, their refinement shared by the idle CTAs."""
    nx = 32
    c = [[0.3, 0.3, 0.3], [0.3 + 3.0 / nx, 0.3, 0.3], [0.7, 0.7, 0.98]]
    pos, ids = host(synth.ball_box(nx, c, [radius] * 3, [count // 4, count // 4, count // 2], seed=count))
    kw = dict(mode=1, nmin=10, nbins=8, ncut=4, delta=100.0)
    same(tables(nx, pos, ids, True, **kw), tables(nx, pos, ids, False, **kw))


def same(a, b):
    (ta, sa), (tb, sb) = a, b
    assert ta.nhalo > 0
    for f in ta.__dataclass_fields__:
        assert np.array_equal(getattr(ta, f), getattr(tb, f)), f
    for f in ("nprocessed", "touched", "cross_touch", "nmember"):
        assert sa[f] == sb[f], f
