"""The particle that the run scan files under a foreign cell: a single particle
in the last cell of the sort order, whose cells start at xxmin (the last cell
is nx - nxbuffer - 1 on every axis).  Boxes in which it decides a centre, is a
centre, or is a member, with the cell that lists it one to three cells away."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from boxes import lattice_points  # noqa: E402
from psod_b200.sod import SphericalOverdensity  # noqa: E402

FIELDS = ("halo_id", "halo_mass", "halo_center", "halo_rdelta", "halo_mass2", "halo_profile", "member_offset",
          "member_index")


def foreign_box(nx, gap, kind, seed):
    """Cell-centred lattice; a dense ball that is found first; two equal clumps
    in the cell below the last one, one of them with one particle more
    ("tips": the particle in the last cell, next to the other, decides), or one
    clump around it ("centre"); the `gap` cells before the last one are empty."""
    rng = np.random.default_rng(seed)
    last = nx - 1
    lat = lattice_points(nx)
    c = np.floor(lat).astype(int)
    lat = lat[~((c[:, 1] == last) & (c[:, 2] == last) & (c[:, 0] >= last - gap))]
    k = int(rng.integers(30, 60))
    off = rng.normal(size=(k, 3)) * 0.012
    off[:, 1] = np.minimum(off[:, 1], 0.01)
    lone = np.array([last + 0.75, last + 0.03, last + 0.5])
    if kind == "tips":
        a = np.array([last + 0.25, last - 0.015, last + 0.5]) + off
        clump = np.concatenate([a, a + [0.5, 0.0, 0.0], [[last + 0.25, last - 0.15, last + 0.5]]])
    else:
        lone[1] = last + 0.002
        r = np.abs(rng.normal(size=(3 * k, 3))) * 0.05
        clump = lone + r * [0.1, -1.0, 0.1] * np.where(rng.random((3 * k, 3)) < 0.5, 1.0, [-1.0, 1.0, -1.0])
        clump[:, 1] = np.minimum(clump[:, 1], last - 0.004)
    big = np.array([last - 3.5, last - 3.5, last - 2.5]) + rng.normal(size=(600, 3)) * 0.2
    p = np.concatenate([lat, lone[None], clump, big]) - nx // 2  # cell 0 starts at -nxbuffer
    pos = np.mod(p, nx) / nx
    pos = pos.astype(np.float32)
    pos[pos >= 1] = 0
    pos = pos[rng.permutation(len(pos))]
    cell = np.floor((pos.astype(np.float64) * nx).astype(np.float32) + nx // 2).astype(int) % nx
    key = cell[:, 0] + nx * (cell[:, 1] + nx * cell[:, 2])
    assert np.sum(key == nx**3 - 1) == 1 and np.max(key[key < nx**3 - 1]) == nx**3 - 2 - gap
    return pos, np.arange(len(pos), dtype=np.int64) * 3 + 5


def table(nx, pos, ids, tuning=None, **kw):
    with SphericalOverdensity(nx, **kw) as s:
        if tuning:
            s.set_tuning(**tuning)
        s.load(pos, ids)
        s.cic()
        rho = s.cicm1()
        s.tri_cic()
        st = s.spherover()
        return s.halos(), st, rho


CASES = [(12, 1, "tips"), (16, 1, "tips"), (17, 1, "tips"), (17, 2, "tips"), (24, 2, "tips"), (33, 3, "tips"),
         (12, 1, "centre"), (16, 2, "centre"), (24, 1, "centre"), (24, 3, "centre")]


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("nx,gap,kind", CASES)
def test_seed_loop_counts_the_foreign_particle(nx, gap, kind, mode):
    for seed in range(3):
        pos, ids = foreign_box(nx, gap, kind, seed)
        kw = dict(mode=mode, nmin=10, nbins=6, ncut=3, delta=100.0)
        a, sa, _ = table(nx, pos, ids, **kw)
        b, sb, _ = table(nx, pos, ids, dict(tail_max_ready=0), **kw)
        assert sa["tail_rounds"] > 0 and sb["tail_rounds"] == 0 and a.nhalo > 1
        for f in FIELDS:
            assert np.array_equal(getattr(a, f), getattr(b, f)), f


@pytest.mark.parametrize("nx,gap,kind", CASES)
def test_plain_mode_matches_oracle(oracle, nx, gap, kind):
    pos, ids = foreign_box(nx, gap, kind, 7)
    kw = dict(nmin=10, nbins=6, ncut=3, delta=100.0)
    p = oracle.Params(nx=nx, **kw)
    r = oracle.run(p, pos, ids, oracle.CANONICAL)
    t, st, rho = table(nx, pos, ids, **kw)
    assert np.array_equal(rho, oracle.rho(p, pos, oracle.CANONICAL))
    assert st["nprocessed"] == r.nprocessed
    for f in FIELDS:
        assert np.array_equal(getattr(t, f), getattr(r, f)), f


@pytest.mark.parametrize("tuning", [{}, dict(tail_max_ready=0), dict(warp_cross_min_ready=1, tail_max_ready=0)])
@pytest.mark.parametrize("nx,gap,kind", CASES)
def test_batched_crossing_matches_oracle(oracle, nx, gap, kind, tuning):
    """Balls that the particle lies in although the cell that lists it does not
    meet them: by the CTA walk of the loop and of the host rounds, and by the
    warp walk."""
    pos, ids = foreign_box(nx, gap, kind, 11)
    for ncut in (3, 5):
        kw = dict(nmin=10, nbins=6, ncut=ncut, delta=100.0)
        r = oracle.run(oracle.Params(nx=nx, **kw), pos, ids, oracle.CANONICAL)
        t, st, _ = table(nx, pos, ids, tuning, mode=1, **kw)
        assert st["nprocessed"] == r.nprocessed and st["cross_touch"] == r.cross_touch
        for f in FIELDS:
            assert np.array_equal(getattr(t, f), getattr(r, f)), f
