"""Distances across the periodic boundary from centres whose coordinates are
tiny: the rounded minimum-image form (nx - |x - xc|) and a plain difference of
shifted coordinates differ in the last bits there, and the device seed loop
gives the former, as the host rounds and the oracle do."""

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


def edge_halos(nx, seed):
    """Clumps on the faces x = 0: cores with x below 1e-8 of a cell, members on
    both sides; one core at exactly 0 and one at exactly 1; a denser ball first."""
    rng = np.random.default_rng(seed)
    parts = [lattice_points(nx) / nx]
    for k, at in enumerate([(4.2, 4.3), (4.4, 14.1), (14.3, 4.6), (14.5, 14.2)]):
        core = np.array([0.0, *at]) + rng.normal(size=(60, 3)) * [0, 0.01, 0.01]
        core[:, 0] = rng.random(60) * 1e-8
        if k == 2:
            core[:, 0] = 0.0
        if k == 3:
            core[:, 0] = nx
        halo = np.array([0.0, *at]) + rng.normal(size=(80, 3)) * 0.25
        halo[:, 0] = np.mod(halo[:, 0], nx)
        parts += [core / nx, halo / nx]
        parts.append((np.array([nx - 3.5, *at]) + rng.normal(size=(600, 3)) * 0.2) / nx)
    pos = np.concatenate(parts).astype(np.float32)
    return pos[rng.permutation(len(pos))], np.arange(len(pos), dtype=np.int64)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("nx", [18, 21, 24])
def test_edge_centres(oracle, nx, mode):
    for seed in range(4):
        pos, ids = edge_halos(nx, seed)
        kw = dict(nmin=10, nbins=6, ncut=3, delta=100.0)
        r = oracle.run(oracle.Params(nx=nx, **kw), pos, ids, oracle.CANONICAL)
        assert r.status == 0
        for tuning in ({}, dict(tail_max_ready=0)):
            with SphericalOverdensity(nx, mode=mode, **kw) as s:
                s.set_tuning(**tuning)
                s.load(pos, ids)
                st = s.run()
                t = s.halos()
            assert (st["tail_rounds"] > 0) == (not tuning) and t.nhalo >= 7
            for f in FIELDS:
                assert np.array_equal(getattr(t, f), getattr(r, f)), (f, tuning)
