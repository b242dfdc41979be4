"""Boxes that the preselect cube nearly spans: cube cells meet a ball across
the periodic boundary too.  Crossing by a warp and by a CTA, host rounds and
device loop, against the oracle."""

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


def clumps(nx, top, seed):
    """Lattice and clumps of 40 to `top` particles at random places, two of them
    on the box edge."""
    rng = np.random.default_rng(seed)
    parts = [lattice_points(nx)]
    for c in [[0.02, nx / 2, nx - 0.03], [nx / 3, 0.01, 0.02], *(rng.random((4, 3)) * nx)]:
        parts.append(np.asarray(c) + rng.normal(size=(int(rng.integers(40, top)), 3)) * rng.uniform(0.2, 0.7))
    pos = (np.mod(np.concatenate(parts), nx) / nx).astype(np.float32)
    pos[pos >= 1] = 0
    return pos[rng.permutation(len(pos))], np.arange(len(pos), dtype=np.int64)


@pytest.mark.parametrize("tuning", [dict(warp_cross_min_ready=1, tail_max_ready=0), dict(tail_max_ready=0), {}])
@pytest.mark.parametrize("nx,ncut", [(5, 2), (6, 2), (7, 2), (8, 2), (9, 4), (11, 4), (12, 4), (13, 5), (14, 5)])
@pytest.mark.parametrize("top,delta", [(700, 60.0), (90, 12.0), (60, 6.0)])
def test_cube_nearly_spans_the_box(oracle, nx, ncut, top, delta, tuning):
    for seed in range(6):
        pos, ids = clumps(nx, top, 10 * nx + seed)
        kw = dict(nmin=10, nbins=6, ncut=ncut, delta=delta, nxbuffer=max(ncut, nx // 2))
        r = oracle.run(oracle.Params(nx=nx, **kw), pos, ids, oracle.CANONICAL)
        if r.status != 0:
            continue
        with SphericalOverdensity(nx, mode=1, **kw) as s:
            s.set_tuning(**tuning)
            s.load(pos, ids)
            s.run()
            t = s.halos()
        assert t.nhalo == r.nhalo
        for f in FIELDS:
            assert np.array_equal(getattr(t, f), getattr(r, f)), f
