"""Scheduler blocks: odd sides, whose last block of an axis is three cells wide,
and windows of 15 blocks and more a side, which the device seed loop tests
without staging them.  The loop, the host rounds and the oracle give one table;
halos on both sides of the wide blocks and of the periodic boundary."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from psod_b200 import synth  # noqa: E402
from psod_b200.sod import SphericalOverdensity  # noqa: E402

FIELDS = ("halo_id", "halo_mass", "halo_center", "halo_rdelta", "halo_mass2", "halo_profile", "member_offset",
          "member_index")


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("nx,ncut", [(5, 2), (7, 3), (11, 2), (25, 2), (31, 4), (37, 1), (30, 7), (35, 7), (62, 8), (63, 9)])
def test_blocks_of_odd_sides_and_wide_windows(oracle, nx, ncut, mode):
    b = synth.make_box(nx, nmax_halo=max(200, nx * nx // 2), seed=500 + nx)
    pos = np.concatenate([b.pos.numpy(), np.float32([0.0, 0.999, 0.5])[None] + np.zeros((1, 3), np.float32)])
    rng = np.random.default_rng(nx)
    clumps = [c + rng.normal(size=(60, 3)) * 0.15 / nx for c in rng.random((12, 3)) * [1, 1, 4 / nx] - [0, 0, 2 / nx]]
    pos = np.mod(np.concatenate([pos, *clumps]).astype(np.float64), 1.0).astype(np.float32)
    pos[pos >= 1] = 0
    ids = np.arange(len(pos), dtype=np.int64)
    kw = dict(nmin=10, nbins=6, ncut=ncut, nxbuffer=max(ncut, nx // 2))
    r = oracle.run(oracle.Params(nx=nx, **kw), pos, ids, oracle.CANONICAL)
    for tuning in ({}, dict(tail_max_ready=0)):
        with SphericalOverdensity(nx, mode=mode, **kw) as s:
            s.set_tuning(**tuning)
            s.load(pos, ids)
            if r.status != 0:
                with pytest.raises(Exception):
                    s.run()
                continue
            st = s.run()
            t = s.halos()
        assert st["nprocessed"] == r.nprocessed and t.nhalo > 0
        for f in FIELDS:
            assert np.array_equal(getattr(t, f), getattr(r, f)), f
