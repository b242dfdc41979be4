"""Potential pass of psod_halo_properties at the edges of its work items
(256 members, two a thread) and of its staged tiles: halos one member below,
at and above them, with the full and the sampled potential.  Each member's
potential sum runs over the others in the oracle's order with terms within
an ulp of its rounded root and quotient, so the most bound member is the
same and the real(4) energies agree to two real(4) roundings (1.2e-7 each)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from psod_b200.sod import SphericalOverdensity  # noqa: E402
from tests.test_props_gpu import UNITS  # noqa: E402

SIZES = [20, 127, 128, 129, 255, 256, 257, 384, 511, 512, 513, 769, 1024, 1100]


@pytest.mark.parametrize("threshold", [30000, 1024, 2570])
def test_potential_at_tile_edges(oracle, threshold):
    rng = np.random.default_rng(17)
    g = (np.arange(3) + 0.5) / 3
    centres = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)[: len(SIZES)]
    # gaussian clumps a tenth of the linking length wide: each is one group
    pos = np.concatenate([c + rng.normal(0, 0.02 / 32, (m, 3)) for c, m in zip(centres, SIZES)])
    pos = pos[rng.permutation(len(pos))].astype(np.float32)
    vel = rng.normal(0, 0.3, pos.shape).astype(np.float32)
    ids = rng.permutation(len(pos)).astype(np.int64)
    with SphericalOverdensity(32) as s:
        s.load(pos, ids, vel=vel)
        s.fof(percolation=0.2, mmin=20, nres=32)
        t = s.fof_halos()
        got, _ = s.halo_properties(**UNITS, source="fof", epot_threshold=threshold)
    assert sorted(t.halo_mass.tolist()) == sorted(SIZES)
    want = oracle.halo_properties(t.member_offset, t.member_index, pos, vel, **UNITS, epot_threshold=threshold)
    assert np.array_equal(got["center_pot"], want["center_pot"])
    for f in ("epot", "lambda"):
        assert np.allclose(got[f], want[f], rtol=2.4e-7, atol=0), f
    for f in ("dens", "dens_int", "vcirc", "dens178", "dens_int178", "circ", "delta_vals"):
        assert np.allclose(got[f], want[f], rtol=2.4e-7, atol=1e-30, equal_nan=True), f
