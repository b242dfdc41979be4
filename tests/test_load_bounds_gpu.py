"""psod_load_particles refuses positions outside [0, 1] (not in box units, not
finite) without computing a cell from them, leaves nothing loaded, and the
context takes the next good load as a fresh one does."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from psod_b200 import capi, synth  # noqa: E402
from psod_b200.sod import PsodError, SphericalOverdensity  # noqa: E402

BAD = [50.0, 1000.0, -5.0, 3e38, -3e38, np.inf, -np.inf, np.nan, np.nextafter(np.float32(1), np.float32(2)),
       np.nextafter(np.float32(0), np.float32(-1))]


@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("nx", [8, 24])
def test_positions_outside_the_box(nx, device):
    box = synth.make_box(nx, nmax_halo=nx * 20, seed=nx)
    good = box.pos.numpy().astype(np.float32)
    ids = box.ids.numpy()
    kw = dict(nmin=10, nbins=8, ncut=3)
    with SphericalOverdensity(nx, **kw) as s:
        s.load(good, ids)
        s.cic()
        want = s.cicm1()
    with SphericalOverdensity(nx, **kw) as s:
        for axis in range(3):
            for v in BAD:
                for where in (slice(None), len(good) // 2):  # every particle, a single one
                    pos = good.copy()
                    pos[where, axis] = v
                    with pytest.raises(PsodError) as e:
                        s.load(torch.from_numpy(pos).cuda() if device else pos, ids)
                    assert e.value.status == capi.ERR_ARG
        for call in (s.cic, s.tri_cic):
            with pytest.raises(PsodError) as e:
                call()
            assert e.value.status == capi.ERR_STATE
        s.load(good, ids)
        s.cic()
        assert np.array_equal(s.cicm1(), want)
