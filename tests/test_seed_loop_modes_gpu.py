"""The device seed loop where its less common parts run, each case asserting
that it ran there: seeds whose records exceed a CTA's list, the learned mode,
and sample collection.  Table and samples are those of the host rounds."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from psod_b200 import synth  # noqa: E402
from psod_b200.sod import SphericalOverdensity  # noqa: E402

FIELDS = ("halo_id", "halo_mass", "halo_rank", "halo_center", "halo_rdelta", "halo_mass2", "halo_profile",
          "member_offset", "member_index")
LIST = 4096  # records that a CTA's list holds


def run(nx, pos, ids, loop, collect=0, model=None, **kw):
    with SphericalOverdensity(nx, **kw) as s:
        if not loop:
            s.set_tuning(tail_max_ready=0)
        if model is not None:
            s.learn_set_model(model)
        if collect:
            s.learn_collect(collect)
        s.load(pos, ids)
        st = s.run()
        t = s.halos()
        x = s.learn_samples() if collect else None
        if collect and model is None:
            s.learn_train(epochs=5, batch=256, lr=1e-3, seed=1)
            model = s.learn_get_model()
    assert (st["tail_rounds"] > 0) == loop
    return t, st, x, model


def same(a, b):
    assert a.nhalo > 0
    for f in FIELDS:
        assert np.array_equal(getattr(a, f), getattr(b, f)), f


def boxes():
    for nx, share in ((64, 10), (96, 20)):
        b = synth.make_box(nx, nmax_halo=3000, n_clusters=2, cluster_size=nx**3 // share, seed=nx)
        yield nx, b.pos, b.ids, dict(ncut=7)
    for count, seed in ((30000, 30000), (28000, 6)):
        nx = 32
        c = [[0.3, 0.3, 0.3], [0.3 + 3.0 / nx, 0.3, 0.3], [0.7, 0.7, 0.98]]
        b = synth.ball_box(nx, c, [2.9] * 3, [count // 4, count // 4, count // 2], seed=seed)
        yield nx, b.pos, b.ids, dict(ncut=4, delta=100.0)


@pytest.mark.parametrize("mode", [0, 1])
def test_seeds_beyond_a_list(mode):
    for nx, pos, ids, kw in boxes():
        kw = dict(mode=mode, nmin=10, nbins=8, **kw)
        a, sa, *_ = run(nx, pos, ids, True, **kw)
        b, sb, *_ = run(nx, pos, ids, False, **kw)
        same(a, b)
        # a halo of more members than a list holds was made by the loop: more
        # members than all smaller halos have together
        small = a.halo_mass[a.halo_mass <= LIST].sum()
        assert sa["tail_members"] > min(small, LIST), (nx, sa["tail_members"], small)
        for f in ("nprocessed", "touched", "cross_touch", "nmember"):
            assert sa[f] == sb[f], f


def test_learned_mode_and_samples():
    """Samples and learned balls of both schedules (window of 8 cells: every
    seed within the features' reach of 4 is resolved in rank order)."""
    for nx, seed, kw in ((64, 3, dict(ncut=4)), (75, 4, dict(ncut=5))):
        b = synth.make_box(nx, nmax_halo=20000, n_clusters=1, cluster_size=20000, seed=seed)
        kw = dict(nmin=10, nbins=8, **kw)
        a, _, xa, model = run(nx, b.pos, b.ids, True, collect=1 << 18, mode=1, **kw)
        h, _, xh, _ = run(nx, b.pos, b.ids, False, collect=1 << 18, mode=1, **kw)
        same(a, h)
        rows = [np.concatenate(v, axis=1) for v in (xa, xh)]
        rows = [r[np.lexsort(r.T)] for r in rows]
        assert len(rows[0]) > 100 and np.array_equal(rows[0], rows[1])
        for loop in (True, False):
            t, *_ = run(nx, b.pos, b.ids, loop, model=model, mode=2, **kw)
            same(t, a)
        t, _, xl, _ = run(nx, b.pos, b.ids, True, collect=1 << 18, model=model, mode=2, **kw)
        same(t, a)
        r = np.concatenate(xl, axis=1)
        assert np.array_equal(r[np.lexsort(r.T)], rows[0])
