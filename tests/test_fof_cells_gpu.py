"""Linking by SOD cells (boxes of at least 2^18 particles) where its classes
meet: cells of 16 / 17, 64 / 65 and 512 / 513 records next to one another and
across the box edge, linking lengths on both sides of the table limit, a single
particle in the last cell (filed under another cell by the run scan).  The
groups are compared with the connected components of the friend pairs within
the linking length (scipy KD-tree, FP64; the boxes keep clear of pairs within
1e-6 of it by construction of the test's tolerance check)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from psod_b200.sod import SphericalOverdensity  # noqa: E402

NX = 64


def partition(pos, b):
    """Component label (lowest member index) of every particle; None where a
    pair lies too near the linking length for FP32 and FP64 to agree."""
    from scipy.sparse import coo_matrix
    from scipy.sparse.csgraph import connected_components
    from scipy.spatial import cKDTree

    ll = float(np.float32(b) / np.float32(NX))
    tree = cKDTree(pos.astype(np.float64), boxsize=1.0)
    out = []
    for f in (1 - 2e-6, 1 + 2e-6):
        p = tree.query_pairs(ll * f, output_type="ndarray")
        n = len(pos)
        _, lab = connected_components(coo_matrix((np.ones(len(p)), (p[:, 0], p[:, 1])), shape=(n, n)), directed=False)
        first = np.full(lab.max() + 1, n)
        np.minimum.at(first, lab, np.arange(n))
        out.append(first[lab])
    return out[0] if np.array_equal(out[0], out[1]) else None


def blocks(rng):
    """A sparse background, and a row of neighbouring cells whose record counts
    straddle every class, once inside the box and once across its edge."""
    counts = [16, 17, 64, 65, 512, 513, 17, 513, 16, 64]
    parts = [rng.random((NX**3 - 2 * sum(counts) - 1, 3))]
    parts[0] = parts[0][~np.all(parts[0] > 1 - 1 / NX, axis=1)]  # the last cell holds one particle
    for base in ((20, 20, 20), (NX - 5, NX - 1, 0)):
        for k, m in enumerate(counts):
            cell = np.array(base) + np.array([k % 5, (k // 5), 0])
            parts.append(((cell + rng.random((m, 3))) % NX) / NX)
    parts.append(np.full((1, 3), 1 - 0.3 / NX))
    pos = np.concatenate(parts)
    pad = rng.random((NX**3 - len(pos), 3)) * (1 - 1 / NX)
    pos = np.concatenate([pos, pad])
    pos = np.minimum(pos[rng.permutation(len(pos))].astype(np.float32), np.float32(1 - 2**-24))
    return pos


@pytest.mark.parametrize("b", [0.45, 0.25, 0.2, 0.15, 0.14])
def test_groups_where_cell_classes_meet(b):
    for seed in range(20):
        pos = blocks(np.random.default_rng(seed))
        want = partition(pos, b)
        if want is not None:
            break
    ids = np.arange(len(pos), dtype=np.int64)
    with SphericalOverdensity(NX) as s:
        s.load(pos, ids)
        st = s.fof(percolation=b, mmin=1, nres=NX)
        t = s.fof_halos()
    got = np.empty(len(pos), np.int64)
    got[t.member_index] = np.repeat(t.halo_id, t.halo_mass)  # the ID of the lowest-index member
    assert st["ngroups"] == len(np.unique(want))
    assert np.array_equal(got, want)
