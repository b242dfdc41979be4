"""Friends-of-friends groups around the particle that the run scan files under
a foreign cell (a single particle in the last cell of the sort order; cell 0
starts at -nxbuffer): friends in the cells below it, a record of the cell that
lists it with the same place inside its cell, cells of every size class there
and beside it, linking by cells and by runs on both sides of the two limits of
the choice.  Groups are compared with the connected components of the friend
pairs (scipy KD-tree, FP64, boxes without pairs within 2e-6 of the linking
length)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from psod_b200.sod import SphericalOverdensity  # noqa: E402


def partition(pos, nx, b):
    from scipy.sparse import coo_matrix
    from scipy.sparse.csgraph import connected_components
    from scipy.spatial import cKDTree

    ll = float(np.float32(b) / np.float32(nx))
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


def lone_box(nx, b, listed, beside, rng):
    """Uniform background; the last cell holds one particle near its lower
    corner, the two cells before it none, the cell before those `listed`
    records, one of them at the same place inside its cell; a friend in the
    cell diagonally below with `beside` records."""
    last = nx - 1
    p = rng.random((nx**3 - listed - beside - 1, 3)) * nx
    c = np.floor(p).astype(int)
    row = (c[:, 1] == last) & (c[:, 2] == last) & (c[:, 0] >= last - 3)
    below = (c == last - 1).all(1)
    p = p[~(row | below)]
    place = np.array([0.03, 0.04, 0.05])
    lone = last + place
    rec = np.array([last - 3, last, last]) + np.concatenate([place[None] + 1e-3, rng.random((listed - 1, 3))])
    near = last - 1 + rng.random((beside, 3))
    near[0] = lone - 0.55 * b  # within b: 0.95 b away, in the cell below on every axis when b > 0.1
    assert (np.floor(near[0]) == last - 1).all()
    p = np.concatenate([p, lone[None], rec, near])
    spare = rng.random((nx**3 - len(p), 3)) * (last - 4)
    p = np.concatenate([p, spare]) - nx // 2
    pos = (np.mod(p, nx) / nx).astype(np.float32)
    pos[pos >= 1] = 0
    pos = pos[rng.permutation(len(pos))]
    cell = np.floor((pos.astype(np.float64) * nx).astype(np.float32) + nx // 2).astype(int) % nx
    key = cell[:, 0] + nx * (cell[:, 1] + nx * cell[:, 2])
    assert np.sum(key == nx**3 - 1) == 1 and np.max(key[key < nx**3 - 1]) == nx**3 - 4
    return pos


# linking cells: k = 9 (0.2), 12 (0.15), 13 (0.14); 64^3 = 2^18 particles
@pytest.mark.parametrize("listed,beside", [(1, 1), (5, 30), (16, 200), (17, 700), (100, 3), (600, 20)])
@pytest.mark.parametrize("nx,b", [(32, 0.2), (64, 0.2), (64, 0.15), (64, 0.14), (32, 0.14)])
def test_groups_around_the_foreign_particle(nx, b, listed, beside):
    for seed in range(20):
        pos = lone_box(nx, b, listed, beside, np.random.default_rng(seed))
        want = partition(pos, nx, b)
        if want is not None:
            break
    ids = np.arange(len(pos), dtype=np.int64)
    with SphericalOverdensity(nx) as s:
        s.load(pos, ids)
        st = s.fof(percolation=b, mmin=1, nres=nx)
        t = s.fof_halos()
    got = np.empty(len(pos), np.int64)
    got[t.member_index] = np.repeat(t.halo_id, t.halo_mass)
    assert st["ngroups"] == len(np.unique(want))
    assert np.array_equal(got, want)
