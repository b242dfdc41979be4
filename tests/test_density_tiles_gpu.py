"""Density and seed order where their passes change path, against the oracle's
canonical arithmetic (fixed-point nodes, a total order of seeds): every value
is equal bit for bit, so no tolerance is involved.

Grids of 9 and 10 cells (below and at the smallest the node tiles take), sides
that are no power of two and no multiple of a tile, a clump that fills one tile
beyond what a CTA deposits alone, empty regions, one zone of several; seeds
whose sort keys agree in runs up to and beyond what the tie pass orders."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from psod_b200 import synth  # noqa: E402
from psod_b200.sod import SphericalOverdensity, select_zone  # noqa: E402


def density(nx, pos, total=0, **kw):
    with SphericalOverdensity(nx, **kw) as s:
        s.load(pos, np.arange(len(pos), dtype=np.int64), npart_total=total)
        s.cic()
        rho = s.cicm1()
        isort, nn = s.tri_cic()
    return rho, isort, nn


def clumped(nx, seed):
    """A synthetic box, a fifth of it moved into a clump half a cell wide and
    one octant emptied; the corners of the box are occupied."""
    pos = synth.make_box(nx, nmax_halo=500, seed=seed).pos.cpu().numpy().copy()
    rng = np.random.default_rng(seed)
    k = len(pos) // 5
    pos[:k] = (0.4 * nx + 0.5 * rng.random((k, 3))) / nx
    out = np.all(pos > 0.55, axis=1)
    pos[out] -= np.float32(0.5)
    pos[-2:] = [[0, 0, 0], [1 - 2**-24, 0, 1 - 2**-24]]
    return np.clip(pos, 0, 1 - 2**-24).astype(np.float32)


@pytest.mark.parametrize("nx", [9, 10, 11, 16, 17, 20, 33, 50])
def test_density_of_any_grid(oracle, nx):
    pos = clumped(nx, nx)
    rho, isort, nn = density(nx, pos)
    assert np.array_equal(rho, oracle.rho(oracle.Params(nx=nx), pos, oracle.CANONICAL))
    want, wn = oracle.tri_cic(rho, oracle.CANONICAL)
    assert nn == wn and np.array_equal(isort[:nn], want[:wn])


@pytest.mark.parametrize("nx,k,zone", [(24, 2, 5), (40, 2, 0), (48, 4, 37)])
def test_density_of_a_zone(oracle, nx, k, zone):
    pos = clumped(nx, nx)
    pos = pos[select_zone(pos, nx, k, zone)]
    kw = dict(nxcpu=k, nzone=zone, ncut=2)
    rho, isort, nn = density(nx, pos, total=nx**3, **kw)
    p = oracle.Params(nx=nx, npart_total=nx**3, **kw)
    assert np.array_equal(rho, oracle.rho(p, pos, oracle.CANONICAL))


@pytest.mark.parametrize("run", [2, 63, 64, 65, 300])
def test_seed_order_of_equal_densities(oracle, run):
    """Clumps of `run` particles at one place each have one density."""
    nx = 32
    rng = np.random.default_rng(run)
    pos = rng.random((nx**3, 3)).astype(np.float32) * np.float32(1 - 2**-23)
    nclump = max(1, min(200, 12000 // run))
    at = rng.choice(nx**3, nclump * run, replace=False)
    # several clumps close together, so that all of them are seeds
    centre = (0.5 + 0.06 * (rng.random((nclump, 3)) - 0.5)).astype(np.float32)
    pos[at] = np.repeat(centre, run, axis=0)
    rho, isort, nn = density(nx, pos)
    want, wn = oracle.tri_cic(rho, oracle.CANONICAL)
    assert nn == wn and np.array_equal(isort[:nn], want[:wn])
