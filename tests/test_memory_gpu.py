"""Device memory that a call takes beyond the arrays it cannot do without: a
size that fits the card keeps fitting."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from psod_b200 import capi  # noqa: E402
from psod_b200.sod import SphericalOverdensity  # noqa: E402

NX, SIDE = 64, 192
SLACK = 12 << 20  # scans, flags, allocation granularity


def used():
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def lattice(side=SIDE):
    g = (torch.arange(side, device="cuda", dtype=torch.float32) + 0.5) / side
    z, y, x = torch.meshgrid(g, g, g, indexing="ij")
    return torch.stack([x, y, z], -1).reshape(-1, 3).contiguous()


def test_load_without_dense_cells():
    """27 particles in every cell: no sub-cell tables."""
    pos = lattice()
    n = len(pos)
    ids = torch.arange(n, device="cuda")
    with SphericalOverdensity(NX) as s:
        before = used()
        s.load(pos, ids)
        # cube and slab records (16 bytes), inverse and cell (4 bytes), IDs (8)
        # a particle; counts and starts of the cells
        assert used() - before <= 48 * n + 8 * (NX**3 + 1) + SLACK


def test_seed_order_to_the_host():
    """Every particle a seed: the order goes to a host array, to a device array
    and to an address that is no multiple of 8, none of which takes memory on
    the device."""
    pos = lattice() / 6  # density 216
    n = len(pos)
    ids = torch.arange(n, device="cuda")
    with SphericalOverdensity(NX) as s:
        s.load(pos, ids)
        s.cic()
        _, nn = s.tri_cic(want_isort=False)
        assert nn > n // 2
        dev = torch.zeros(nn, dtype=torch.int64, device="cuda")
        odd = torch.zeros(8 * nn + 4, dtype=torch.uint8, device="cuda")
        before = used()
        host, _ = s.tri_cic()
        for ptr in (dev.data_ptr(), odd.data_ptr() + 4):
            out = C.c_int64(0)
            assert s.lib.psod_tri_cic(s.ctx, C.c_void_p(ptr), C.byref(out)) == capi.OK and out.value == nn
        assert used() - before <= SLACK
        got = [dev.cpu().numpy(), odd[4 : 4 + 8 * nn].cpu().numpy().view(np.int64)]
    assert np.array_equal(np.sort(host), np.sort(np.unique(host))) and len(host) == nn
    for g in got:
        assert np.array_equal(g, host)


def test_linking_by_runs():
    """Fine linking cells: the lists of large cells need no memory of their own."""
    pos = lattice(384)
    n = len(pos)
    ids = torch.arange(n, device="cuda")
    with SphericalOverdensity(2 * NX) as s:
        s.load(pos, ids)
        before = used()
        st = s.fof(percolation=0.14, mmin=2, nres=2 * NX)  # 13 linking cells a cell and axis
        assert st["fine_cells"] == n  # one record each
        # keys (2 + 2 bytes a particle), order, parents, inverse, two work arrays,
        # the runs' heads and list, halo scan, group codes (4 each); memory comes
        # in pieces of 2 MiB, which n fills and the five arrays of n + 1 do not;
        # the rest is small (the lists took 17 MB)
        assert used() - before <= 40 * n + (16 << 20)
