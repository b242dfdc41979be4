"""Device memory that a call takes beyond the arrays it cannot do without: a
size that fits the card keeps fitting."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from psod_b200.sod import SphericalOverdensity  # noqa: E402

NX, SIDE = 64, 192
SLACK = 12 << 20  # scans, flags, allocation granularity


def used():
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def lattice():
    g = (torch.arange(SIDE, device="cuda", dtype=torch.float32) + 0.5) / SIDE
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
