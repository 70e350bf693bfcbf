"""The count walk's tensor-core test at the edges of its tiles, chunks, windows and band, against the C
oracle (pair sets are whole numbers: no tolerance)."""
import numpy as np
import pytest

import cases
from helpers import csr_rows, gpu_search
from oracle import compact

pytestmark = pytest.mark.gpu


def check(xq, hq, xr, hr, lo, hi, per, mode):
    o = compact.radius_search(xq, hq, xr, hr, lo, hi, per, mode, 4096)
    adj = gpu_search(xq, hq, xr, hr, lo, hi, per, mode, 4096, "csr")
    np.testing.assert_array_equal(adj.rowEntries.cpu().numpy(), o.counts)
    got, want = cases.canonical(*csr_rows(adj)), cases.canonical(o.row, o.col)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])
    return len(want[0])


@pytest.mark.parametrize("mode", cases.MODES)
@pytest.mark.parametrize("nq,nr", [(1, 1), (7, 31), (8, 32), (9, 33), (16, 63), (17, 64), (24, 65), (25, 1023), (31, 1024),
                                   (32, 1025), (33, 2100)])
def test_tiles_and_windows(mode, nq, nr):
    """Queries of one cell (the product's tiles of 8, units of 32) against references around it (chunks
    of 32, pairs of chunks, windows of 1024)."""
    rng = np.random.default_rng(100 * nq + nr)
    xq = rng.uniform(0.01, 0.19, (nq, 3)).astype(np.float32)
    xr = rng.uniform(-0.19, 0.39, (nr, 3)).astype(np.float32)
    hq = rng.uniform(0.1, 0.2, nq).astype(np.float32)
    hr = rng.uniform(0.1, 0.2, nr).astype(np.float32)
    hq[0] = hr[0] = 0.2
    check(xq, hq, xr, hr, [-1.0] * 3, [1.0] * 3, [False] * 3, mode)


@pytest.mark.parametrize("mode", cases.MODES)
@pytest.mark.parametrize("dim,per,side", [(1, [1], 64), (2, [0, 0], 40), (2, [1, 1], 32), (3, [0, 0, 0], 14), (3, [1, 0, 1], 16)])
def test_lattice_at_the_threshold(mode, dim, per, side):
    """Lattice points whose distances equal the support: most queries have pairs inside the band (more
    than the band list holds in three dimensions)."""
    d = np.float32(2.0 / side)
    c = -1 + d * (np.arange(side, dtype=np.float32) + np.float32(0.5))
    x = np.stack(np.meshgrid(*[c] * dim, indexing="ij"), -1).reshape(-1, dim).astype(np.float32)
    for reach in (1.0, 2.0 ** 0.5, 2.0):
        h = np.full(len(x), np.float32(d * np.float32(reach)))
        assert check(x, h, None, None, [-1.0] * dim, [1.0] * dim, [bool(p) for p in per], mode) >= len(x)


@pytest.mark.parametrize("mode", cases.MODES)
@pytest.mark.parametrize("cells", [2, 3, 4, 5, 6, 9])
@pytest.mark.parametrize("dim,per", [(2, [1, 1]), (3, [1, 0, 1])])
def test_few_periodic_cells(mode, cells, dim, per):
    """Periodic domains of a few cells: candidates across the seam are shifted from four cells on."""
    rng = np.random.default_rng(cells + 10 * dim)
    n = 900
    x = rng.uniform(-1, 1, (n, dim)).astype(np.float32)
    h = (rng.uniform(0.6, 1.0, n) * (2.0 / cells - 1e-3)).astype(np.float32)
    h[0] = np.float32(2.0 / cells - 1e-3)
    check(x, h, None, None, [-1.0] * dim, [1.0] * dim, [bool(p) for p in per], mode)


@pytest.mark.parametrize("mode", cases.MODES)
def test_far_domain_and_tiny_supports(mode):
    """A domain far from the origin (few bits left in the cell), and supports much smaller than the cell."""
    rng = np.random.default_rng(5)
    x = (1000 + rng.uniform(0, 2, (4000, 3))).astype(np.float32)
    h = rng.uniform(0.1, 0.2, 4000).astype(np.float32)
    check(x, h, None, None, [1000.0] * 3, [1002.0] * 3, [False] * 3, mode)
    check(x, h, None, None, [1000.0] * 3, [1002.0] * 3, [True, False, True], mode)
    h = (10.0 ** rng.uniform(-3, -0.7, 4000)).astype(np.float32)
    y = rng.uniform(-1, 1, (4000, 3)).astype(np.float32)
    check(y, h, None, None, [-1.0] * 3, [1.0] * 3, [False] * 3, mode)


@pytest.mark.parametrize("mode", ["gather", "superSymmetric"])
@pytest.mark.parametrize("per", [[0, 0, 0], [1, 1, 0]])
@pytest.mark.parametrize("h,outside", [(0.3, False), (0.02, False), (0.002, False), (0.3, True), (0.02, True)])
def test_cell_maps(mode, per, h, outside):
    """Grids of fewer and of more cells than the map has slots, and points outside a non-periodic domain:
    cells found in place and through the open-addressing table."""
    rng = np.random.default_rng(int(1000 * h))
    n = 1500
    x = rng.uniform(-1, 1, (n, 3)).astype(np.float32)
    x[: n // 2] = x[0] + rng.uniform(-2 * h, 2 * h, (n // 2, 3)).astype(np.float32)  # some neighbours in any case
    x = np.clip(x, -1, 0.9999).astype(np.float32)
    if outside:
        x[:5, 2] += np.float32(3.0)
    hs = rng.uniform(0.7 * h, h, n).astype(np.float32)
    assert check(x, hs, None, None, [-1.0] * 3, [1.0] * 3, [bool(p) for p in per], mode) > n
