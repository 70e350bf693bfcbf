"""The record expansion at the edges of its windows, shares and table, against the C oracle (whole
numbers: no tolerance)."""
import numpy as np
import pytest
import torch

import cases
from helpers import coo_arrays, csr_rows, gpu_search
from oracle import compact

pytestmark = pytest.mark.gpu


def cloud(nq, nr, spread, seed):
    """nq queries in one cell and nr references around it, all of them hits when spread is small."""
    rng = np.random.default_rng(seed)
    xq = rng.uniform(0.05, 0.15, (nq, 3)).astype(np.float32)
    xr = (0.1 + rng.uniform(-spread, spread, (nr, 3))).astype(np.float32)
    return xq, np.full(nq, 0.2, np.float32), xr, np.full(nr, 0.2, np.float32)


@pytest.mark.parametrize("nq", [1, 2, 3, 15, 16, 17, 31, 32, 33])
@pytest.mark.parametrize("nr", [1, 32, 33, 129, 511, 512, 513, 1100])
@pytest.mark.parametrize("spread", [0.04, 0.29])  # every pair a hit (windows shrink to fit the table); one in ten
def test_windows_and_shares(nq, nr, spread):
    xq, hq, xr, hr = cloud(nq, nr, spread, nq * 2000 + nr)
    box = ([-1.0] * 3, [1.0] * 3, [False] * 3)
    o = compact.radius_search(xq, hq, xr, hr, *box, "gather", 4096)
    for fmt, pairs in (("coo", coo_arrays), ("csr", csr_rows)):
        adj = gpu_search(xq, hq, xr, hr, *box, "gather", 4096, fmt)
        row, col = pairs(adj)
        assert np.all(np.diff(row) >= 0)
        got, want = cases.canonical(row, col), cases.canonical(o.row, o.col)
        np.testing.assert_array_equal(got[0], want[0])
        np.testing.assert_array_equal(got[1], want[1])


@pytest.mark.parametrize("n", [1, 40, 700])
def test_composed_ids(n):
    """radius with shuffled batch vectors: columns and rows go through the callers' ids."""
    import torchcompactradius_b200 as tcr
    g = torch.Generator().manual_seed(n)
    x = torch.rand(n, 3, generator=g)
    batch = torch.randint(0, 3, (n,), generator=g)
    i, j = tcr.radius(x.cuda(), None, 0.2, batch.cuda())
    d = (x[:, None].double() - x[None].double()).norm(dim=2)
    want = ((d < 0.2) & (batch[:, None] == batch[None])).nonzero()
    near = ((d - 0.2).abs() < 1e-6).any()
    assert not near, "the draw must not put a pair at the threshold"
    got = torch.stack([i, j], 1).cpu()
    got = got[(got[:, 0] * n + got[:, 1]).argsort()]
    assert torch.equal(got, want)
