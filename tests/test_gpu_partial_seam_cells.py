"""Periodic dimensions of four cells whose last cell is partial: the candidates a query meets across the
seam, with supports up to and above the cell size (a kept structure searched with other supports).  Against
the C oracle's distance test, restricted to the stencil of the structure's grid (whole numbers: no tolerance)."""
import numpy as np
import pytest
import torch

import cases
from oracle import compact

pytestmark = pytest.mark.gpu


def expected(xq, hq, xr, hcell, hi, per, mode):
    """Pairs within the support whose reference lies in the 3^d stencil of the query's cell."""
    o = compact.brute_force(xq, hq, xr, np.full(len(xr), 0.1, np.float32), [0.0] * len(hi), hi, per, mode)
    keep = np.ones(len(o.row), bool)
    for d, e in enumerate(hi):
        n = int(np.ceil(np.float32(e) / np.float32(hcell)))
        cq, cr = ((x[:, d] / np.float32(hcell)).astype(np.int64) for x in (xq, xr))
        step = np.abs(cq[o.row] - cr[o.col])
        keep &= (np.minimum(step, n - step) if per[d] else step) <= 1
    return o.row[keep], o.col[keep]


@pytest.mark.parametrize("short", [0.55, 0.6, 0.625, 0.65, 0.9, 0.95])
@pytest.mark.parametrize("reach", [0.9, 1.1, 1.4, 1.5, 1.9])
def test_kept_structure_on_four_cells(short, reach):
    """Box 1 x short: the short side sets the cell size, so that the periodic side holds 3 to 4 of them."""
    import torchcompactradius_b200 as tcr
    rng = np.random.default_rng(int(1000 * short))
    hi, per = [1.0, short], [True, False]
    h0 = np.float32(0.2499)
    hcell, count = compact.compute_hcell([0.0, 0.0], hi, h0)
    assert count[0] == 4
    xr = (rng.uniform(0.001, 0.999, (400, 2)) * hi).astype(np.float32)
    xq = (rng.uniform(0.001, 0.999, (400, 2)) * hi).astype(np.float32)
    xr[0], xq[0] = [0.596, 0.3], [0.002, 0.3]
    dom = tcr.DomainDescription(torch.zeros(2), torch.tensor(hi), torch.tensor(per), 2)
    _, ds = tcr.radiusSearch(tcr.PointCloud(torch.tensor(xr).cuda(), torch.full((len(xr),), float(h0)).cuda()), None,
                             mode="gather", domain=dom, algorithm="compact", returnStructure=True)
    hq = np.full(len(xq), np.float32(reach * hcell))
    adj = tcr.neighborSearchExisting(tcr.PointCloud(torch.tensor(xq).cuda(), torch.tensor(hq).cuda()), ds,
                                     mode="gather", format="coo")
    got = cases.canonical(adj.row.cpu().numpy(), adj.col.cpu().numpy())
    want = cases.canonical(*expected(xq, hq, xr, hcell, hi, per, "gather"))
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])
