"""tcr_f64_prepare against the torch operations it stands for (bit for bit)."""
import math

import pytest
import torch

from torchcompactradius_b200.search64 import prepare64, wrap64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,mask", [(1, 1), (2, 0), (2, 2), (3, 5), (3, 7)])
@pytest.mark.parametrize("n,m", [(1, 1), (255, 257), (5000, 20001)])
@pytest.mark.parametrize("self_search", [True, False])
def test_wraps_copies_and_maxima(dim, mask, n, m, self_search):
    g = torch.Generator().manual_seed(n + dim)
    lo, hi = [-1.0, -0.5, 0.1][:dim], [1.0, 0.75, 2.0][:dim]
    xq = ((torch.rand(n, dim, generator=g, dtype=torch.float64) - 0.5) * 9).cuda()
    xr = xq if self_search else ((torch.rand(m, dim, generator=g, dtype=torch.float64) - 0.5) * 9).cuda()
    xq[0] = torch.tensor(lo, dtype=torch.float64)
    hq = torch.rand(n, generator=g, dtype=torch.float64).cuda()
    hr = hq if self_search else torch.rand(m, generator=g, dtype=torch.float64).cuda()
    xq_w, xq_f, hq_f, xr_w, xr_f, hr_f, maxima = prepare64(xq, hq, xr, hr, lo, hi, mask, self_search, self_search)
    want_q = wrap64(xq, lo, hi, mask)
    want_r = wrap64(wrap64(xr, lo, hi, mask), lo, hi, mask)
    assert torch.equal(xq_w, want_q) and torch.equal(xr_w, want_r)
    assert torch.equal(xq_f, want_q.float()) and torch.equal(xr_f, want_q.float() if self_search else want_r.float())
    assert torch.equal(hq_f, hq.float()) and torch.equal(hr_f, hr.float())
    assert maxima == [float(want_q.abs().max()), float(want_r.abs().max()), float(hq.max()), float(hr.max())]


def test_nan_and_missing_supports():
    x = torch.rand(100, 2, dtype=torch.float64).cuda()
    h = -torch.rand(100, dtype=torch.float64).cuda()
    out = prepare64(x, h, x, h, [0.0, 0.0], [1.0, 1.0], 0, True, True)
    assert out[6][2] == float(h.max())
    h[7] = float("nan")
    out = prepare64(x, None, x, h, [0.0, 0.0], [1.0, 1.0], 0, True, False)
    assert out[2] is None and math.isinf(out[6][2]) and math.isnan(out[6][3])
