"""Self searches against a kept structure with other supports than it was built from, against the C oracle's
distance test (whole numbers: no tolerance)."""
import numpy as np
import pytest
import torch

import cases
from oracle import compact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,per", [(2, [1, 1]), (2, [0, 1]), (3, [1, 1, 1]), (3, [1, 0, 0])])
@pytest.mark.parametrize("n", [300, 6000])
@pytest.mark.parametrize("odd", ["none", "negative", "zero", "tiny", "nan"])
def test_other_supports_on_a_kept_structure(dim, per, n, odd):
    """The queries' supports of the second call decide (gather), also where they leave the range of the fast
    test, which the structure's own supports did not."""
    from torchcompactradius_b200 import ops
    ns = ops.load()
    rng = np.random.default_rng(n + dim)
    x = rng.uniform(-1, 1, (n, dim)).astype(np.float32)
    h = np.full(n, np.float32(0.5 * (50 / n) ** (1 / dim)))
    h2 = (h * rng.uniform(0.2, 1.0, n)).astype(np.float32)
    some = rng.choice(n, 9, replace=False)
    if odd != "none":
        h2[some] = dict(negative=-h[some], zero=0.0, tiny=1e-20, nan=np.nan)[odd]
    lo, hi, pt = torch.full((dim,), -1.0), torch.full((dim,), 1.0), torch.tensor([bool(p) for p in per])
    xt, ht = torch.tensor(x).cuda(), torch.tensor(h).cuda()
    s = ns.buildStructure(xt, ht, xt, ht, lo, hi, pt, 4096, "gather", True)
    ht.copy_(torch.tensor(h2))
    r, c, _ = ns.radiusSearchWithStructure(s, xt, ht, xt, ht, lo, hi, pt, 4096, "gather", True)
    o = compact.brute_force(x, h2, None, None, [-1.0] * dim, [1.0] * dim, [bool(p) for p in per], "gather")
    got, want = cases.canonical(r.cpu().numpy(), c.cpu().numpy()), cases.canonical(o.row, o.col)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])
