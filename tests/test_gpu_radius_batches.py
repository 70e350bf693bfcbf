"""radius() with sorted batch vectors (counted by their boundaries) against the same call with the points
shuffled (ordered by a stable sort): the same pairs, whole numbers."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ids", [[0], [0, 1, 2], [3, 5, 9], [-2, 0, 7], [0, 70000]])
@pytest.mark.parametrize("mode", ["gather", "symmetric"])
@pytest.mark.parametrize("two_clouds", [False, True])
def test_sorted_equals_shuffled(ids, mode, two_clouds):
    import torchcompactradius_b200 as tcr
    g = torch.Generator().manual_seed(len(ids))
    n, m = 700, 500
    x, y = torch.rand(n, 3, generator=g).cuda(), torch.rand(m, 3, generator=g).cuda()
    hx, hy = 0.05 + 0.1 * torch.rand(n, generator=g).cuda(), 0.05 + 0.1 * torch.rand(m, generator=g).cuda()
    pick = torch.tensor(ids)
    bx = pick[torch.randint(0, len(ids), (n,), generator=g).sort().values].cuda()
    by = pick[torch.randint(0, len(ids), (m,), generator=g).sort().values].cuda()
    p, q = torch.randperm(n, generator=g).cuda(), torch.randperm(m, generator=g).cuda()
    if two_clouds:
        i, j = tcr.radius(x, y, (hx, hy), bx, by, mode=mode)
        si, sj = tcr.radius(x[p], y[q], (hx[p], hy[q]), bx[p], by[q], mode=mode)
        si, sj = p[si], q[sj]
    else:
        i, j = tcr.radius(x, None, hx, bx, mode=mode)
        si, sj = tcr.radius(x[p], None, hx[p], bx[p], mode=mode)
        si, sj = p[si], p[sj]
    assert i.numel() > 0 and torch.all(bx[i] == (by if two_clouds else bx)[j])
    key, want = (i * n + j).sort().values, (si * n + sj).sort().values
    assert torch.equal(key, want)
    assert torch.all(bx[i][1:] >= bx[i][:-1]) and torch.all(i[1:] >= i[:-1])
