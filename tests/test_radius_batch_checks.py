"""radius() with batch vectors: which calls take their points in place, and what calls with too few supports
or with batch ids at the end of int64 do."""
import numpy as np
import pytest
import torch

from torchcompactradius_b200.batched import _one_each


@pytest.mark.parametrize("support,one", [(None, True), (torch.rand(5), True), (torch.rand(5, 1), True), (torch.rand(4), False),
                                         (torch.rand(6), False), (torch.tensor(0.1), False), (0.1, False),
                                         (np.full(5, 0.1, np.float32), False)])
def test_points_stay_in_place_only_with_a_support_each(support, one):
    x, batch = torch.rand(5, 3), torch.zeros(5, dtype=torch.long)
    assert _one_each(x, batch, support) is one
    assert not _one_each(x, batch[:4], support) and not _one_each(x, batch[:, None], support)


@pytest.mark.gpu
@pytest.mark.parametrize("same", [True, False])
@pytest.mark.parametrize("short", ["first", "second", "numpy", "number", "scalar"])
def test_too_few_supports_are_refused(same, short):
    import torchcompactradius_b200 as tcr
    n = 300
    x = torch.rand(n, 3).cuda()
    batch = torch.arange(3).repeat_interleave(100).cuda()
    h, few = torch.full((n,), 0.1).cuda(), torch.full((n - 50,), 0.1).cuda()
    support = dict(first=(few, h), second=(h, few), numpy=(h, np.full(n - 50, 0.1, np.float32)), number=(0.1, 0.1),
                   scalar=(h, torch.tensor(0.1)))[short]
    with pytest.raises(ValueError):
        tcr.radius(x, None if same else x.clone(), support, batch, batch, mode="symmetric")


@pytest.mark.gpu
@pytest.mark.parametrize("last", [2 ** 62, 2 ** 63 - 3, 2 ** 63 - 2, 2 ** 63 - 1])
def test_ids_at_the_end_of_int64(last):
    import torchcompactradius_b200 as tcr
    g = torch.Generator().manual_seed(1)
    x = torch.rand(400, 3, generator=g).cuda()
    low = torch.arange(2).repeat_interleave(200)
    i, j = tcr.radius(x, None, 0.2, low.cuda())
    a, b = tcr.radius(x, None, 0.2, (low + (last - 1)).cuda())
    assert i.numel() > 400 and torch.equal(i, a) and torch.equal(j, b)


@pytest.mark.gpu
def test_numpy_and_longer_supports_are_taken():
    import torchcompactradius_b200 as tcr
    g = torch.Generator().manual_seed(2)
    x, h = torch.rand(400, 3, generator=g).cuda(), 0.1 + 0.1 * torch.rand(400, generator=g)
    batch = torch.arange(4).repeat_interleave(100).cuda()
    i, j = tcr.radius(x, None, (h.cuda(), h.cuda()), batch, mode="symmetric")
    longer = torch.cat([h, torch.full((7,), 9.0)]).cuda()
    for other in (h.numpy(), longer):
        a, b = tcr.radius(x, None, (h.cuda(), other), batch, mode="symmetric")
        assert torch.equal(i, a) and torch.equal(j, b)
