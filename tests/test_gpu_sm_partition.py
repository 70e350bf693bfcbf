"""Searches on a partition of the device's SMs (a green context): the sort's cooperative launch fits what is
there, and the result is the whole device's (whole numbers: no tolerance)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def few_sms():
    from torch.cuda import green_contexts
    if not green_contexts.SUPPORTED:
        pytest.skip("this torch has no green contexts")
    torch.zeros(1, device="cuda")
    try:
        ctx = green_contexts.GreenContext.create(16, 0)
    except RuntimeError as e:
        pytest.skip(f"no SM partition here: {e}")
    return ctx


@pytest.mark.parametrize("n", [3000, 150000])  # one block's sort, and one that takes more blocks than the partition has
def test_search_on_a_partition(few_sms, n):
    import torchcompactradius_b200 as tcr
    g = torch.Generator().manual_seed(n)
    x = torch.rand(n, 3, generator=g).cuda()
    cloud = tcr.PointCloud(x, torch.full((n,), (8 / n) ** (1 / 3)).cuda())
    dom = tcr.DomainDescription(torch.zeros(3), torch.ones(3), torch.tensor([True, False, True]), 3)

    def search():
        adj = tcr.radiusSearch(cloud, mode="gather", domain=dom, algorithm="compact", format="csr")
        torch.cuda.current_stream().synchronize()
        return adj

    whole = search()
    torch.cuda.synchronize()
    few_sms.set_context()
    try:
        part = search()
        indices, indptr = part.indices.cpu(), part.indptr.cpu()
    finally:
        few_sms.pop_context()
    assert torch.equal(indptr, whole.indptr.cpu()) and torch.equal(indices, whole.indices.cpu())
