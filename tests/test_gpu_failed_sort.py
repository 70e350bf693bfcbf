"""A build whose sort gave up waiting (its flag, set here in the structure's buffer): the count behind it
finds nothing and reports -1, the emit writes nothing, and a structure whose flag is clear searches as ever."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def cloud(n, seed=0):
    g = torch.Generator().manual_seed(seed)
    return torch.rand(n, 3, generator=g).cuda(), torch.full((n,), (6 / n) ** (1 / 3)).cuda()


@pytest.mark.parametrize("mask", [0, 5])
@pytest.mark.parametrize("self_search", [True, False])
@pytest.mark.parametrize("n", [900, 30000])
@pytest.mark.parametrize("staged", [True, False])
def test_count_and_emit_behind_a_failed_build(mask, self_search, n, staged):
    from torchcompactradius_b200 import _lib
    from torchcompactradius_b200.search import make_desc
    lib = _lib.load()
    (x, h), (y, k) = cloud(n), cloud(n // 2, 1)
    xq, hq = (x, h) if self_search else (y, k)
    nq = len(xq)
    d = make_desc(3, "gather", mask, [0.0] * 3, [1.0] * 3, 4096, xq, hq, x, h, self_search)
    s_bytes, w_bytes = _lib.search_sizes(nq, n, 3)
    st, sc = (torch.empty(b, dtype=torch.uint8, device="cuda") for b in (s_bytes, w_bytes))
    flag = _lib.structure_offsets(n)["num_cells"] + 4
    words = 1 << 22 if staged else 0
    stage = torch.empty(max(words, 1), dtype=torch.int32, device="cuda")
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    at = lambda t: ctypes.c_void_p(t.data_ptr())
    _lib.check(lib.tcr_build_structure(ctypes.byref(d), at(st), s_bytes, at(sc), w_bytes, sp), "build")

    def search(failed):
        st[flag:flag + 4].view(torch.int32).fill_(failed)
        info = torch.zeros(8, dtype=torch.int64, pin_memory=True)
        offsets = torch.full((nq + 1,), -1, dtype=torch.int64, device="cuda")
        row, col = (torch.full((60 * nq,), -1, dtype=torch.int64, device="cuda") for _ in range(2))
        _lib.check(lib.tcr_count(ctypes.byref(d), at(st), at(sc), w_bytes, at(stage) if words else None, words,
                                 at(offsets), None, None, at(info), sp), "count")
        _lib.check(lib.tcr_emit(ctypes.byref(d), at(st), at(sc), w_bytes, at(stage) if words else None, at(offsets),
                                at(row), at(col), len(col), sp), "emit")
        torch.cuda.synchronize()
        return info.tolist(), offsets, row, col

    info, offsets, row, col = search(0)
    total = info[0]
    assert info[1] == 0 and nq < total < len(col)
    bad, off2, row2, col2 = search(1)
    assert bad[0] == 0 and bad[1] == -1 and not off2.any()
    assert bool((row2 == -1).all()) and bool((col2 == -1).all())
    info, off3, row3, col3 = search(0)  # (only the build's flag stays with the structure)
    assert info[0] == total and torch.equal(offsets, off3) and torch.equal(row, row3) and torch.equal(col, col3)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_kept_structure_reports_its_failed_build(dtype):
    import torchcompactradius_b200 as tcr
    x, h = (t.to(dtype) for t in cloud(2000))
    dom = tcr.DomainDescription(torch.zeros(3, dtype=dtype), torch.ones(3, dtype=dtype), torch.tensor([True] * 3), 3)
    adj, ds = tcr.radiusSearch(tcr.PointCloud(x, h), mode="gather", domain=dom, algorithm="compact", format="csr",
                               returnStructure=True)
    flag = ds._buf[ds._off["num_cells"] + 4:ds._off["num_cells"] + 8].view(torch.int32)
    flag.fill_(1)
    with pytest.raises(RuntimeError, match="did not complete"):
        tcr.neighborSearchExisting(tcr.PointCloud(x, h), ds, mode="gather", format="csr")
    flag.fill_(0)
    again = tcr.neighborSearchExisting(tcr.PointCloud(x, h), ds, mode="gather", format="csr")
    assert torch.equal(adj.indptr, again.indptr)


def test_operators_report_a_failed_build():
    from torchcompactradius_b200 import _lib, ops
    ns = ops.load()
    x, h = cloud(2000)
    lo, hi, per = torch.zeros(3), torch.ones(3), torch.tensor([False] * 3)
    s = ns.buildStructure(x, h, x, h, lo, hi, per, 4096, "gather", True)
    flag = _lib.structure_offsets(2000)["num_cells"] + 4
    s[flag:flag + 4].view(torch.int32).fill_(1)
    with pytest.raises(RuntimeError, match="did not complete"):
        ns.radiusSearchWithStructure(s, x, h, x, h, lo, hi, per, 4096, "gather", True)


def test_query_sort_has_its_own_flag():
    """Nothing of a search of new queries is written to the structure it searches."""
    import torchcompactradius_b200 as tcr
    x, h = cloud(30000)
    _, ds = tcr.radiusSearch(tcr.PointCloud(x, h), mode="gather", algorithm="compact", format="csr", returnStructure=True)
    before = ds._buf.cpu().numpy().copy()
    tcr.neighborSearchExisting(tcr.PointCloud(*cloud(20000, 3)), ds, mode="gather", format="csr")
    np.testing.assert_array_equal(ds._buf.cpu().numpy(), before)
