"""Rows and columns written through the caller's ids: int32 values of either sign, whether a unit's record was
expanded or the unit was walked again (whole numbers: no tolerance)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 3000])
@pytest.mark.parametrize("fmt", ["coo", "csr"])
@pytest.mark.parametrize("stage_words", [1 << 22, 0])
@pytest.mark.parametrize("cap", ["whole", "short"])
def test_negative_ids(n, fmt, stage_words, cap):
    from torchcompactradius_b200 import _lib
    from torchcompactradius_b200.search import make_desc
    lib = _lib.load()
    g = torch.Generator().manual_seed(n)
    x, h = torch.rand(n, 3, generator=g).cuda(), torch.full((n,), 0.2).cuda()
    ids = (torch.randperm(n, generator=g) - n // 2).to(torch.int32).cuda()
    ids[0], ids[1] = -2 ** 31, 2 ** 31 - 1
    s_bytes, w_bytes = _lib.search_sizes(n, n, 3)
    st, sc = (torch.empty(b, dtype=torch.uint8, device="cuda") for b in (s_bytes, w_bytes))
    stage = torch.empty(max(stage_words, 1), dtype=torch.int32, device="cuda")
    offsets = torch.empty(n + 1, dtype=torch.int64, device="cuda")
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    at = lambda t: ctypes.c_void_p(None if t is None else t.data_ptr())
    out = []
    for own in (None, ids):
        d = make_desc(3, "gather", 0, [0.0] * 3, [1.0] * 3, 4096, x, h, x, h, True)
        d.query_ids = d.ref_ids = None if own is None else own.data_ptr()
        _lib.check(lib.tcr_build_structure(ctypes.byref(d), at(st), s_bytes, at(sc), w_bytes, sp), "build")
        _lib.check(lib.tcr_count(ctypes.byref(d), at(st), at(sc), w_bytes, at(stage) if stage_words else None,
                                 stage_words, at(offsets), None, None, None, sp), "count")
        total = int(offsets[-1])
        room = total if cap == "whole" else total * 2 // 3
        row, col = (torch.full((room,), -7, dtype=torch.int64, device="cuda") for _ in range(2))
        _lib.check(lib.tcr_emit(ctypes.byref(d), at(st), at(sc), w_bytes, at(stage) if stage_words else None,
                                at(offsets), at(row if fmt == "coo" else None), at(col), room, sp), "emit")
        out.append((row, col))
    (r0, c0), (r1, c1) = out
    assert len(c0) > n // 2
    assert torch.equal(c1, ids[c0].long())
    if fmt == "coo":
        assert torch.equal(r1, ids[r0].long())
