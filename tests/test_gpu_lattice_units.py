"""Units with several pairs inside the band of the product test (points on a lattice): decided in the unit,
with and without a staged record, over several windows of candidates, and in float64.  Against the C and the
double oracle (whole numbers: no tolerance)."""
import ctypes

import numpy as np
import pytest
import torch

import cases
from helpers import csr_rows
from oracle import compact, search64

pytestmark = pytest.mark.gpu


def lattice(dim, side, off_share=0.0, seed=0):
    """Cell centres of a grid over [-1, 1]^dim; a share of the points moved off them."""
    d = np.float32(2.0 / side)
    c = -1 + d * (np.arange(side, dtype=np.float32) + np.float32(0.5))
    x = np.stack(np.meshgrid(*[c] * dim, indexing="ij"), -1).reshape(-1, dim).astype(np.float32)
    rng = np.random.default_rng(seed)
    off = rng.random(len(x)) < off_share
    x[off] += rng.uniform(-0.3, 0.3, (int(off.sum()), dim)).astype(np.float32) * d
    return x[rng.permutation(len(x))], d


def search(x, h, mask, mode, stage_words):
    """Rows and columns of one self search over [-1, 1]^d through the C calls."""
    from torchcompactradius_b200 import _lib
    from torchcompactradius_b200.search import make_desc
    lib = _lib.load()
    x, h = torch.tensor(x).cuda(), torch.tensor(h).cuda()
    n, dim = x.shape
    d = make_desc(dim, mode, mask, [-1.0] * dim, [1.0] * dim, 4096, x, h, x, h, True)
    s_bytes, w_bytes = _lib.search_sizes(n, n, dim)
    st, sc = (torch.empty(b, dtype=torch.uint8, device="cuda") for b in (s_bytes, w_bytes))
    stage = torch.empty(max(stage_words, 1), dtype=torch.int32, device="cuda")
    offsets = torch.empty(n + 1, dtype=torch.int64, device="cuda")
    info = torch.zeros(8, dtype=torch.int64, pin_memory=True)
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    at = lambda t: ctypes.c_void_p(t.data_ptr())
    own = at(stage) if stage_words else None
    _lib.check(lib.tcr_build_structure(ctypes.byref(d), at(st), s_bytes, at(sc), w_bytes, sp), "build")
    _lib.check(lib.tcr_count(ctypes.byref(d), at(st), at(sc), w_bytes, own, stage_words, at(offsets), None, None,
                             at(info), sp), "count")
    torch.cuda.synchronize()
    total = int(info[0])
    row, col = (torch.full((total,), -1, dtype=torch.int64, device="cuda") for _ in range(2))
    _lib.check(lib.tcr_emit(ctypes.byref(d), at(st), at(sc), w_bytes, own, at(offsets), at(row), at(col), total, sp),
               "emit")
    return row.cpu().numpy(), col.cpu().numpy(), info.tolist()


@pytest.mark.parametrize("mode", cases.MODES)
@pytest.mark.parametrize("mask", [0, 7])
@pytest.mark.parametrize("stage_words", [1 << 22, 20000, 0])  # every record staged, some, none
@pytest.mark.parametrize("side,reach,off", [(14, 2.0, 0.0), (14, 2.0, 0.9), (20, 1.0, 0.5), (13, 3.0, 0.0)])
def test_staged_or_not(mode, mask, stage_words, side, reach, off):
    x, d = lattice(3, side, off, side)
    h = np.full(len(x), np.float32(d * np.float32(reach)))
    o = compact.radius_search(x, h, None, None, [-1.0] * 3, [1.0] * 3, [bool(mask)] * 3, mode, 4096)
    row, col, info = search(x, h, mask, mode, stage_words)
    got, want = cases.canonical(row, col), cases.canonical(o.row, o.col)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])
    if off == 0.0 and mask == 0:
        assert info[6] > len(x)  # (more than one pair a point lies on its threshold)


@pytest.mark.parametrize("mode", cases.MODES)
@pytest.mark.parametrize("dim,side,reach", [(2, 60, 12.0), (3, 16, 4.0), (1, 2000, 400.0)])
def test_several_windows(mode, dim, side, reach):
    """More than 1024 candidates a unit."""
    x, d = lattice(dim, side, 0.1, side)
    h = np.full(len(x), np.float32(d * np.float32(reach)))
    o = compact.radius_search(x, h, None, None, [-1.0] * dim, [1.0] * dim, [False] * dim, mode, 4096)
    row, col, _ = search(x, h, 0, mode, 1 << 24)
    got, want = cases.canonical(row, col), cases.canonical(o.row, o.col)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])


@pytest.mark.parametrize("mode", cases.MODES)
@pytest.mark.parametrize("per", [False, True])
def test_float64(mode, per):
    """Lattice points in double; some supports one rounding above the distance, which float32 does not see."""
    import torchcompactradius_b200 as tcr
    side = 9
    d = 2.0 / side
    c = -1 + d * (np.arange(side) + 0.5)
    x = np.stack(np.meshgrid(c, c, c, indexing="ij"), -1).reshape(-1, 3)
    h = np.full(len(x), 2.0 * d)
    h[::3] = np.nextafter(np.nextafter(h[::3], 1.0), 1.0)
    dom = tcr.DomainDescription(torch.full((3,), -1.0, dtype=torch.float64), torch.full((3,), 1.0, dtype=torch.float64),
                                torch.tensor([per] * 3), 3)
    adj = tcr.radiusSearch(tcr.PointCloud(torch.tensor(x).cuda(), torch.tensor(h).cuda()), mode=mode, domain=dom,
                           algorithm="compact", format="csr")
    want = cases.canonical(*search64.radius_search(x, h, None, None, [-1.0] * 3, [1.0] * 3, [per] * 3, mode))
    got = cases.canonical(*csr_rows(adj))
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])
