"""Grids of more than 2^32 cells, whose int32 linear indices wrap (neighborhood.h:51-61): two cells of the
grid then share one key, one run of the sorted points and one query group.  Against the C oracle (whole
numbers: no tolerance)."""
import ctypes

import numpy as np
import pytest
import torch

import cases
from oracle import compact

pytestmark = pytest.mark.gpu

SIDE = 2048  # cells per dimension of the unit box: cell (x, y, z + 1024) has the linear index of (x, y, z)
H = np.float32(1 / 2048.9)


def points(m, seed):
    """m points in and around each of two cells that share a linear index, and single points elsewhere."""
    rng = np.random.default_rng(seed)
    a = np.array([100, 200, 300]) + rng.uniform(-1.2, 2.2, (m, 3))
    a[: m // 2] = np.array([100, 200, 300]) + rng.uniform(0.02, 0.98, (m // 2, 3))
    b = a + [0, 0, 1024] + rng.uniform(-0.3, 0.3, (m, 3))
    x = np.concatenate([a, b, rng.uniform(10, SIDE - 10, (64, 3))]) / SIDE
    return x[rng.permutation(len(x))].astype(np.float32)


def search(x, h, per, mode, stage_words):
    """One self search through the C calls, with a staging list of stage_words (0: every unit is walked
    again by the emit)."""
    from torchcompactradius_b200 import _lib
    from torchcompactradius_b200.search import make_desc
    lib = _lib.load()
    x, h = torch.tensor(x).cuda(), torch.tensor(h).cuda()
    n, dim = x.shape
    mask = sum(1 << k for k, p in enumerate(per) if p)
    d = make_desc(dim, mode, mask, [0.0] * dim, [1.0] * dim, 4096, x, h, x, h, True)
    s_bytes, w_bytes = _lib.search_sizes(n, n, dim)
    st, sc = (torch.empty(b, dtype=torch.uint8, device="cuda") for b in (s_bytes, w_bytes))
    stage = torch.empty(max(stage_words, 1), dtype=torch.int32, device="cuda")
    offsets = torch.empty(n + 1, dtype=torch.int64, device="cuda")
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    at = lambda t: ctypes.c_void_p(t.data_ptr())
    _lib.check(lib.tcr_build_structure(ctypes.byref(d), at(st), s_bytes, at(sc), w_bytes, sp), "build")
    _lib.check(lib.tcr_count(ctypes.byref(d), at(st), at(sc), w_bytes, at(stage) if stage_words else None, stage_words,
                             at(offsets), None, None, None, sp), "count")
    total = int(offsets[-1])
    row, col = (torch.full((total,), -1, dtype=torch.int64, device="cuda") for _ in range(2))
    _lib.check(lib.tcr_emit(ctypes.byref(d), at(st), at(sc), w_bytes, at(stage), at(offsets), at(row), at(col), total,
                            sp), "emit")
    return row.cpu().numpy(), col.cpu().numpy()


@pytest.mark.parametrize("per", [[1, 1, 1], [0, 0, 0], [1, 0, 1]])
@pytest.mark.parametrize("mode", ["gather", "superSymmetric"])
@pytest.mark.parametrize("stage_words", [1 << 20, 0])
@pytest.mark.parametrize("m", [8, 40])
def test_cells_sharing_a_linear_index(per, mode, stage_words, m):
    x = points(m, 10 * m + sum(per))
    h = np.full(len(x), H)
    o = compact.radius_search(x, h, None, None, [0.0] * 3, [1.0] * 3, [bool(p) for p in per], mode, 4096)
    assert np.prod(o.cell_count.astype(np.float64)) > 2.0 ** 32
    got, want = cases.canonical(*search(x, h, per, mode, stage_words)), cases.canonical(o.row, o.col)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])
