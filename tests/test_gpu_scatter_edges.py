"""The scatter kernels at the edges of their chunks, rows, tiles and alignments, bit for bit against the
oracle (the folds keep the reference's order of operations: no tolerance)."""
import numpy as np
import pytest
import torch

from test_gpu_scatter import check_bits, oracle, run

pytestmark = pytest.mark.gpu


def values(dtype, shape, seed):
    g = torch.Generator().manual_seed(seed)
    if dtype.is_floating_point:
        return torch.randn(shape, generator=g).to(dtype)
    return torch.randint(-100, 100, shape, generator=g).to(dtype)


@pytest.mark.parametrize("reduce", ["sum", "max"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.float16, torch.int8])
@pytest.mark.parametrize("rows,longest", [(1, 1), (1, 9000), (31, 40), (32, 300), (33, 7), (100, 500), (257, 60)])
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_sorted_rows(reduce, dtype, rows, longest, shift):
    """Runs of 0 to `longest` elements (some rows empty, some longer than a tile), src and index starting off
    a 16-byte boundary."""
    rng = np.random.default_rng(rows * 31 + longest)
    counts = rng.integers(0, longest + 1, rows)
    counts[rows // 2] = longest
    index = torch.from_numpy(np.repeat(np.arange(rows), counts))
    n = index.numel()
    src = values(dtype, (n + shift,), rows)[shift:]
    src_d, index_d = torch.empty(n + shift, dtype=dtype, device="cuda")[shift:], torch.empty(n + shift, dtype=torch.int64, device="cuda")[shift:]
    src_d.copy_(src)
    index_d.copy_(index)
    got, arg = run(src_d, index_d, 0, reduce, None, rows)
    want, want_arg = oracle(src, index, 0, reduce, None, rows)
    check_bits(got, want, dtype)
    if arg is not None:
        assert np.array_equal(arg.cpu().numpy(), want_arg)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 15, 16, 17, 255, 4097])
@pytest.mark.parametrize("kind", ["gaps", "one", "descent_last", "descent_first", "unsorted"])
def test_index_chunks(n, kind):
    """Indices whose runs start, skip slots or descend at any place of a chunk of eight."""
    rng = np.random.default_rng(n)
    if kind == "gaps":
        index = np.sort(rng.integers(0, 40 * n + 1, n))
    elif kind == "one":
        index = np.full(n, 5)
    else:
        index = np.sort(rng.integers(0, n, n))
        if kind == "descent_last":
            index[-1] = 0
        elif kind == "descent_first":
            index[0] = n - 1
        else:
            rng.shuffle(index)
    size = int(index.max()) + 3
    src = values(torch.float32, (n,), n)
    index = torch.from_numpy(index)
    for dim_size in (size, None):
        got, _ = run(src.cuda(), index.cuda(), 0, "sum", None, dim_size)
        want, _ = oracle(src, index, 0, "sum", None, dim_size)
        check_bits(got, want, torch.float32)
    with pytest.raises(IndexError):
        run(src.cuda(), index.cuda(), 0, "sum", None, int(index.max()))
    bad = index.clone()
    bad[n // 2] = -1
    with pytest.raises(IndexError):
        run(src.cuda(), bad.cuda(), 0, "sum", None, size)


@pytest.mark.parametrize("features", [1, 3, 8])
@pytest.mark.parametrize("mean", [1, 7, 8, 9, 40])
def test_permuted_folds(features, mean):
    """Unsorted indices: folds through the sort's permutation, eight elements at a time."""
    rng = np.random.default_rng(mean)
    n = 300
    index = torch.from_numpy(rng.integers(0, n, n * mean))
    src = values(torch.float32, (n * mean, features), mean)
    for reduce in ("mean", "min"):
        got, arg = run(src.cuda(), index.cuda(), 0, reduce, None, n)
        want, want_arg = oracle(src, index, 0, reduce, None, n)
        check_bits(got, want, torch.float32)
        if arg is not None:
            assert np.array_equal(arg.cpu().numpy(), want_arg)
    full = torch.from_numpy(rng.integers(0, n, (n * mean, features)))
    got, _ = run(src.cuda(), full.cuda(), 0, "sum", None, n)
    check_bits(got, oracle(src, full, 0, "sum", None, n)[0], torch.float32)
