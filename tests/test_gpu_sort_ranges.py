"""The one-launch sort (csrc/tcr_sort.cuh) launched on its own: ranges of several tiles per block at small
sizes, against numpy's stable sort (whole numbers: no tolerance), and what it does when a wait at its
barrier runs out.  The launcher is compiled by the test from the header."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "torchcompactradius_b200", "csrc")

SOURCE = r"""
#include "tcr_sort.cuh"
using namespace tcr;

// Where every sorted pair and run start goes, in plain arrays.
template <typename K>
struct PlainTail {
    static constexpr bool kPlace = true, kRuns = true;
    int32_t* starts;
    int32_t* num_runs;
    int32_t* placed;
    K* run_key;
    __device__ void place(int64_t i, K, int32_t v) const { placed[i] = v; }
    __device__ void run(const K* keys, int64_t i, int32_t r) const { run_key[r] = keys[i]; }
};

// One launch of `blocks` blocks over n pairs; `bar` is what the barrier counter starts from.
template <typename K>
static int sort_on(void* keys0, void* keys1, int32_t* vals0, int32_t* vals1, int64_t n, SortStateT<K>* state,
                   int32_t* hist, int32_t* failed, int32_t* starts, int32_t* num_runs, int32_t* placed, void* run_key,
                   int blocks, unsigned bar, K lo, K hi, cudaStream_t st) {
    SortStateT<K> h;
    memset(&h, 0, sizeof(h));
    h.key_min = lo;
    h.key_max = hi;
    h.n_dev = -1;
    h.bar = bar;
    cudaError_t e = cudaMemcpyAsync(state, &h, sizeof(h), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(sort_coop_kernel<K, PlainTail<K>>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(CoopSmem<K>));
    if (e != cudaSuccess) return (int)e;
    K *k0 = (K*)keys0, *k1 = (K*)keys1;
    PlainTail<K> tail{starts, num_runs, placed, (K*)run_key};
    int chained = 1;
    void* args[] = {&k0, &k1, &vals0, &vals1, &n, &state, &hist, &failed, &chained, &tail};
    return (int)cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(sort_coop_kernel<K, PlainTail<K>>),
                                            dim3((unsigned)blocks), dim3(kCoopThreads), args, sizeof(CoopSmem<K>), st);
}
extern "C" int sort_probe(int wide, void* k0, void* k1, int32_t* v0, int32_t* v1, int64_t n, void* state, int32_t* hist,
                          int32_t* failed, int32_t* starts, int32_t* num_runs, int32_t* placed, void* run_key, int blocks,
                          unsigned bar, unsigned long long lo, unsigned long long hi, void* st) {
    if (wide)
        return sort_on<unsigned long long>(k0, k1, v0, v1, n, (SortState64*)state, hist, failed, starts, num_runs, placed,
                                           run_key, blocks, bar, lo, hi, (cudaStream_t)st);
    return sort_on<uint32_t>(k0, k1, v0, v1, n, (SortState32*)state, hist, failed, starts, num_runs, placed, run_key,
                             blocks, bar, (uint32_t)lo, (uint32_t)hi, (cudaStream_t)st);
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    from torchcompactradius_b200 import build
    d = tmp_path_factory.mktemp("sort")
    src, lib = str(d / "sort_probe.cu"), str(d / "sort_probe.so")
    with open(src, "w") as f:
        f.write("#include <cstring>\n" + SOURCE)
    subprocess.check_call([build._nvcc()] + build.NVCC_FLAGS + ["-I" + CSRC, "-o", lib, src])
    fn = ctypes.CDLL(lib).sort_probe
    vp = ctypes.c_void_p
    fn.argtypes = [ctypes.c_int] + [vp] * 4 + [ctypes.c_int64] + [vp] * 7 + [ctypes.c_int, ctypes.c_uint] + [
        ctypes.c_uint64] * 2 + [vp]
    return fn


def run(probe, keys, blocks, bar=0, failed=0):
    """Sorts keys (uint32 or uint64) on `blocks` blocks; returns the device arrays of the result."""
    n, wide = len(keys), keys.dtype == np.uint64
    new = lambda m, t: torch.full((max(m, 1),), -1, dtype=t, device="cuda")
    kt = torch.int64 if wide else torch.int32
    k0 = torch.from_numpy(keys.view(np.int64 if wide else np.int32).copy()).cuda()
    r = dict(k0=k0, k1=new(n, kt), v0=torch.arange(n, dtype=torch.int32, device="cuda"), v1=new(n, torch.int32),
             state=new(512, torch.int64), hist=new(256 * max(blocks, 1), torch.int32),
             failed=torch.tensor([failed], dtype=torch.int32, device="cuda"), starts=new(n + 1, torch.int32),
             num_runs=new(1, torch.int32), placed=new(n, torch.int32), run_key=new(n, kt))
    p = {k: ctypes.c_void_p(t.data_ptr()) for k, t in r.items()}
    rc = probe(int(wide), p["k0"], p["k1"], p["v0"], p["v1"], n, p["state"], p["hist"], p["failed"], p["starts"],
               p["num_runs"], p["placed"], p["run_key"], blocks, bar, int(keys.min()), int(keys.max()),
               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    return r


@pytest.mark.parametrize("dtype", [np.uint32, np.uint64])
@pytest.mark.parametrize("blocks,n", [(1, 1), (1, 8192), (1, 8193), (1, 30011), (2, 16384), (2, 16417), (3, 24577), (3, 70001),
                                      (8, 200003)])
@pytest.mark.parametrize("bits", [0, 5, 8, 17, 32, 44])
def test_tiles_per_block(probe, dtype, blocks, n, bits):
    """One tile a block (8192 pairs), one more pair, several tiles with a remainder."""
    if dtype is np.uint32 and bits > 32:
        pytest.skip("no such key")
    rng = np.random.default_rng(1000 * blocks + n + bits)
    keys = (rng.integers(0, 1 << bits, n) + (7 if bits < 30 else 0)).astype(dtype)
    r = run(probe, keys, blocks)
    order = np.argsort(keys, kind="stable")
    np.testing.assert_array_equal(r["placed"].cpu().numpy()[:n], order)
    srt = keys[order]
    starts = np.concatenate([[0], np.nonzero(srt[1:] != srt[:-1])[0] + 1])
    assert int(r["failed"][0]) == 0 and int(r["num_runs"][0]) == len(starts)
    np.testing.assert_array_equal(r["starts"].cpu().numpy()[:len(starts) + 1], np.append(starts, n))
    np.testing.assert_array_equal(r["run_key"].cpu().numpy()[:len(starts)].view(dtype), srt[starts])


def test_wait_that_runs_out(probe):
    """One arrival is missing at the first barrier: every block gives up within its limit, sets the flag and
    returns; the context stays usable."""
    keys = np.random.default_rng(0).integers(0, 1 << 20, 60000).astype(np.uint32)
    r = run(probe, keys, 4, bar=0xffffffff)
    assert int(r["failed"][0]) == 1
    assert int(r["num_runs"][0]) == -1 and bool((r["placed"] == -1).all())
    r = run(probe, keys, 4)
    assert int(r["failed"][0]) == 0
    np.testing.assert_array_equal(r["placed"].cpu().numpy(), np.argsort(keys, kind="stable"))


@pytest.mark.parametrize("blocks", [1, 4])
def test_after_a_failed_sort(probe, blocks):
    """A sort enqueued behind one that gave up (the flag is set already) touches nothing."""
    keys = np.random.default_rng(1).integers(0, 1 << 20, 8000 * blocks).astype(np.uint32)
    r = run(probe, keys, blocks, failed=1)
    assert int(r["failed"][0]) == 1 and int(r["num_runs"][0]) == -1
    assert bool((r["placed"] == -1).all()) and bool((r["starts"] == -1).all())
